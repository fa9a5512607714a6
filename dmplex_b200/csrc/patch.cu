// Host side of the patch decomposition: building the patches' sets and packed tables, and the
// launches of their kernels (patch.cuh).
#include <algorithm>
#include <cstring>
#include <utility>

#include "model.hpp"
#include "patch.cuh"

namespace trisk {

namespace {

// What a model's tables say, in internal numbering, as the sets and tables are built from them.
struct Numbered {
  const TriskModel& m;
  const Coefficients& C;
  const bool cell, vert, tr;
  const int sw;
  const std::vector<int64_t>& stencil;
  explicit Numbered(const TriskModel& model)
      : m(model), C(model.C), cell(model.C.alpha != 0.0), vert(model.C.alpha != 1.0),
        tr(model.C.pv_flux == PV_TRISK), sw(tr ? model.C.tw : 12), stencil(tr ? model.C.trisk_edges : model.C.g_edges) {}
  // entry k of internal entity i's row in a file-numbered table
  static int64_t row(const std::vector<int64_t>& tab, int w, const std::vector<int32_t>& n2o, int64_t i, int k) {
    return tab[(int64_t)n2o[i] * w + k];
  }
  int32_t stencil_edge(int64_t e, int k) const { return m.edge_o2n[row(stencil, sw, m.edge_n2o, e, k)]; }
  int32_t pv_edge(int64_t e, int k) const { return m.edge_o2n[row(C.g_pv_edges, 12, m.edge_n2o, e, k)]; }
  int32_t edge_cell(int64_t e, int k) const { return m.cell_o2n[row(C.edge_cells, 2, m.edge_n2o, e, k)]; }
  int32_t edge_vertex(int64_t e, int k) const { return m.vert_o2n[row(C.edge_vertices, 2, m.edge_n2o, e, k)]; }
  int32_t cell_edge(int64_t i, int k) const { return m.edge_o2n[row(C.cell_edges, C.cw, m.cell_n2o, i, k)]; }
  int32_t cell_vertex(int64_t i, int k) const { return m.vert_o2n[row(C.vk_cell_vertices, C.cw, m.cell_n2o, i, k)]; }
  int32_t vertex_edge(int64_t v, int k) const { return m.edge_o2n[row(C.vertex_edges, C.vw, m.vert_n2o, v, k)]; }
  int32_t vertex_cell(int64_t v, int k) const { return m.cell_o2n[row(C.vertex_cells, C.vw, m.vert_n2o, v, k)]; }
};

// A growing list of distinct entities with their positions (a stamp per entity, reused from one
// patch to the next).
struct LocalSet {
  std::vector<int32_t> stamp, pos, list;
  int32_t mark = 0;
  explicit LocalSet(int64_t n) : stamp(n, 0), pos(n) {}
  void clear() {
    ++mark;
    list.clear();
  }
  void add(int32_t x) {
    if (stamp[x] == mark) return;
    stamp[x] = mark;
    pos[x] = (int32_t)list.size();
    list.push_back(x);
  }
  int at(int32_t x) const { return pos[x]; }
};

struct Sets {
  LocalSet e, c, v;
  int nLE = 0, nLC = 0;
  Sets(int64_t ne, int64_t nc, int64_t nv) : e(ne), c(nc), v(nv) {}
};

// The entities of the patch with cells [c0, c1) and edges [e0, e1).
void collect(const Numbered& N, Sets& S, int32_t c0, int32_t c1, int32_t e0, int32_t e1, bool pv_table) {
  const Coefficients& C = N.C;
  S.e.clear();
  S.c.clear();
  S.v.clear();
  for (int32_t e = e0; e < e1; ++e) S.e.add(e);
  for (int32_t e = e0; e < e1; ++e)
    for (int k = 0; k < N.sw; ++k) {
      S.e.add(N.stencil_edge(e, k));
      if (pv_table) S.e.add(N.pv_edge(e, k));
    }
  for (int32_t i = c0; i < c1; ++i) {
    S.c.add(i);
    for (int k = 0; k < C.cw; ++k) S.e.add(N.cell_edge(i, k));
  }
  S.nLE = (int)S.e.list.size();
  for (int32_t e = e0; e < e1; ++e)
    for (int k = 0; k < 2; ++k) S.c.add(N.edge_cell(e, k));
  S.nLC = (int)S.c.list.size();
  for (int j = 0; j < S.nLE; ++j)
    for (int k = 0; k < 2; ++k) S.v.add(N.edge_vertex(S.e.list[j], k));
  if (N.vert)
    for (int j = 0; j < S.nLC; ++j)
      for (int k = 0; k < C.cw; ++k) S.v.add(N.cell_vertex(S.c.list[j], k));
  for (int32_t v : S.v.list)
    for (int k = 0; k < C.vw; ++k) {
      S.e.add(N.vertex_edge(v, k));
      S.c.add(N.vertex_cell(v, k));
    }
  if (N.cell) {
    for (int j = 0; j < S.nLC; ++j)
      for (int k = 0; k < C.cw; ++k) S.e.add(N.cell_edge(S.c.list[j], k));
    for (int j = 0; j < S.nLE; ++j)
      for (int k = 0; k < 2; ++k) S.c.add(N.edge_cell(S.e.list[j], k));
  }
}

// Rows of one phase's tables for n entities: index pairs, then weights, as PatchTab reads them.
struct Rows {
  std::vector<char>& out;
  const size_t off;
  const int n, np, NI, ND;
  int ni = 0, nd = 0;
  Rows(std::vector<char>& o, int n_, int ni_, int nd_)
      : out(o), off(o.size()), n(n_), np(patch_pad(n_)), NI(ni_), ND(nd_) {
    out.resize(off + (size_t)np * (4 * NI + 8 * ND), 0);
  }
  template <class F>
  void index(F&& f) {  // the next index of every entity
    for (int i = 0; i < n; ++i) {
      const uint16_t x = (uint16_t)f(i);
      std::memcpy(out.data() + off + 4 * ((size_t)(ni / 2) * np + i) + 2 * (ni % 2), &x, 2);
    }
    ++ni;
  }
  template <class F>
  void weight(F&& f) {  // the next weight of every entity
    const size_t base = off + 4 * (size_t)NI * np, row = base + 16 * (size_t)(nd / 2) * np;
    const bool single = ND % 2 && nd == ND - 1;
    for (int i = 0; i < n; ++i) {
      const double x = f(i);
      std::memcpy(out.data() + (single ? row + 8 * (size_t)i : row + 16 * (size_t)i + 8 * (nd % 2)), &x, 8);
    }
    ++nd;
  }
};

}  // namespace

bool build_patches(const TriskModel& m, PatchSet& S, int patches) {
  const Numbered N(m);
  const Coefficients& C = N.C;
  const bool pv_table = m.pv == PVM_GASSMANN;
  if (C.cw > CW || C.vw > VW || C.tw > TWD) return false;
  patches = (int)std::min<int64_t>(patches, m.nc);
  // the patches' cells, and their edges: those that appear first in them
  std::vector<int32_t> c0(patches + 1), e0(patches + 1);
  for (int p = 0; p <= patches; ++p) c0[p] = (int32_t)(m.nc * p / patches);
  {
    std::vector<int32_t> owner(m.ne, -1);
    for (int p = 0; p < patches; ++p)
      for (int32_t i = c0[p]; i < c0[p + 1]; ++i)
        for (int k = 0; k < C.cw; ++k) {
          if (C.divergence[(int64_t)m.cell_n2o[i] * C.cw + k] == 0.0) continue;
          int32_t& o = owner[N.cell_edge(i, k)];
          if (o < 0) o = p;
        }
    for (int64_t e = 0; e < m.ne; ++e) {
      if (owner[e] < 0) owner[e] = patches - 1;          // an edge of no cell
      if (e > 0 && owner[e] < owner[e - 1]) return false;  // not numbered by first appearance
    }
    int64_t e = 0;
    for (int p = 0; p <= patches; ++p) {
      while (e < m.ne && owner[e] < p) ++e;
      e0[p] = (int32_t)e;
    }
    e0[patches] = (int32_t)m.ne;
  }
  auto owner_of = [&](const std::vector<int32_t>& start, int32_t x) {
    return (int)(std::upper_bound(start.begin(), start.end(), x) - start.begin()) - 1;
  };
  // What each patch reads of the others, and its symmetric closure: a patch that is read by one
  // it does not read itself gets one entity of that one in its halo, unused, so that every pair
  // exchanges both ways.
  std::vector<std::vector<int32_t>> reads(patches), extra(patches);
#pragma omp parallel
  {
    Sets L(m.ne, m.nc, m.nv);
#pragma omp for schedule(dynamic, 4)
    for (int p = 0; p < patches; ++p) {
      collect(N, L, c0[p], c0[p + 1], e0[p], e0[p + 1], pv_table);
      std::vector<int32_t>& r = reads[p];
      for (size_t j = e0[p + 1] - e0[p]; j < L.e.list.size(); ++j) r.push_back(owner_of(e0, L.e.list[j]));
      for (size_t j = c0[p + 1] - c0[p]; j < L.c.list.size(); ++j) r.push_back(owner_of(c0, L.c.list[j]));
      std::sort(r.begin(), r.end());
      r.erase(std::unique(r.begin(), r.end()), r.end());
    }
  }
  for (int p = 0; p < patches; ++p)
    for (int32_t q : reads[p])
      if (!std::binary_search(reads[q].begin(), reads[q].end(), p)) extra[q].push_back(p);
  std::vector<PatchDesc> desc(patches);
  std::vector<std::vector<char>> blocks(patches);
  std::vector<uint8_t> shared(m.N, 0);  // in some patch's halo
  bool ok = true;
#pragma omp parallel
  {
    Sets L(m.ne, m.nc, m.nv);
#pragma omp for schedule(dynamic, 4)
    for (int p = 0; p < patches; ++p) {
      collect(N, L, c0[p], c0[p + 1], e0[p], e0[p + 1], pv_table);
      for (int32_t q : extra[p]) {
        if (e0[q + 1] > e0[q])
          L.e.add(e0[q]);
        else
          L.c.add(c0[q]);
      }
      PatchDesc D{};
      D.c0 = c0[p];
      D.e0 = e0[p];
      D.nOC = c0[p + 1] - c0[p];
      D.nOE = e0[p + 1] - e0[p];
      D.nLC = L.nLC;
      D.nLE = L.nLE;
      D.nLV = (int)L.v.list.size();
      D.nSC = (int)L.c.list.size();
      D.nSE = (int)L.e.list.size();
      if (std::max(std::max(D.nSE, D.nSC), D.nLV) > PATCH_INDEX) {
#pragma omp atomic write
        ok = false;
        continue;
      }
      for (int j = D.nOE; j < D.nSE; ++j) {
#pragma omp atomic write
        shared[L.e.list[j]] = 1;
      }
      for (int j = D.nOC; j < D.nSC; ++j) {
#pragma omp atomic write
        shared[m.ne + L.c.list[j]] = 1;
      }
      std::vector<char>& out = blocks[p];
      auto halo = [&](const std::vector<int32_t>& list, int from) {
        const uint32_t off = (uint32_t)out.size();
        const size_t bytes = (list.size() - from) * sizeof(int32_t);
        out.resize(off + (size_t)round_up((int64_t)bytes, 16), 0);
        if (bytes) std::memcpy(out.data() + off, list.data() + from, bytes);
        return off;
      };
      D.halo_e = halo(L.e.list, D.nOE);
      D.halo_c = halo(L.c.list, D.nOC);
      const auto& en = m.edge_n2o;
      const auto& cn = m.cell_n2o;
      const auto& vn = m.vert_n2o;
      const auto& le = L.e.list;
      const auto& lc = L.c.list;
      const auto& lv = L.v.list;
      {  // vertices
        D.vert = (uint32_t)out.size();
        Rows R(out, D.nLV, 3, 6 + (N.vert ? 3 : 0) + (N.tr ? 1 : 0));
        auto w = [&](const std::vector<double>& t, int k) {
          R.weight([&](int i) { return k < C.vw ? t[(int64_t)vn[lv[i]] * C.vw + k] : 0.0; });
        };
        for (int k = 0; k < VW; ++k)
          R.index([&](int i) { return k < C.vw ? L.e.at(N.vertex_edge(lv[i], k)) : 0; });
        for (int k = 0; k < VW; ++k)
          R.index([&](int i) { return k < C.vw ? L.c.at(N.vertex_cell(lv[i], k)) : 0; });
        for (int k = 0; k < VW; ++k) w(C.curl, k);
        for (int k = 0; k < VW; ++k) w(C.vertex_height, k);
        if (N.vert)
          for (int k = 0; k < VW; ++k) w(C.vk_weights, k);
        if (N.tr) R.weight([&](int i) { return C.coriolis[vn[lv[i]]]; });
      }
      auto cell_edges = [&](Rows& R) {
        for (int k = 0; k < CW; ++k)
          R.index([&](int i) { return k < C.cw ? L.e.at(N.cell_edge(lc[i], k)) : 0; });
      };
      auto cell_weights = [&](Rows& R, const std::vector<double>& t) {
        for (int k = 0; k < CW; ++k)
          R.weight([&](int i) { return k < C.cw ? t[(int64_t)cn[lc[i]] * C.cw + k] : 0.0; });
      };
      {  // cells: B
        D.fcell = (uint32_t)out.size();
        Rows R(out, D.nLC, (N.cell ? 3 : 0) + (N.vert ? 3 : 0), (N.cell ? 6 : 0) + (N.vert ? 6 : 0));
        if (N.cell) cell_edges(R);
        if (N.vert)
          for (int k = 0; k < CW; ++k)
            R.index([&](int i) { return k < C.cw ? L.v.at(N.cell_vertex(lc[i], k)) : 0; });
        if (N.cell) cell_weights(R, C.kinetic);
        if (N.vert) cell_weights(R, C.vk_kites);
      }
      {  // edges: F and q
        D.fedge = (uint32_t)out.size();
        Rows R(out, D.nLE, 1 + (N.cell ? 1 : 0), (N.cell ? 2 : 0) + (N.vert ? 2 : 0) + (N.tr ? 0 : 3));
        auto w2 = [&](const std::vector<double>& t) {
          for (int k = 0; k < 2; ++k) R.weight([&](int i) { return t[2 * (int64_t)en[le[i]] + k]; });
        };
        for (int k = 0; k < 2; ++k) R.index([&](int i) { return L.v.at(N.edge_vertex(le[i], k)); });
        if (N.cell) {
          for (int k = 0; k < 2; ++k) R.index([&](int i) { return L.c.at(N.edge_cell(le[i], k)); });
          w2(C.edge_height);
        }
        if (N.vert) w2(C.vk_height);
        if (!N.tr) {
          w2(C.rhombus);
          R.weight([&](int i) { return C.g_coriolis[en[le[i]]]; });
        }
      }
      {  // owned edges: du
        D.tedge = (uint32_t)out.size();
        const int width = N.tr ? TWD : GW;
        Rows R(out, D.nOE, width / 2 + (pv_table ? GW / 2 : 0) + 1, width + 1);
        const std::vector<double>& t = N.tr ? C.trisk : C.g_weights;
        for (int k = 0; k < width; ++k)
          R.index([&](int i) { return k < N.sw ? L.e.at(N.stencil_edge(le[i], k)) : 0; });
        if (pv_table)
          for (int k = 0; k < GW; ++k) R.index([&](int i) { return L.e.at(N.pv_edge(le[i], k)); });
        for (int k = 0; k < 2; ++k) R.index([&](int i) { return L.c.at(N.edge_cell(le[i], k)); });
        for (int k = 0; k < width; ++k)
          R.weight([&](int i) { return k < N.sw ? t[(int64_t)en[le[i]] * N.sw + k] : 0.0; });
        R.weight([&](int i) { return C.inverse_dual[en[le[i]]]; });
      }
      {  // owned cells: dh
        D.tcell = (uint32_t)out.size();
        Rows R(out, D.nOC, 3, 6);
        cell_edges(R);
        cell_weights(R, C.divergence);
      }
      D.bytes = (uint32_t)out.size();
      desc[p] = D;
    }
  }
  if (!ok) return false;
  size_t total = 0;
  for (int p = 0; p < patches; ++p) total += blocks[p].size();
  S = PatchSet{};
  S.host_tables.resize(total);
  int64_t at = 0;
  const int varrays = N.tr ? 1 + (N.vert ? 2 : 0) : 2 + (N.vert ? 1 : 0);
  auto mark = [&](char* first) {  // the publish bit of an entity's packed index
    uint16_t x;
    std::memcpy(&x, first, 2);
    x |= (uint16_t)PATCH_PUBLISH;
    std::memcpy(first, &x, 2);
  };
  for (int p = 0; p < patches; ++p) {
    PatchDesc& D = desc[p];
    const int tei = (N.tr ? TWD : GW) / 2 + (pv_table ? GW / 2 : 0) + 1;
    for (int e = 0; e < D.nOE; ++e)
      if (shared[D.e0 + e]) mark(blocks[p].data() + D.tedge + 4 * ((size_t)(tei - 1) * patch_pad(D.nOE) + e));
    for (int i = 0; i < D.nOC; ++i)
      if (shared[m.ne + D.c0 + i]) mark(blocks[p].data() + D.tcell + 4 * (size_t)i);
    D.block = at;
    std::memcpy(S.host_tables.data() + at, blocks[p].data(), blocks[p].size());
    at += (int64_t)blocks[p].size();
    // as PatchVectors lays them out
    const size_t common = (size_t)D.nSE + D.nSC + D.nLE + (size_t)varrays * D.nLV;
    S.work_doubles = std::max(S.work_doubles, common + (N.vert ? 0 : D.nLE) + (N.cell ? D.nLC : 0));
    S.apart_doubles = std::max(S.apart_doubles, common + D.nLE + D.nLC + 2 * (size_t)(D.nOE + D.nOC));
    S.max_bytes = std::max(S.max_bytes, (size_t)D.bytes);
    S.max_items = std::max(S.max_items, std::max(std::max(D.nSE, D.nLV), std::max(D.nLE + D.nLC, D.nOE + D.nOC)));
  }
  S.n = patches;
  S.host = std::move(desc);
  return true;
}

namespace {

// Dynamic shared memory of a block with an SM to itself (227 KB less its static part).
constexpr size_t PATCH_SMEM = 225 * 1024;
constexpr int PATCH_STEPS = 4096;  // RK4 steps a launch

template <int PV, int KE>
const void* rk4_kernel() {
  return reinterpret_cast<const void*>(k_patch_rk4<PV, KE>);
}

}  // namespace

void patch_allow_smem(const void* kernel) {
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PATCH_SMEM));
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
}

namespace {

PatchParams params(TriskModel& m) {
  PatchSet& S = m.patches;
  PatchParams A{};
  A.desc = S.desc;
  A.tables = S.tables;
  A.ne = (int)m.ne;
  A.N = (int)m.N;
  A.gravity = m.gravity;
  A.y = m.y;
  A.exchange = S.exchange;
  A.err = S.err;
  A.nonfinite = m.flag;
  return A;
}

}  // namespace

void choose_patches(TriskModel& m) {
  PatchSet& S = m.patches;
  S = PatchSet{};
  if (m.nc_own != m.nc || m.ne_own != m.ne) return;  // a distributed model's part: ghosts, exchanges
  int coop = 0, sms = 0;
  CUDA_CHECK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, m.device));
  CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device));
  // A patch an SM, of at least four cells. On a B200 a patch of 96 cells with its halo takes about
  // all of an SM's shared memory; hexagon 5 has 69 a patch and takes 92 to 125 KB. (With the tables in
  // L2 instead larger patches run too, at hexagon 6 a few per cent either way: patch.cuh.)
  if (m.nc > 96 * (int64_t)sms) return;
  const int n = (int)std::max<int64_t>(1, std::min<int64_t>(sms, m.nc / 4));
  if (!build_patches(m, S, n)) {
    S = PatchSet{};
    return;
  }
  S.smem = S.max_bytes + S.apart_doubles * sizeof(double);
  if (S.smem > PATCH_SMEM) {  // a numbering that is not compact
    S = PatchSet{};
    return;
  }
  S.threads = (int)std::min<int64_t>(512, std::max<int64_t>(128, round_up(S.max_items, 32)));
  int occ = 0;
  with_modes(m.pv, m.ke, [&](auto pvc, auto kec) {
    constexpr int PV = decltype(pvc)::value, KE = decltype(kec)::value;
    const void* k = rk4_kernel<PV, KE>();
    patch_allow_smem(k);
    patch_allow_smem(reinterpret_cast<const void*>(k_patch_tendency<PV, KE>));
    CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, S.threads, S.smem));
  });
  if ((int64_t)occ * sms < S.n) {
    S = PatchSet{};
    return;
  }
  S.runs = coop != 0;  // the blocks of a run wait for one another
  S.tables = m.alloc<char>(S.host_tables.size());
  S.desc = m.alloc<PatchDesc>(S.n);
  CUDA_CHECK(cudaMemcpy(S.tables, S.host_tables.data(), S.host_tables.size(), cudaMemcpyHostToDevice));
  CUDA_CHECK(cudaMemcpy(S.desc, S.host.data(), S.n * sizeof(PatchDesc), cudaMemcpyHostToDevice));
  S.host_tables = std::vector<char>();
  if (!S.runs) return;
  S.exchange = m.alloc<Tagged>(2 * m.N);
  CUDA_CHECK(cudaMemset(S.exchange, 0, 2 * m.N * sizeof(Tagged)));
  S.base = 1;
  S.err = m.flag + 1;  // read with the non-finite flag in one copy
}

void patch_tendency(TriskModel& m, const double* y, double* dy, const int32_t* map) {
  PatchSet& S = m.patches;
  PatchParams A = params(m);
  A.u_in = y;
  A.dy = dy;
  A.map = map;
  with_modes(m.pv, m.ke, [&](auto pvc, auto kec) {
    constexpr int PV = decltype(pvc)::value, KE = decltype(kec)::value;
    k_patch_tendency<PV, KE><<<S.n, S.threads, S.work_doubles * sizeof(double), m.stream>>>(A);
  });
  CUDA_CHECK(cudaGetLastError());
  m.launches++;
}

void patch_rk4(TriskModel& m, double dt, int64_t nsteps) {
  PatchSet& S = m.patches;
  PatchParams A = params(m);
  A.dt = dt;
  const void* expire = S.expire ? patch_expire_kernel() : nullptr;
  S.expire = false;
  for (int64_t left = nsteps; left > 0; left -= A.nsteps) {
    A.nsteps = (int)std::min<int64_t>(left, PATCH_STEPS);
    A.base = S.base;
    with_modes(m.pv, m.ke, [&](auto pvc, auto kec) {
      constexpr int PV = decltype(pvc)::value, KE = decltype(kec)::value;
      void* args[] = {&A};
      CUDA_CHECK(cudaLaunchCooperativeKernel(expire ? expire : rk4_kernel<PV, KE>(), dim3((unsigned)S.n),
                                             dim3((unsigned)S.threads), args, S.smem, m.stream));
    });
    S.base += 4u * (unsigned)A.nsteps;
    m.launches++;
  }
}

void patch_restart(TriskModel& m) {
  PatchSet& S = m.patches;
  S.base = 1;
  CUDA_CHECK(cudaMemsetAsync(S.exchange, 0, 2 * m.N * sizeof(Tagged), m.stream));
}

}  // namespace trisk
