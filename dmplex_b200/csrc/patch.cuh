// Device side of the patch decomposition (patch.hpp): the phases of a tendency for one patch,
// from the stage state to the RK4 update, with every intermediate in shared memory.
//
// What it replaces on meshes small enough to hold whole in the SMs' shared memory: twelve launches
// an RK4 step, each a few microseconds of launch latency and of dependent L2 reads around well
// under a microsecond of work. Here a block loads its patch's stage state with a halo of about
// two cells once, forms the vertex values, F, q and B of the patch and its rim in shared memory
// (the rim is formed again by its neighbours: 1.6 to 1.7 times the edges on hexagon 5), and
// gathers from there with 16-bit local indices. Every value is formed by the expressions of
// kernels.cuh in the same order, so results are the same bit for bit.
//
// Measured (wall clock around a synchronous call of 200 steps, us per RK4 step, launches / patches):
// hexagon 4 18.7 / 7.9 (TRiSK, cell K), 20.6 / 7.9 (Gassmann, vertex K); hexagon 5 20.7 / 10.6 and
// 22.1 / 10.6. Of a stage's 2.65 us on hexagon 5 the exchange of the halo takes about 1.5, the three
// phases the rest: latency of barriers, shared-memory gathers and the FP64 sums. Larger meshes stay
// with the launches, since the tables no longer fit. Hexagon 6 with this kernel reading them from L2,
// launches / patches by scheme (runs of 100): TRiSK with cell, vertex, mixed K 33.5 / 31.7, 35.2 /
// 34.7, 35.5 / 34.9; Gassmann 33.2 / 32.0, 33.6 / 32.2, 35.2 / 39.7; Gassmann mean 36.4 / 38.1, 37.2 /
// 34.5, 37.6 / 43.8: 2 to 7 % faster for six pairs, 5 to 17 % slower for three, which no one rule on
// the mesh's size separates. On hexagon 7 such forms measured 118 to 208 (launches 123 to 148).
#pragma once
#include "kernels.cuh"
#include "patch.hpp"

namespace trisk {

struct Tagged;
struct PatchParams {
  const PatchDesc* desc;
  const char* tables;
  int ne, N;            // edges, state elements
  double gravity;
  // one tendency
  const double* u_in;   // the state ...
  double* dy;           // ... its tendency ...
  const int32_t* map;   // ... and where internal element j of both is (nullptr: at j)
  // RK4 runs
  double* y;
  Tagged* exchange;     // 2 x N published values
  int* err;             // a wait for a neighbour gave up
  int* nonfinite;
  double dt;
  int nsteps;
  unsigned base;        // the version of the state in y
};

// A patch's table block, in global memory (read past L1) or in shared memory.
template <bool RES>
struct PatchTab {
  const char* p;
  __device__ __forceinline__ uint32_t u32(uint32_t off) const {
    if constexpr (RES) return *reinterpret_cast<const uint32_t*>(p + off);
    uint32_t v;
    asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p + off));
    return v;
  }
  __device__ __forceinline__ double f64(uint32_t off) const {
    if constexpr (RES) return *reinterpret_cast<const double*>(p + off);
    double v;
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p + off));
    return v;
  }
  __device__ __forceinline__ double2 f64x2(uint32_t off) const {
    if constexpr (RES) return *reinterpret_cast<const double2*>(p + off);
    double2 v;
    asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p + off));
    return v;
  }
  // 2 NI local indices of entity i: NI rows of packed pairs, np entities a row
  template <int NI>
  __device__ __forceinline__ void idx(uint32_t off, int np, int i, int (&x)[2 * NI]) const {
#pragma unroll
    for (int r = 0; r < NI; ++r) {
      const uint32_t v = u32(off + 4u * (uint32_t)(r * np + i));
      x[2 * r] = (int)(v & 0xFFFFu);
      x[2 * r + 1] = (int)(v >> 16);
    }
  }
  // ND weights of entity i: rows of pairs, then a single row if ND is odd
  template <int ND>
  __device__ __forceinline__ void dbl(uint32_t off, int np, int i, double (&d)[ND]) const {
#pragma unroll
    for (int r = 0; r < ND / 2; ++r) {
      const double2 v = f64x2(off + 16u * (uint32_t)(r * np + i));
      d[2 * r] = v.x;
      d[2 * r + 1] = v.y;
    }
    if (ND % 2) d[ND - 1] = f64(off + 16u * (uint32_t)((ND / 2) * np) + 8u * (uint32_t)i);
  }
};

// Rows of the phases' packed tables: index pairs and weights of one entity.
template <int PV, int KE>
struct PatchRows {
  static constexpr bool CELL = KE != KE_VERTEX, VERT = KE != KE_CELL, TR = PV == PVM_TRISK;
  static constexpr int VI = 3, VD = 6 + (VERT ? 3 : 0) + (TR ? 1 : 0);
  static constexpr int FEI = 1 + (CELL ? 1 : 0), FED = (CELL ? 2 : 0) + (VERT ? 2 : 0) + (TR ? 0 : 3);
  static constexpr int FCI = (CELL ? 3 : 0) + (VERT ? 3 : 0), FCD = (CELL ? 6 : 0) + (VERT ? 6 : 0);
  static constexpr int SW = TR ? TWD : GW;  // stencil width
  static constexpr int TEI = SW / 2 + (PV == PVM_GASSMANN ? GW / 2 : 0) + 1, TED = SW + 1;
  static constexpr int TCI = 3, TCD = 6;
  static constexpr int VARRAYS = TR ? 1 + (VERT ? 2 : 0) : 2 + (VERT ? 1 : 0);  // vertex vectors kept
};

__host__ __device__ __forceinline__ int patch_pad(int n) { return (n + 7) & ~7; }

// A published state value: its two halves, each with the 32-bit version it belongs to, as two
// 64-bit words (each is written and read whole, so a reader that sees both versions has the
// value: no flag, fence or second round trip).
struct Tagged {
  unsigned long long lo, hi;
};
__device__ __forceinline__ void publish(Tagged* p, double x, unsigned version) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long t = (unsigned long long)version << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"((b & 0xFFFFFFFFull) | t), "l"((b >> 32) | t)
               : "memory");
}
// The longest wait for a neighbour's value, which takes microseconds (the neighbour may have to wait
// for an SM that another stream's kernel holds), and that of a run that tests the wait.
constexpr long long PATCH_WAIT_NS = 10000000000LL, PATCH_TEST_WAIT_NS = 5000000LL;
// The value of `version` at p, waited for; false if the wait gave up: after WAIT_NS (or 2^31 polls,
// which the clock always beats), or when another block's has.
template <long long WAIT_NS>
__device__ __forceinline__ bool receive(const Tagged* p, unsigned version, double& x, int* err) {
  long long start = 0;
  for (unsigned i = 1;; ++i) {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    if ((unsigned)(lo >> 32) == version && (unsigned)(hi >> 32) == version) {
      x = __longlong_as_double((long long)((lo & 0xFFFFFFFFull) | (hi << 32)));
      return true;
    }
    if ((i & 255u) == 0) {
      const long long now = barrier_ns();
      if (start == 0) start = now;
      if (now - start > WAIT_NS || *reinterpret_cast<volatile int*>(err) != 0 || i >= (1u << 31)) {
        atomicExch(err, 1);
        x = 0.0;
        return false;
      }
    }
  }
}

__device__ __forceinline__ void prefetch_l2(const char* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// One entity's row of a phase's tables.
template <int NI, int ND>
struct PatchRow {
  int ix[2 * NI];
  double w[ND];
  template <bool RES>
  __device__ __forceinline__ void load(const PatchTab<RES>& T, uint32_t off, int np, int i) {
    T.template idx<NI>(off, np, i, ix);
    T.template dbl<ND>(off + 4u * NI * (uint32_t)np, np, i, w);
  }
};

constexpr int PATCH_PUBLISH = 0x8000;  // in a packed index: the owned entity is in some halo
constexpr int PATCH_INDEX = 0x7FFF;

// A patch's vectors in shared memory: the stage state u, h; F, q of the edges and B of the cells; the
// vertex values (TRiSK q_v, h_v, K_v; Gassmann zeta_v, h_v, K_v). Without APART, F takes the place of
// u (an edge's F is formed from its own u; the cells, which read other edges' u, come first) except
// with the cell K alone, and, with no cell part in K, B that of h.
template <int PV, int KE, bool APART>
struct PatchVectors {
  using W = PatchRows<PV, KE>;
  static constexpr bool F_OWN = APART || KE == KE_CELL, B_OWN = APART || W::CELL;
  double *u, *h, *q, *v0, *v1, *v2, *F, *B;
  __device__ __forceinline__ PatchVectors(double* sm, const PatchDesc& D) {
    u = sm;
    h = u + D.nSE;
    q = h + D.nSC;
    v0 = q + D.nLE;
    v1 = v0 + D.nLV;
    v2 = v1 + D.nLV;
    double* p = v0 + W::VARRAYS * D.nLV;
    F = F_OWN ? p : u;
    B = B_OWN ? p + (F_OWN ? D.nLE : 0) : h;
  }
};

// vertices: zeta_v, h_v, q_v, K_v
template <int PV, int KE, class Vec>
__device__ __forceinline__ void patch_vertex(const PatchRow<PatchRows<PV, KE>::VI, PatchRows<PV, KE>::VD>& r,
                                             const Vec& S, int v) {
  using W = PatchRows<PV, KE>;
  double u[VW], z = 0.0, eta = 0.0;
#pragma unroll
  for (int k = 0; k < VW; ++k) u[k] = S.u[r.ix[k]];
#pragma unroll
  for (int k = 0; k < VW; ++k) z += r.w[k] * u[k];
#pragma unroll
  for (int k = 0; k < VW; ++k) eta += r.w[VW + k] * S.h[r.ix[VW + k]];
  S.v0[v] = W::TR ? (z + r.w[W::VD - 1]) / eta : z;
  if (!W::TR || W::VERT) S.v1[v] = eta;
  if (W::VERT) {
    double kv = 0.0;
#pragma unroll
    for (int k = 0; k < VW; ++k) kv += r.w[(W::VERT ? 6 : 0) + k] * (u[k] * u[k]);
    S.v2[v] = kv;
  }
}

// edges: the mass flux F and the edge PV q
template <int PV, int KE, class Vec>
__device__ __forceinline__ void patch_edge(const PatchRow<PatchRows<PV, KE>::FEI, PatchRows<PV, KE>::FED>& r,
                                           const Vec& S, int e) {
  using W = PatchRows<PV, KE>;
  constexpr int wV = W::CELL ? 2 : 0, wR = W::TR ? 0 : wV + (W::VERT ? 2 : 0), iC = W::CELL ? 2 : 0;
  const double ue = S.u[e], a0 = S.v0[r.ix[0]], a1 = S.v0[r.ix[1]];
  double hv0 = 0.0, hv1 = 0.0, hc0 = 0.0, hc1 = 0.0;
  if (W::VERT || !W::TR) {
    hv0 = S.v1[r.ix[0]];
    hv1 = S.v1[r.ix[1]];
  }
  if (W::CELL) {
    hc0 = S.h[r.ix[iC]];
    hc1 = S.h[r.ix[iC + (W::CELL ? 1 : 0)]];
  }
  double he;
  if (KE == KE_CELL)
    he = r.w[0] * hc0 + r.w[1] * hc1;
  else if (KE == KE_VERTEX)
    he = r.w[wV] * hv0 + r.w[wV + 1] * hv1;
  else
    he = r.w[0] * hc0 + r.w[1] * hc1 + r.w[wV] * hv0 + r.w[wV + 1] * hv1;
  S.F[e] = he * ue;
  if (W::TR) {
    S.q[e] = (a0 + a1) / 2;
  } else {
    const double z = r.w[wR] * a0 + r.w[wR + 1] * a1;
    const double eta = r.w[wR] * hv0 + r.w[wR + 1] * hv1;
    S.q[e] = (z + r.w[W::FED - 1]) / eta;
  }
}

// cells: the Bernoulli function B
template <int PV, int KE, class Vec>
__device__ __forceinline__ void patch_cell(const PatchRow<PatchRows<PV, KE>::FCI, PatchRows<PV, KE>::FCD>& r,
                                           const Vec& S, double gravity, int i) {
  using W = PatchRows<PV, KE>;
  constexpr int wV = W::CELL ? 6 : 0;
  double B = gravity * S.h[i];
  if (W::CELL) {
    double K = 0.0;
#pragma unroll
    for (int k = 0; k < CW; ++k) {
      const double x = S.u[r.ix[k]];
      K += r.w[k] * (x * x);
    }
    B = K + B;
  }
  if (W::VERT) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < CW; ++k) s += r.w[wV + k] * S.v2[r.ix[wV + k]];
    B += s;
  }
  S.B[i] = B;
}

// owned edges: du
template <int PV, int KE, class Vec>
__device__ __forceinline__ double patch_du(const PatchRow<PatchRows<PV, KE>::TEI, PatchRows<PV, KE>::TED>& r,
                                           const Vec& S, int e) {
  using W = PatchRows<PV, KE>;
  constexpr int C0 = 2 * W::TEI - 2;
  double s = 0.0;
  if (W::TR) {
    const double qself = S.q[e];
#pragma unroll
    for (int k = 0; k < W::SW; ++k) s += r.w[k] * S.F[r.ix[k]] * (qself + S.q[r.ix[k]]);
    s = s / 2;
  } else if (PV == PVM_GASSMANN_DERIVED) {
#pragma unroll
    for (int b = 0; b < 2; ++b) {  // the two vertices' blocks of six
      const double qa = S.q[r.ix[6 * b]], qb = S.q[r.ix[6 * b + 3]];
#pragma unroll
      for (int k = 6 * b; k < 6 * b + 6; ++k) s += r.w[k] * S.F[r.ix[k]] * (derived_pv_source(k) % 6 == 0 ? qa : qb);
    }
  } else {
    const double qself = PV == PVM_GASSMANN_MEAN ? S.q[e] : 0.0;
#pragma unroll
    for (int k = 0; k < W::SW; ++k) {
      const double q = S.q[r.ix[PV == PVM_GASSMANN ? W::SW + k : k]];
      s += r.w[k] * S.F[r.ix[k]] * (PV == PVM_GASSMANN_MEAN ? (qself + q) / 2 : q);
    }
  }
  return s - (S.B[r.ix[C0 + 1]] - S.B[r.ix[C0] & PATCH_INDEX]) * r.w[W::TED - 1];
}

// owned cells: dh
template <class Vec>
__device__ __forceinline__ double patch_dh(const PatchRow<3, 6>& r, const Vec& S) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < CW; ++k) s += r.w[k] * S.F[k == 0 ? r.ix[k] & PATCH_INDEX : r.ix[k]];
  return -s;
}

// One tendency of every patch (a block each), from the caller's state to the caller's tendency.
template <int PV, int KE>
__global__ void __launch_bounds__(512, 2) k_patch_tendency(const PatchParams A) {
  extern __shared__ __align__(16) double patch_sm[];
  __shared__ PatchDesc D;
  using W = PatchRows<PV, KE>;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid < (int)(sizeof(PatchDesc) / 4))
    reinterpret_cast<int*>(&D)[tid] = reinterpret_cast<const int*>(A.desc + blockIdx.x)[tid];
  __syncthreads();
  const PatchTab<false> T{A.tables + D.block};
  using Vec = PatchVectors<PV, KE, false>;
  const Vec S(patch_sm, D);
  const int vp = patch_pad(D.nLV), ep = patch_pad(D.nLE), cp = patch_pad(D.nLC), tp = patch_pad(D.nOE),
            op = patch_pad(D.nOC);
  if (tid == 0) prefetch_l2(T.p + D.vert, D.tcell - D.vert);
  for (int i = tid; i < D.nSE; i += nt) {
    const int g = i < D.nOE ? D.e0 + i : (int)T.u32(D.halo_e + 4u * (uint32_t)(i - D.nOE));
    S.u[i] = __ldcg(A.u_in + (A.map ? A.map[g] : g));
  }
  for (int i = tid; i < D.nSC; i += nt) {
    const int g = A.ne + (i < D.nOC ? D.c0 + i : (int)T.u32(D.halo_c + 4u * (uint32_t)(i - D.nOC)));
    S.h[i] = __ldcg(A.u_in + (A.map ? A.map[g] : g));
  }
  __syncthreads();
  for (int v = tid; v < D.nLV; v += nt) {
    PatchRow<W::VI, W::VD> r;
    r.load(T, D.vert, vp, v);
    patch_vertex<PV, KE>(r, S, v);
  }
  __syncthreads();
  for (int i = tid; i < D.nLC; i += nt) {
    PatchRow<W::FCI, W::FCD> r;
    r.load(T, D.fcell, cp, i);
    patch_cell<PV, KE>(r, S, A.gravity, i);
  }
  if (W::CELL && !Vec::F_OWN) __syncthreads();
  for (int e = tid; e < D.nLE; e += nt) {
    PatchRow<W::FEI, W::FED> r;
    r.load(T, D.fedge, ep, e);
    patch_edge<PV, KE>(r, S, e);
  }
  __syncthreads();
  for (int e = tid; e < D.nOE; e += nt) {
    PatchRow<W::TEI, W::TED> r;
    r.load(T, D.tedge, tp, e);
    const int g = D.e0 + e;
    A.dy[A.map ? A.map[g] : g] = patch_du<PV, KE>(r, S, e);
  }
  for (int i = tid; i < D.nOC; i += nt) {
    PatchRow<3, 6> r;
    r.load(T, D.tcell, op, i);
    const int g = A.ne + D.c0 + i;
    A.dy[A.map ? A.map[g] : g] = patch_dh(r, S);
  }
}

// nsteps RK4 steps in one cooperative launch, a block a patch, with the patch's tables, state and
// accumulator in shared memory for the whole run. Only the stage states of the halos move: as
// tagged values (`publish`, `receive`), so a block waits for the values themselves (no grid
// barrier, flag or fence), and blocks may run a stage ahead of one another. The values alternate
// between two buffers; a patch overwrites version k with k + 2 only after it has received k + 1
// from every patch that reads it (the halos are symmetric), which those formed after reading k.
// With EXPIRE (a test of the waits) the first block publishes nothing, so its neighbours give up.
template <int PV, int KE, bool EXPIRE>
__device__ __forceinline__ void patch_rk4_run(const PatchParams& A) {
  extern __shared__ __align__(16) double patch_sm[];
  __shared__ PatchDesc D;
  __shared__ int gave_up;
  using W = PatchRows<PV, KE>;
  constexpr long long WAIT_NS = EXPIRE ? PATCH_TEST_WAIT_NS : PATCH_WAIT_NS;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid < (int)(sizeof(PatchDesc) / 4))
    reinterpret_cast<int*>(&D)[tid] = reinterpret_cast<const int*>(A.desc + blockIdx.x)[tid];
  if (tid == 0) gave_up = 0;
  __syncthreads();
  char* kept = reinterpret_cast<char*>(patch_sm);
  for (uint32_t i = tid; i < D.bytes / 16; i += nt)
    reinterpret_cast<uint4*>(kept)[i] = reinterpret_cast<const uint4*>(A.tables + D.block)[i];
  const PatchTab<true> T{kept};
  const int nHE = D.nSE - D.nOE, nH = nHE + D.nSC - D.nOC, nO = D.nOE + D.nOC;
  double* ykept = reinterpret_cast<double*>(kept + D.bytes);  // y of the owned edges and cells
  double* akept = ykept + nO;                                 // their accumulator
  const PatchVectors<PV, KE, true> S(akept + nO, D);
  const int vp = patch_pad(D.nLV), ep = patch_pad(D.nLE), cp = patch_pad(D.nLC), tp = patch_pad(D.nOE),
            op = patch_pad(D.nOC);
  const double half = A.dt / 2, sixth = A.dt / 6;
  // of owned element j (edges, then cells): its global state index, its place in the stage state
  auto global = [&](int j) { return j < D.nOE ? D.e0 + j : A.ne + D.c0 + (j - D.nOE); };
  auto slot = [&](int j) { return j < D.nOE ? S.u + j : S.h + (j - D.nOE); };
  for (int j = tid; j < nO; j += nt) {
    const double y = __ldcg(A.y + global(j));
    ykept[j] = y;
    *slot(j) = y;
  }
  __syncthreads();  // the kept tables, the halo lists among them
  unsigned version = A.base;
  for (int step = 0; step < A.nsteps; ++step) {
#pragma unroll 1
    for (int stage = EPI_STAGE1; stage <= EPI_STAGE4; ++stage, ++version) {
      int ok = 1;
      for (int j = tid; j < nH; j += nt) {
        const bool edge = j < nHE;
        const int i = edge ? j : j - nHE;
        const int g = (edge ? 0 : A.ne) + (int)T.u32((edge ? D.halo_e : D.halo_c) + 4u * (uint32_t)i);
        double x;
        if (step == 0 && stage == EPI_STAGE1)
          x = __ldcg(A.y + g);
        else
          ok &= receive<WAIT_NS>(A.exchange + (size_t)(version & 1u) * A.N + g, version, x, A.err) ? 1 : 0;
        (edge ? S.u[D.nOE + i] : S.h[D.nOC + i]) = x;
      }
      if (!ok) gave_up = 1;
      __syncthreads();
      if (gave_up) return;
      for (int v = tid; v < D.nLV; v += nt) {
        PatchRow<W::VI, W::VD> r;
        r.load(T, D.vert, vp, v);
        patch_vertex<PV, KE>(r, S, v);
      }
      __syncthreads();
      for (int e = tid; e < D.nLE; e += nt) {
        PatchRow<W::FEI, W::FED> r;
        r.load(T, D.fedge, ep, e);
        patch_edge<PV, KE>(r, S, e);
      }
      for (int i = nt - 1 - tid; i < D.nLC; i += nt) {  // from the last thread down: the first have more edges
        PatchRow<W::FCI, W::FCD> r;
        r.load(T, D.fcell, cp, i);
        patch_cell<PV, KE>(r, S, A.gravity, i);
      }
      __syncthreads();
      const double c = stage == EPI_STAGE3 ? A.dt : half;
      Tagged* out = A.exchange + (size_t)((version + 1u) & 1u) * A.N;
      for (int j = tid; j < nO; j += nt) {
        double kv, next;
        bool shared;
        if (j < D.nOE) {
          PatchRow<W::TEI, W::TED> r;
          r.load(T, D.tedge, tp, j);
          kv = patch_du<PV, KE>(r, S, j);
          shared = (r.ix[2 * W::TEI - 2] & PATCH_PUBLISH) != 0;
        } else {
          PatchRow<3, 6> r;
          r.load(T, D.tcell, op, j - D.nOE);
          kv = patch_dh(r, S);
          shared = (r.ix[0] & PATCH_PUBLISH) != 0;
        }
        const double y = ykept[j];
        if (stage == EPI_STAGE4) {
          next = y + sixth * (akept[j] + kv);
          if (!isfinite(next)) atomicOr(A.nonfinite, 1);
          ykept[j] = next;
          if (step == A.nsteps - 1) A.y[global(j)] = next;
        } else {
          akept[j] = stage == EPI_STAGE1 ? kv : akept[j] + 2 * kv;
          next = y + c * kv;
        }
        if (shared && !(EXPIRE && blockIdx.x == 0)) publish(out + global(j), next, version + 1u);
        *slot(j) = next;  // no phase reads the stage state any more
      }
    }
  }
}

template <int PV, int KE>
__global__ void __launch_bounds__(512, 1) k_patch_rk4(const PatchParams A) {
  patch_rk4_run<PV, KE, false>(A);
}

}  // namespace trisk
