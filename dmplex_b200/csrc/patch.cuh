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
// Measured (CUDA events around a synchronous call of 200 steps, us per RK4 step, before / after):
// hexagon 4 18.6 / 8.3 (TRiSK, cell K), 20.7 / 8.3 (Gassmann, vertex K); hexagon 5 21.5 / 10.4 and
// 22.4 / 11.0. Of a stage's 2.6 us on hexagon 5 the exchange of the halo takes about 1.5, the three
// phases 0.4 each: latency of barriers, shared-memory gathers and the FP64 sums. Larger meshes stay
// with the launches: the tables no longer fit, and with them read from L2 or streamed from HBM in
// every stage the patches measured 37 to 53 us on hexagon 6 (launches: 37 to 45) and 118 to 208 on
// hexagon 7 (123 to 148).
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
// The value of `version` at p, waited for; false if the wait gave up: after ten seconds (or 2^31
// polls, which the clock always beats; a neighbour may have to wait for an SM that another
// stream's kernel holds), or when another block's has.
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
      if (now - start > 10000000000LL || *reinterpret_cast<volatile int*>(err) != 0 || i >= (1u << 31)) {
        atomicExch(err, 1);
        x = 0.0;
        return false;
      }
    }
  }
}

template <class R, int P>
__device__ __forceinline__ void ldcg_members(const R* p, double (&x)[P]) {
  if constexpr (P == 1) {
    x[0] = (double)__ldcg(p);
  } else if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int q = 0; q < P; q += 2) {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(p + q));
      x[q] = v.x;
      x[q + 1] = v.y;
    }
  } else if constexpr (P == 2) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
    x[0] = v.x;
    x[1] = v.y;
  } else {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
  }
}

// the value a storage of type R would hold
template <class R, int P>
__device__ __forceinline__ void round_to(double (&x)[P]) {
  if constexpr (sizeof(R) == 4) {
#pragma unroll
    for (int p = 0; p < P; ++p) x[p] = (double)(float)x[p];
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

// A patch's vectors in shared memory, [entity][MC] doubles: the stage state u, h; F, q of the
// edges and B of the cells; the vertex values (TRiSK q_v, h_v, K_v; Gassmann zeta_v, h_v, K_v).
// Without APART, F takes the place of u (an edge's F is formed from its own u; the cells, which
// read other edges' u, come first) and, with no cell part in K, B that of h.
template <int PV, int KE, int MC, bool APART>
struct PatchVectors {
  using W = PatchRows<PV, KE>;
  static constexpr bool F_OWN = APART || KE == KE_CELL, B_OWN = APART || W::CELL;
  double *u, *h, *q, *v0, *v1, *v2, *F, *B;
  __device__ __forceinline__ PatchVectors(double* sm, const PatchDesc& D) {
    u = sm;
    h = u + (size_t)D.nSE * MC;
    q = h + (size_t)D.nSC * MC;
    v0 = q + (size_t)D.nLE * MC;
    v1 = v0 + (size_t)D.nLV * MC;
    v2 = v1 + (size_t)D.nLV * MC;
    double* p = v0 + (size_t)W::VARRAYS * D.nLV * MC;
    F = F_OWN ? p : u;
    B = B_OWN ? p + (F_OWN ? (size_t)D.nLE * MC : 0) : h;
  }
};

// Thread t of a phase over [entity][MC]: the entity and its first member, P members a thread.
template <int MC, int P>
__device__ __forceinline__ void patch_slot(int t, int& i, int& mm) {
  constexpr int L = MC / P;
  if constexpr (L == 1) {
    i = t;
    mm = 0;
  } else {
    i = t / L;
    mm = (t % L) * P;
  }
}

// vertices: zeta_v, h_v, q_v, K_v
template <int PV, int KE, class R, int MC, int P, class Vec>
__device__ __forceinline__ void patch_vertex(const PatchRow<PatchRows<PV, KE>::VI, PatchRows<PV, KE>::VD>& r,
                                             const Vec& S, int v, int mm) {
  using W = PatchRows<PV, KE>;
  double uu[VW][P], hh[VW][P], z[P], eta[P], q[P], kv[P];
#pragma unroll
  for (int k = 0; k < VW; ++k) {
    ld_members<double, P>(S.u + r.ix[k] * MC + mm, uu[k]);
    ld_members<double, P>(S.h + r.ix[VW + k] * MC + mm, hh[k]);
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    z[p] = 0.0;
    eta[p] = 0.0;
#pragma unroll
    for (int k = 0; k < VW; ++k) z[p] += r.w[k] * uu[k][p];
#pragma unroll
    for (int k = 0; k < VW; ++k) eta[p] += r.w[VW + k] * hh[k][p];
    if (W::TR) q[p] = (z[p] + r.w[W::VD - 1]) / eta[p];
    if (W::VERT) {
      kv[p] = 0.0;
#pragma unroll
      for (int k = 0; k < VW; ++k) kv[p] += r.w[(W::VERT ? 6 : 0) + k] * (uu[k][p] * uu[k][p]);
    }
  }
  const int o = v * MC + mm;
  if (W::TR) {
    round_to<R, P>(q);
    st_members<double, P>(S.v0 + o, q);
  } else {
    round_to<R, P>(z);
    st_members<double, P>(S.v0 + o, z);
  }
  if (!W::TR || W::VERT) {
    round_to<R, P>(eta);
    st_members<double, P>(S.v1 + o, eta);
  }
  if (W::VERT) {
    round_to<R, P>(kv);
    st_members<double, P>(S.v2 + o, kv);
  }
}

// edges: the mass flux F and the edge PV q
template <int PV, int KE, class R, int MC, int P, class Vec>
__device__ __forceinline__ void patch_edge(const PatchRow<PatchRows<PV, KE>::FEI, PatchRows<PV, KE>::FED>& r,
                                           const Vec& S, int e, int mm) {
  using W = PatchRows<PV, KE>;
  constexpr int wV = W::CELL ? 2 : 0, wR = W::TR ? 0 : wV + (W::VERT ? 2 : 0);
  double ue[P], hv0[P], hv1[P], hc0[P], hc1[P], a0[P], a1[P], Fo[P], qo[P];
  ld_members<double, P>(S.u + e * MC + mm, ue);
  ld_members<double, P>(S.v0 + r.ix[0] * MC + mm, a0);
  ld_members<double, P>(S.v0 + r.ix[1] * MC + mm, a1);
  if (W::VERT || !W::TR) {
    ld_members<double, P>(S.v1 + r.ix[0] * MC + mm, hv0);
    ld_members<double, P>(S.v1 + r.ix[1] * MC + mm, hv1);
  }
  if (W::CELL) {
    ld_members<double, P>(S.h + r.ix[W::CELL ? 2 : 0] * MC + mm, hc0);
    ld_members<double, P>(S.h + r.ix[W::CELL ? 3 : 0] * MC + mm, hc1);
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    double he;
    if (KE == KE_CELL)
      he = r.w[0] * hc0[p] + r.w[1] * hc1[p];
    else if (KE == KE_VERTEX)
      he = r.w[wV] * hv0[p] + r.w[wV + 1] * hv1[p];
    else
      he = r.w[0] * hc0[p] + r.w[1] * hc1[p] + r.w[wV] * hv0[p] + r.w[wV + 1] * hv1[p];
    Fo[p] = he * ue[p];
    if (W::TR) {
      qo[p] = (a0[p] + a1[p]) / 2;
    } else {
      const double z = r.w[wR] * a0[p] + r.w[wR + 1] * a1[p];
      const double eta = r.w[wR] * hv0[p] + r.w[wR + 1] * hv1[p];
      qo[p] = (z + r.w[W::FED - 1]) / eta;
    }
  }
  round_to<R, P>(Fo);
  round_to<R, P>(qo);
  st_members<double, P>(S.F + e * MC + mm, Fo);
  st_members<double, P>(S.q + e * MC + mm, qo);
}

// cells: the Bernoulli function B
template <int PV, int KE, class R, int MC, int P, class Vec>
__device__ __forceinline__ void patch_cell(const PatchRow<PatchRows<PV, KE>::FCI, PatchRows<PV, KE>::FCD>& r,
                                           const Vec& S, double gravity, int i, int mm) {
  using W = PatchRows<PV, KE>;
  constexpr int wV = W::CELL ? 6 : 0;
  double hi[P], K[P], B[P];
  ld_members<double, P>(S.h + i * MC + mm, hi);
#pragma unroll
  for (int p = 0; p < P; ++p) K[p] = 0.0;
  if (W::CELL) {
#pragma unroll
    for (int k = 0; k < CW; ++k) {
      double x[P];
      ld_members<double, P>(S.u + r.ix[k] * MC + mm, x);
#pragma unroll
      for (int p = 0; p < P; ++p) K[p] += r.w[k] * (x[p] * x[p]);
    }
  }
#pragma unroll
  for (int p = 0; p < P; ++p) B[p] = W::CELL ? K[p] + gravity * hi[p] : gravity * hi[p];
  if (W::VERT) {
    double s[P];
#pragma unroll
    for (int p = 0; p < P; ++p) s[p] = 0.0;
#pragma unroll
    for (int k = 0; k < CW; ++k) {
      double x[P];
      ld_members<double, P>(S.v2 + r.ix[wV + k] * MC + mm, x);
#pragma unroll
      for (int p = 0; p < P; ++p) s[p] += r.w[wV + k] * x[p];
    }
#pragma unroll
    for (int p = 0; p < P; ++p) B[p] += s[p];
  }
  round_to<R, P>(B);
  st_members<double, P>(S.B + i * MC + mm, B);
}

// owned edges: du
template <int PV, int KE, int MC, int P, class Vec>
__device__ __forceinline__ void patch_du(const PatchRow<PatchRows<PV, KE>::TEI, PatchRows<PV, KE>::TED>& r,
                                         const Vec& S, int e, int mm, double (&du)[P]) {
  using W = PatchRows<PV, KE>;
  constexpr int C0 = 2 * W::TEI - 2;
  double s[P], b0[P], b1[P];
#pragma unroll
  for (int p = 0; p < P; ++p) s[p] = 0.0;
  if (W::TR) {
    double qself[P];
    ld_members<double, P>(S.q + e * MC + mm, qself);
#pragma unroll
    for (int k = 0; k < W::SW; ++k) {
      double f[P], q[P];
      ld_members<double, P>(S.F + r.ix[k] * MC + mm, f);
      ld_members<double, P>(S.q + r.ix[k] * MC + mm, q);
#pragma unroll
      for (int p = 0; p < P; ++p) s[p] += r.w[k] * f[p] * (qself[p] + q[p]);
    }
  } else if (PV == PVM_GASSMANN_DERIVED) {
#pragma unroll
    for (int b = 0; b < 2; ++b) {  // the two vertices' blocks of six
      double qa[P], qb[P];
      ld_members<double, P>(S.q + r.ix[6 * b] * MC + mm, qa);
      ld_members<double, P>(S.q + r.ix[6 * b + 3] * MC + mm, qb);
#pragma unroll
      for (int k = 6 * b; k < 6 * b + 6; ++k) {
        double f[P];
        ld_members<double, P>(S.F + r.ix[k] * MC + mm, f);
#pragma unroll
        for (int p = 0; p < P; ++p) s[p] += r.w[k] * f[p] * (derived_pv_source(k) % 6 == 0 ? qa[p] : qb[p]);
      }
    }
  } else {
    double qself[P];
    if (PV == PVM_GASSMANN_MEAN) ld_members<double, P>(S.q + e * MC + mm, qself);
#pragma unroll
    for (int k = 0; k < W::SW; ++k) {
      double f[P], q[P];
      ld_members<double, P>(S.F + r.ix[k] * MC + mm, f);
      ld_members<double, P>(S.q + r.ix[PV == PVM_GASSMANN ? W::SW + k : k] * MC + mm, q);
#pragma unroll
      for (int p = 0; p < P; ++p) s[p] += r.w[k] * f[p] * (PV == PVM_GASSMANN_MEAN ? (qself[p] + q[p]) / 2 : q[p]);
    }
  }
  ld_members<double, P>(S.B + (r.ix[C0] & PATCH_INDEX) * MC + mm, b0);
  ld_members<double, P>(S.B + r.ix[C0 + 1] * MC + mm, b1);
#pragma unroll
  for (int p = 0; p < P; ++p) du[p] = (W::TR ? s[p] / 2 : s[p]) - (b1[p] - b0[p]) * r.w[W::TED - 1];
}

// owned cells: dh
template <int PV, int KE, int MC, int P, class Vec>
__device__ __forceinline__ void patch_dh(const PatchRow<3, 6>& r, const Vec& S, int mm, double (&dh)[P]) {
  double s[P];
#pragma unroll
  for (int p = 0; p < P; ++p) s[p] = 0.0;
#pragma unroll
  for (int k = 0; k < CW; ++k) {
    double f[P];
    ld_members<double, P>(S.F + (k == 0 ? r.ix[k] & PATCH_INDEX : r.ix[k]) * MC + mm, f);
#pragma unroll
    for (int p = 0; p < P; ++p) s[p] += r.w[k] * f[p];
  }
#pragma unroll
  for (int p = 0; p < P; ++p) dh[p] = -s[p];
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
  using Vec = PatchVectors<PV, KE, 1, false>;
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
    patch_vertex<PV, KE, double, 1, 1>(r, S, v, 0);
  }
  __syncthreads();
  for (int i = tid; i < D.nLC; i += nt) {
    PatchRow<W::FCI, W::FCD> r;
    r.load(T, D.fcell, cp, i);
    patch_cell<PV, KE, double, 1, 1>(r, S, A.gravity, i, 0);
  }
  if (W::CELL && !Vec::F_OWN) __syncthreads();
  for (int e = tid; e < D.nLE; e += nt) {
    PatchRow<W::FEI, W::FED> r;
    r.load(T, D.fedge, ep, e);
    patch_edge<PV, KE, double, 1, 1>(r, S, e, 0);
  }
  __syncthreads();
  for (int e = tid; e < D.nOE; e += nt) {
    PatchRow<W::TEI, W::TED> r;
    r.load(T, D.tedge, tp, e);
    double du[1];
    patch_du<PV, KE, 1, 1>(r, S, e, 0, du);
    const int g = D.e0 + e;
    A.dy[A.map ? A.map[g] : g] = du[0];
  }
  for (int i = tid; i < D.nOC; i += nt) {
    PatchRow<3, 6> r;
    r.load(T, D.tcell, op, i);
    double dh[1];
    patch_dh<PV, KE, 1, 1>(r, S, 0, dh);
    const int g = A.ne + D.c0 + i;
    A.dy[A.map ? A.map[g] : g] = dh[0];
  }
}

// nsteps RK4 steps in one cooperative launch, a block a patch, with the patch's tables, state and
// accumulator in shared memory for the whole run. Only the stage states of the halos move: as
// tagged values (`publish`, `receive`), so a block waits for the values themselves (no grid
// barrier, flag or fence), and blocks may run a stage ahead of one another. The values alternate
// between two buffers; a patch overwrites version k with k + 2 only after it has received k + 1
// from every patch that reads it (the halos are symmetric), which those formed after reading k.
template <int PV, int KE>
__global__ void __launch_bounds__(512, 1) k_patch_rk4(const PatchParams A) {
  extern __shared__ __align__(16) double patch_sm[];
  __shared__ PatchDesc D;
  __shared__ int gave_up;
  using W = PatchRows<PV, KE>;
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
  const PatchVectors<PV, KE, 1, true> S(akept + nO, D);
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
          ok &= receive(A.exchange + (size_t)(version & 1u) * A.N + g, version, x, A.err) ? 1 : 0;
        (edge ? S.u[D.nOE + i] : S.h[D.nOC + i]) = x;
      }
      if (!ok) gave_up = 1;
      __syncthreads();
      if (gave_up) return;
      for (int v = tid; v < D.nLV; v += nt) {
        PatchRow<W::VI, W::VD> r;
        r.load(T, D.vert, vp, v);
        patch_vertex<PV, KE, double, 1, 1>(r, S, v, 0);
      }
      __syncthreads();
      for (int e = tid; e < D.nLE; e += nt) {
        PatchRow<W::FEI, W::FED> r;
        r.load(T, D.fedge, ep, e);
        patch_edge<PV, KE, double, 1, 1>(r, S, e, 0);
      }
      for (int i = nt - 1 - tid; i < D.nLC; i += nt) {  // from the last thread down: the first have more edges
        PatchRow<W::FCI, W::FCD> r;
        r.load(T, D.fcell, cp, i);
        patch_cell<PV, KE, double, 1, 1>(r, S, A.gravity, i, 0);
      }
      __syncthreads();
      const double c = stage == EPI_STAGE3 ? A.dt : half;
      Tagged* out = A.exchange + (size_t)((version + 1u) & 1u) * A.N;
      for (int j = tid; j < nO; j += nt) {
        double kv[1], next;
        bool shared;
        if (j < D.nOE) {
          PatchRow<W::TEI, W::TED> r;
          r.load(T, D.tedge, tp, j);
          patch_du<PV, KE, 1, 1>(r, S, j, 0, kv);
          shared = (r.ix[2 * W::TEI - 2] & PATCH_PUBLISH) != 0;
        } else {
          PatchRow<3, 6> r;
          r.load(T, D.tcell, op, j - D.nOE);
          patch_dh<PV, KE, 1, 1>(r, S, 0, kv);
          shared = (r.ix[0] & PATCH_PUBLISH) != 0;
        }
        const double y = ykept[j];
        if (stage == EPI_STAGE4) {
          next = y + sixth * (akept[j] + kv[0]);
          if (!isfinite(next)) atomicOr(A.nonfinite, 1);
          ykept[j] = next;
          if (step == A.nsteps - 1) A.y[global(j)] = next;
        } else {
          akept[j] = stage == EPI_STAGE1 ? kv[0] : akept[j] + 2 * kv[0];
          next = y + c * kv[0];
        }
        if (shared) publish(out + global(j), next, version + 1u);
        *slot(j) = next;  // no phase reads the stage state any more
      }
    }
  }
}

}  // namespace trisk
