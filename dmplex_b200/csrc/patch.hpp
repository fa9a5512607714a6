// Patch decomposition of a model's mesh: whole tendencies and RK4 runs from shared memory, for
// meshes whose tables fit there (up to about hexagon 5). A patch is a run of consecutive cells of the
// internal numbering (compact, along the Hilbert curve) with the edges that appear first in them; its
// halo is every entity its tendency reads, directly or through the vertex and flux values it
// recomputes. Each patch has one packed block of tables in local 16-bit indices.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

struct TriskModel;

namespace trisk {

// One patch. Local orders: state edges = [owned | further edges whose F and q are formed |
// edges read only by vertices and cells], state cells likewise, so an owned entity's local
// index is its offset from the patch's first one.
struct PatchDesc {
  int32_t c0, e0;              // first owned cell and edge (internal numbering)
  int32_t nOC, nOE;            // owned cells and edges: tendencies and RK4 updates
  int32_t nLC, nLE, nLV;       // cells (B), edges (F, q) and vertices formed here
  int32_t nSC, nSE;            // cells (h) and edges (u) of the stage state read here
  uint32_t halo_e, halo_c;     // offsets in the block: int32 ids of the halo's edges and cells
  uint32_t vert, fedge, fcell, tedge, tcell;  // offsets of the phases' tables
  uint32_t bytes;              // of the block (a multiple of 16)
  int64_t block;               // offset of the block in the table memory
};

struct Tagged;
struct PatchSet {
  int n = 0;                   // patches (0: the mesh does not decompose well)
  std::vector<PatchDesc> host;
  std::vector<char> host_tables;
  PatchDesc* desc = nullptr;   // device
  char* tables = nullptr;      // device: the patches' blocks
  size_t work_doubles = 0;     // the largest patch's vectors with F and B in the state's place ...
  size_t apart_doubles = 0;    // ... and with room of their own, y and the accumulator
  size_t max_bytes = 0;        // the largest block of tables
  int max_items = 0;           // the largest phase's entities
  int threads = 0;             // threads a block
  bool runs = false;           // RK4 runs in one launch (the device has cooperative launches)
  size_t smem = 0;             // a run's dynamic shared memory a block
  Tagged* exchange = nullptr;  // the halos' published values
  int* err = nullptr;          // a wait for a neighbour gave up
  unsigned base = 0;           // version of the state between calls
  bool expire = false;         // the next run tests the bounded wait (trisk_model_expire_wait_once)
};

// Decomposes the mesh into `patches` runs of cells (host side only); false if the edges are not
// numbered by first appearance in the cells or a patch outgrows 15-bit indices.
bool build_patches(const TriskModel& m, PatchSet& S, int patches);
// The model's patches for its RK4 runs and tendencies, uploaded, where its numbering and the
// shared memory allow (m.patches.n stays 0 otherwise).
void choose_patches(TriskModel& m);
// dy = tendency of y, both in file numbering (map = state_n2o) or internal (map = nullptr).
void patch_tendency(TriskModel& m, const double* y, double* dy, const int32_t* map);
// nsteps RK4 steps of the internal state m.y in one cooperative launch.
void patch_rk4(TriskModel& m, double dt, int64_t nsteps);
// Lets a kernel have the shared memory of a patch.
void patch_allow_smem(const void* kernel);
// The RK4 run whose first block publishes nothing (TRiSK, cell K).
const void* patch_expire_kernel();
// The exchanged versions start again, after a run in which a wait gave up.
void patch_restart(TriskModel& m);

}  // namespace trisk
