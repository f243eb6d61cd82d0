// path_route.cuh — the path engine: accu_threshold, accu_fraction, accu_capacity and accu_trigger (float32) and accu
// (float64) as prefix scans along the heavy paths of the flow forest.
//
// Along one flow path the threshold rule maps the outflow x of the upstream cell to
// max(x + s - threshold, 0), the fraction rule to fraction * (x + s), the capacity rule to
// min(x + s, capacity) and the trigger rule to x + s where that reaches the trigger, else 0, where s is the material
// of the cell plus the outflow of its other upstream cells.  These maps compose into maps of the same form
// (path_route.cu, PMap), so the outflows of a whole path follow from a prefix scan of the per-cell maps instead of a
// cell-by-cell walk (ALG/definition/accumulating_router.hpp:525-599 walks them one cell after the other;
// ALG/definition/accu_threshold.hpp:124-169, ALG/definition/accu_fraction.hpp:124-162 and
// ALG/definition/accu_capacity.hpp and accu_trigger.hpp enter_cell are the cell rules).
//
// The flow forest is cut into heavy paths: each cell continues the path of its upstream neighbour with
// the largest upstream area (the heavy one); the other upstream neighbours (light) end paths of their
// own.  A path's level is 0 when no cell of it has a light upstream neighbour, else one more than the
// largest level of those light paths; every path crosses at most log2(cells) light edges, so there are
// few levels.  Paths are laid out level by level, and within a level by the 64 x 64 tile of their bottom, each
// from its top (a cell without inflow) to its bottom (the cell whose downstream cell is on another path, off the
// array, a sink or no-data).  A call runs the levels in order; within a level every path is one segment of a
// single scan (a path's top map ignores its input, so segments need no flags).  What leaves a path at its
// bottom goes to a slot of the cell that it flows into; the slots of a cell are consecutive, and so are those
// of neighbouring positions, so a level reads its light inflow densely and not by gathers over the raster.
//
// Calls with infinite inputs or totals, which the float-float compositions cannot carry, are redone along the same paths
// with the cell rules of the walk engine (k_path_redo).
//
// Built once per flow-direction raster (on the first call that needs it) and kept by the topology.
#pragma once

#include <vector>

#include "common.cuh"

namespace lue_gb300 {

constexpr int kPathThreads = 256;  // CTA of the per-call kernels

// One level: positions [p0, p1).
struct PathLevel {
    int32_t p0 = 0, p1 = 0;
    int32_t cut0 = 0, ncut = 0;        // CTA ranges cut[cut0 + i] .. cut[cut0 + i + 1], i < ncut
    int longest = 0;                   // cells of the longest path
    int per = 1;                       // positions per thread
};

struct PathCore {
    int64_t npos = 0;                   // valid cells (positions)
    int32_t* order = nullptr;           // [npos] cell index, bit 31 set at the top cell of a path
    int32_t* path_slot = nullptr;       // [npos] at the bottom of a path: the slot that takes its outflow, or -1
    int32_t* slot_first = nullptr;      // [npos - slot_base + 1] first slot of a position
    // Large rasters, from the first call with two results on: [cells] position of a cell, -1 for no-data.
    int32_t* at = nullptr;
    bool at_decided = false;
    int32_t* cut = nullptr;             // path tops at which the CTAs of a level begin
    int64_t slot_base = 0;              // first position of level 1 (level 0 has no light inflow)
    int64_t nslots = 0;                 // light edges of the forest
    std::vector<PathLevel> levels;
    int64_t tiles = 0;                  // most CTAs of one level's scan
    int64_t bytes = 0;
};

struct TopologyCore;

// Builds the path layout of an acyclic raster (work: a scratch array of words_for(n) counters).
// LUE_GPU_ERANGE when the raster is beyond the engine's limits (2^31 cells).
int path_core_build(const TopologyCore* core, uint32_t* work, cudaStream_t stream, PathCore** out);
void path_core_free(PathCore* pc);

}  // namespace lue_gb300

struct lue_gpu_topology;

namespace lue_gb300 {

// accu_threshold (rule 1), accu_fraction (rule 2), accu_capacity (rule 3) and accu_trigger (rule 4), float32.
// *done is false when the engine does not apply (flow cycles, a raster beyond its limits, accu_trigger in place,
// LUE_GB300_ENGINE=walk or =stage): the caller then runs another engine.
int path_route_f32(lue_gpu_topology* t, int rule, const float* a, float as, const float* b, float bs, float* out,
                   float* rem, cudaStream_t stream, bool* done);
// accu, float64: prefix sums along the paths in plain doubles (only additions of terms >= 0, so no cancellation); not
// in place.
int path_accu_f64(lue_gpu_topology* t, const double* a, double as, double* out, cudaStream_t stream, bool* done);
// Frees the handle's path-engine buffers.
void path_buffers_free(lue_gpu_topology* t);
// Builds the path layout of t now (lue_gpu_topology_prepare).
int path_prepare(lue_gpu_topology* t, cudaStream_t stream);

}  // namespace lue_gb300
