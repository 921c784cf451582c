// Work planners (host only, no CUDA types: also compiled on their own by the CPU tests, which check
// that the items cover every node exactly once). plan_sweep plans the fused schedule's sweep;
// plan_fused planned an earlier form of it, a sweep of the interior tiles and passes over the rest, and
// is reached by its tests only.
//
// plan_fused. A fused step reads buffer A and writes buffer B. Its nodes are split into
//   * interior items {x0, y0, k0, k1}: a kTileX x kTileY column over planes [k0, k1) whose nodes
//     and E halo are all interior (no CPML slab, no boundary plane), for the TMA sweep;
//   * shell items {x0, y0, k, code} for the per-node shell passes: blocks of up to 256 nodes of
//     planes k .. k + nk - 1, shape s = code & 15 (widths 32, 16, 64, 128, 256, 8, 4, 2, 1),
//     columns (code >> 4) & 511, rows (code >> 13) & 511, nk - 1 = (code >> 22) & 15; in four
//     lists by the CPML slabs their nodes may lie in (kPlanShellZ: z slabs only; kPlanShellYZ: y
//     and z; kPlanShellX: x only; kPlanShellAny: any), so that each list's kernel leaves the
//     impossible slab tests out;
//   * CPML items {x0, y0, k0, k1} (when asked for): kTileX x kTileY columns over planes [k0, k1)
//     whose x range (E halo included) is interior, for the CPML sweep (z and y slabs, boundary
//     planes and rows): the planes outside the interior z range above and below every interior
//     tile, and the y bands beside the swept rectangle over all planes. A band tile's rows may
//     reach outside the grid (rows below 0 or from ny on: the sweep leaves them out); its rows
//     inside the grid are all outside the swept rectangle. They replace the kPlanShellZ and
//     kPlanShellYZ items of those nodes.
#pragma once

#include <vector>

namespace fdtd {

constexpr int kTileX = 32, kTileY = 16;  // interior sweep tiles
constexpr int kMaxItemPlanes = 512;      // planes one sweep item streams (chunk + 2)
constexpr int kShellPlanes = 4;          // planes per shell item
enum { kPlanShellZ = 0, kPlanShellYZ = 1, kPlanShellX = 2, kPlanShellAny = 3, kPlanShellLists = 4 };

struct PlanItem {
    int x, y, z, w;  // same layout as int4
};


struct FusedPlan {
    std::vector<PlanItem> interior;
    std::vector<PlanItem> shell[kPlanShellLists];
    std::vector<PlanItem> cpml;
};

// Thickest CPML slab (cells) the CPML sweep takes: a slab then fits in one tile row band.
constexpr int kCpmlMaxSlab = kTileY - 1;

struct PlanGrid {
    int nx, ny, nz;
    int pxn, pxp, pyn, pyp, pzn, pzp;
};

// The sweep of the whole grid (yee_sweep.cu): tiles of kTileX x kSweepRows nodes from the origin, each
// cut into chunks of planes of nearly equal length: n_lo chunks of the planes below zlo, n_mid of
// [zlo, zhi) and n_hi of the rest. The middle chunks, and the E above their top plane, meet neither a
// z slab nor a z wall; grids where cutting there does not pay have n_mid chunks only (zlo 0, zhi nz).
constexpr int kSweepRows = 16;
constexpr int kMaxSweepChunk = 32;                   // planes of a chunk
constexpr int kMaxSweepPlanes = kMaxSweepChunk + 2;  // planes a chunk streams
#ifdef __CUDACC__
#define FDTD_HD __host__ __device__
#else
#define FDTD_HD
#endif
struct SweepPlan {
    int nbx, nby, nz;
    int zlo, zhi, n_lo, n_mid, n_hi;
    FDTD_HD int chunks() const { return n_lo + n_mid + n_hi; }
    FDTD_HD int chunk(int c) const {  // first plane of chunk c; nz for c = chunks()
        if (c < n_lo) return (int)((long long)c * zlo / n_lo);
        if (c < n_lo + n_mid) return zlo + (int)((long long)(c - n_lo) * (zhi - zlo) / n_mid);
        return c == chunks() ? nz : zhi + (int)((long long)(c - n_lo - n_mid) * (nz - zhi) / n_hi);
    }
};
// The sweep's ring of n stages. Plane q of a chunk (0: the plane below its first) lies in stage(q), its copy
// completes the phase with parity(q) of that stage's barrier. At the top of plane step k, before its copy is
// issued, the planes up to k - 2 have arrived and those below drain_end(k) have been asked for: a chunk that
// gives up there waits for the planes from drain_begin(k) on, the one whose wait failed among them.
struct SweepRing {
    FDTD_HD static constexpr int stage(int q, int n) { return q % n; }
    FDTD_HD static constexpr unsigned parity(int q, int n) { return (unsigned)(q / n) & 1u; }
    FDTD_HD static constexpr int drain_begin(int k) { return k - 1; }
    FDTD_HD static constexpr int drain_end(int k, int k1, int n) { return (k + n - 2 < k1 ? k + n - 2 : k1) + 1; }
};

// share: the part of the device the grid has to itself (1 / n for one of n grids swept at once). rows: materials
// lie in the CPML slabs (SlabRows).
SweepPlan plan_sweep(const PlanGrid& g, double share = 1.0, bool rows = false);

// Planes per interior item (see plan_chunk in planner.cpp).
int plan_chunk(const PlanGrid& g);

// design_box: the design region's cells {i0, j0, k0, i1, j1, k1} (edge box: nodes i0..i1,
// j0..j1, k0..k1) or NULL; interior tiles whose E positions reach it go to the shell.
// cpml_tiles: plan CPML items where the grid allows them (no design region, every y and z slab
// at most kCpmlMaxSlab cells, interior tiles present); otherwise those nodes stay in the shell.
void plan_fused(const PlanGrid& g, int kc, const int* design_box, FusedPlan& out, bool cpml_tiles = false);

}  // namespace fdtd
