// Launch interface of the update kernels (host-visible declarations).
#pragma once

#include <cuda.h>

#include <vector>

#include "fdtd_device.cuh"
#include "planner.h"

namespace fdtd {

struct FieldPtrs {
    float *ex, *ey, *ez, *hx, *hy, *hz;
};

// Six CPML faces in the order x_n, x_p, y_n, y_p, z_n, z_p.
struct PsiSet {
    PsiFace f[6];
    float* base;  // the allocation that holds them all (StepParams::psi_off), 16-byte aligned size
    long long pad;
};

// One time step m with the two-pass schedule (E pass then H pass, in place). probes: those outside the
// CPML slabs; late: step m - 1 belongs to the same call, and its H probes are sampled here. After a call's
// last step launch_sample_probes does that.
cudaError_t launch_two_pass(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const ProbeAt* probes, int n_probes, bool late,
                            long long m, cudaStream_t st);

// A box of nodes [x0, x1) x [y0, y1) x [z0, z1).
struct NodeBox {
    int x0, y0, z0, x1, y1, z1;
};

// One two-pass step m over the nodes of box b only (inside the grid; the design region's E and
// the plate nodes as in launch_two_pass). Nodes outside b keep their values.
cudaError_t launch_two_pass_box(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const NodeBox& b, long long m,
                                cudaStream_t st);

// One two-pass step whose step index is *base + s (device counter; s counts a call's steps), for graph
// replay; handles without a design region or plates only.
cudaError_t launch_two_pass_rel(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const ProbeAt* probes, int n_probes,
                                const long long* base, int s, cudaStream_t st);

// E of the design region's nodes, fi/pin -> fo/pout, after a schedule's E kernels; nothing
// without a design region.
cudaError_t launch_design_e(const StepParams& p, const FieldPtrs& fi, const FieldPtrs& fo, const PsiSet& pin,
                            const PsiSet& pout, long long m, cudaStream_t st);

// E of the plate nodes (StepParams::plate_nodes), fi/pin -> fo/pout, after a schedule's E kernels; rows:
// of those without a coefficient row only.
cudaError_t launch_plate_e(const StepParams& p, const FieldPtrs& fi, const FieldPtrs& fo, const PsiSet& pin,
                           const PsiSet& pout, bool rows, long long m, cudaStream_t st);

// Fused schedule (yee_sweep.cu): one kernel per time step sweeps the whole grid, fields A -> B,
// CPML memory pin -> pout.
struct FusedMaps {  // tensor maps of buffer A
    CUtensorMap h[3];
    CUtensorMap e[3];
    CUtensorMap rec;  // coefficient rows (StepParams::rec)
};
cudaError_t launch_count_general(const DeviceGrid& g, const uint16_t* rec, const int4* nodes, int n, int* count, cudaStream_t st);
// *differ (device int) becomes 1 if a row's H coefficients are not those of row bg.
cudaError_t launch_rows_h(const MatCoef* coef, int n_rows, int bg, int* differ, cudaStream_t st);
cudaError_t launch_slab_rows(const DeviceGrid& g, const MatCoef* coef, int n_rows, float* const prof_kappa[6], float4* out,
                             cudaStream_t st);

// What a grid asks of the sweep: nothing but its rows; coefficient rows other than the background's in a
// CPML slab or on a low wall (SlabRows); a design region's rows besides.
enum { kSweepPlain = 0, kSweepMat = 1, kSweepDesign = 2 };
constexpr int kSweepSources = 8;  // lumped sources whose signal comes with the launch
struct SweepStep {
    const ProbeAt* probes;  // probes outside the CPML slabs
    int n_probes;
    int late;               // sample them for step m - 1 from fi
    const long long* base;  // device step counter that m counts from (captured launches), or NULL: the
                            // sources' signals are then read on the device
    int kind;
    float sig[kSweepSources];
};
cudaError_t sweep_configure();
cudaError_t launch_sweep(const FusedMaps& maps, const StepParams& p, const FieldPtrs& fi, const FieldPtrs& fo,
                         const PsiSet& pin, const PsiSet& pout, const SweepPlan& sg, const SweepStep& ss, long long m,
                         cudaStream_t st);
// The same probes for step m (from *base, if not NULL) from its finished fields f.
cudaError_t launch_sample_probes(const StepParams& p, const FieldPtrs& f, const ProbeAt* probes, int n, const long long* base,
                                 long long m, cudaStream_t st);
// encode_fn: the driver's cuTensorMapEncodeTiled. Returns 0 on success.
int encode_sweep_maps(FusedMaps* out, const DeviceGrid& g, float* const h[3], float* const e[3], const uint16_t* rec,
                      void* encode_fn);

// Setup kernels (setup_kernels.cu).
// r0 = 0: the reference's grading (sigma_opt); r0 > 0: sigma_max from that reflection coefficient.
cudaError_t launch_cpml_profiles(const DeviceGrid& g, float pi, float r0, float* const prof[18], cudaStream_t st);
cudaError_t launch_material_tables(const DeviceGrid& g, const MatProps* props, int n, MatCoef* coef,
                                   cudaStream_t st);
cudaError_t launch_lumped_coefs(const DeviceGrid& g, const uint8_t* mat, const MatProps* props,
                                LumpedEdge* edges, const int* boxes, const float* resist, const int* owner,
                                int n_edges, cudaStream_t st);
// kappa_dev: device array of 6 pointers {kappa_e x, kappa_m x, kappa_e y, kappa_m y, kappa_e z,
// kappa_m z}; out_dev: device array of 12 pointers, per axis {E slot 0, E slot 1, H slot 0, H slot 1}.
cudaError_t launch_bg_curl(const DeviceGrid& g, const MatCoef* coef, int bg, const float* const* kappa_dev,
                           float* const* out_dev, cudaStream_t st);
// tab: per axis the packed E and H tables (StepParams::te, th) from the profiles and out_dev's arrays.
cudaError_t launch_axis_tables(const DeviceGrid& g, float* const prof[18], float* const bg_curl[12], float4* const te[3],
                               float4* const th[3], cudaStream_t st);
cudaError_t launch_fill(float* p, long long n, float v, cudaStream_t st);
// Columns nx .. pitch-1 of every row of a field array set to v.
cudaError_t launch_fill_padding(float* p, const DeviceGrid& g, float v, cudaStream_t st);
// Node classes (StepParams::cls) from the material index and the lumped edges.
// design_box: the design region's cells or NULL (its edge box gets class kDesignNode).
// Set the node class of the listed nodes ({i, j, k, -}) to `value`.
cudaError_t launch_class_nodes(const DeviceGrid& g, const int4* nodes, int n, int value, uint8_t* cls, cudaStream_t st);
cudaError_t launch_node_class(const DeviceGrid& g, const uint8_t* mat, const LumpedEdge* edges, int n_edges,
                              const int* design_box, uint8_t* cls, cudaStream_t st);
// Largest material index of the grid's cells into *out (device int).
cudaError_t launch_index_max(const uint8_t* mat, const DeviceGrid& g, int* out, cudaStream_t st);
cudaError_t launch_paint(uint8_t* mat, const DeviceGrid& g, const int box[6], uint8_t value, cudaStream_t st);
// Interface rows (setup_kernels.cu). launch_iface_set collects the distinct seven-cell keys of the
// kInterfaceNode nodes in a device hash set (table: kIfaceTableSize slots; counters: 2 ints) and
// lists them, unsorted, in keys (kIfaceTableSize entries; counters[1] = their number).
// launch_iface_rows, given the n_keys sorted keys that get rows, writes the per-node coefficient
// rows (StepParams::rec; nodes without a row become kGeneral; slot_row: kIfaceTableSize ints of
// scratch). launch_iface_coefs computes the rows themselves (p: the handle's parameters with the
// material rows in place).
constexpr int kIfaceTableBits = 17;
constexpr int kIfaceTableSize = 1 << kIfaceTableBits;
cudaError_t launch_iface_set(const DeviceGrid& g, const uint8_t* cls, const uint8_t* mat, unsigned long long* table,
                             int* counters, unsigned long long* keys, cudaStream_t st);
// *edge_mat (device int) becomes 1 if such a row lies in a CPML slab or on a low wall.
cudaError_t launch_iface_rows(const DeviceGrid& g, uint8_t* cls, const uint8_t* mat, const unsigned long long* table,
                              const unsigned long long* keys, int n_keys, int* slot_row, uint16_t* rec, int* edge_mat,
                              cudaStream_t st);
cudaError_t launch_iface_coefs(const StepParams& p, const unsigned long long* keys, int n_keys, MatCoef* coef,
                               cudaStream_t st);
// The nodes of the probes inside a CPML slab to the general path (after launch_iface_rows), which
// samples them before the CPML correction.
cudaError_t launch_rec_probes(const DeviceGrid& g, const Probe* probes, int n, uint16_t* rec, cudaStream_t st);
// The listed plate nodes inside a CPML slab to the general path (grids without SlabRows).
cudaError_t launch_rec_slab_plates(const DeviceGrid& g, const int4* nodes, int n, uint16_t* rec, cudaStream_t st);
// Coefficient rows of listed nodes ({i, j, k, source or -1}: nodes with plate-covered or lumped
// edges, which no seven-cell key describes). launch_special_set collects their distinct rows by a
// 64-bit hash of the row and the source in the set of launch_iface_set (bit 63: a source), the list
// unsorted in keys, counters[1] their number. launch_special_rows, given the sorted keys, writes rows
// first + q of the coefficient table, the nodes' entries of rec, and the source rows' table (rows from
// first + n_plain on). A node whose row differs from its key's (equal hashes) stays general.
// launch_special_each gives node q row first + q instead (nodes with a source from n_plain on).
cudaError_t launch_special_each(const StepParams& p, const int4* nodes, int n, int n_plain, int first, MatCoef* coef,
                                SrcRow* src, uint16_t* rec, cudaStream_t st);
cudaError_t launch_special_set(const StepParams& p, const int4* nodes, int n, unsigned long long* table, int* counters,
                               unsigned long long* keys, cudaStream_t st);
cudaError_t launch_special_rows(const StepParams& p, const int4* nodes, int n, const unsigned long long* table,
                                const unsigned long long* keys, int n_keys, int n_plain, int first, int* slot_row,
                                MatCoef* coef, SrcRow* src, uint16_t* rec, cudaStream_t st);
// The lumped edges' nodes back to kRecGeneral | class in rec (after launch_iface_rows and launch_design_rows).
cudaError_t launch_rec_general(const DeviceGrid& g, const LumpedEdge* edges, int n_edges, const uint8_t* cls, uint16_t* rec,
                               cudaStream_t st);
// Rows of the nodes of the design edge box (class kDesignNode), like those of the interface nodes: their
// distinct keys, then the nodes' entries of rec (row first + q for the sorted key q; nodes without one stay
// general). launch_iface_coefs computes the rows, whose H coefficients apply.
cudaError_t launch_design_set(const DeviceGrid& g, const int* dbox, const uint8_t* cls, const uint8_t* mat, unsigned long long* table,
                              int* counters, unsigned long long* keys, cudaStream_t st);
cudaError_t launch_design_rows(const DeviceGrid& g, const int* dbox, const uint8_t* cls, const uint8_t* mat,
                               const unsigned long long* table, const unsigned long long* keys, int n_keys, int first, int* slot_row,
                               uint16_t* rec, cudaStream_t st);
// The nodes of the design edge box back to the general path.
cudaError_t launch_rec_design_general(const DeviceGrid& g, const int* dbox, const uint8_t* cls, uint16_t* rec, cudaStream_t st);
// StepParams::dcoef from the material index, the table and the design cells' eps_r.
cudaError_t launch_design_coefs(const StepParams& p, float4* dcoef, cudaStream_t st);

}  // namespace fdtd
