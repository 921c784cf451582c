// Two-pass schedule: an E pass then an H pass per time step, both in place, one thread per node.
//
// This is the reference's own order of work (calc_e then calc_h, solver fdtdrav.h:3222-3333)
// expressed over the compact data layout. It runs at any grid size and is the schedule the fused
// sweep is checked against bit for bit; both call the same update primitives (yee_common.cuh).
//
// Every pass may start while the one before it drains (launch_dependent). A step with boxes clear of the CPML, us,
// without that / now: 24^3 12.4 / 7.0, 64^3 16.5 / 11.5, 128^3 45.2 / 41.4, 160^3 92.5 / 88.0.
//
// The H pass goes through the planes from the top down: it begins with what the E pass wrote last, which L2
// still holds when the grid as a whole does not fit. From the bottom up / now: 160^3 94.3 / 88.0, 192^3 152 / 146,
// 225^3 257 / 252.
#include "node_rows.cuh"
#include "tma.cuh"

namespace fdtd {

// Grids of up to this many nodes take the kernels by coefficient row (node_rows.cuh), larger ones those
// by node class (node_global.cuh), whose byte per node and sixth CTA an SM tell where HBM bounds the
// pass. Per step, class / row, us: 24^3 9.0 / 7.0, 64^3 15.0 / 11.5, 128^3 45.7 / 41.4, 160^3 91.9 / 88.0, 192^3 147 /
// 146, 200^3 189 / 189, 225^3 252 / 270, 256^3 318 / 332.
constexpr long long kRowsNodes = 7LL << 20;

// CTAs of 256 per SM the kernels are compiled for. By class: 6 caps them at 40 registers (48 warps
// resident; the general path spills a few words), which measured 4-7 % faster at 512^3 than the
// compiler's own choice of 48 registers (5 CTAs). By row: 5, without spills in the common path
// (at 128^3 6 CTAs were 5 % slower, 4 CTAs 9 %).
template <bool kRows>
constexpr int kCtas = kRows ? 5 : 6;

// The nodes [b.x0, b.x1) x [b.y0, b.y1) x [b.z0, ..).
// Probes outside the CPML slabs hold the step's final values, so the kernels by row read them from the
// finished fields, a thread per probe: the H pass E's of its step, the next step's E pass H's (`late`,
// a step of the same call), and k_sample_probes those of a call's last step. (Kernels by class look
// each node up in its plane's list, which on a plane of 30 probes takes longer than the update.) Probes in
// a slab hold the value before the CPML correction and are the general path's.
struct ProbeList {
    const ProbeAt* at;
    int n, late;
};
__device__ __forceinline__ void sample_list(const StepParams& p, const FieldPtrs& f, const ProbeList& l, bool h, long long m) {
    if (blockIdx.z != 0) return;  // one plane's blocks: the others do not even look (128^3 44.0 -> 41.4 us a step)
    const int block = blockIdx.y * gridDim.x + blockIdx.x, step = 256 * gridDim.x * gridDim.y;
    for (long long q = block * 256 + threadIdx.y * 32 + threadIdx.x; q < l.n; q += step) {
        const ProbeAt r = l.at[q];
        if ((r.comp >= 3) == h) sample_at(r, f, p, m);
    }
}

// kRel (by class): the step counts from a device counter. The other kernels by class take it as it is: with
// the test for a counter in every thread, 512^3 took 2238 us a step, without 2197.
template <typename Idx, bool kRows, bool kDesign = false, bool kRel = false>
__global__ void __launch_bounds__(256, kCtas<kRows>)
    k_update_e(const __grid_constant__ StepParams p, const __grid_constant__ FieldPtrs f, const __grid_constant__ PsiSet ps,
               const __grid_constant__ NodeBox b, const __grid_constant__ ProbeList probes, const __grid_constant__ StepIndex step) {
    grid_dependency_wait();
    grid_launch_dependents();
    if (kRows && probes.late) sample_list(p, f, probes, true, step.at() - 1);
    const int i = b.x0 + blockIdx.x * 32 + threadIdx.x, j = b.y0 + blockIdx.y * 8 + threadIdx.y, k = b.z0 + blockIdx.z;
    if (i >= b.x1 || j >= b.y1) return;
    if constexpr (kRows) e_node_rows<Idx, kDesign>(p, f, ps, i, j, k, step);
    else e_node_global<false, false, false, Idx>(p, f, f, ps, ps, i, j, k, kRel ? step.at() : step.m);
}
template <typename Idx, bool kRows, bool kRel = false>
__global__ void __launch_bounds__(256, kCtas<kRows>)
    k_update_h(const __grid_constant__ StepParams p, const __grid_constant__ FieldPtrs f, const __grid_constant__ PsiSet ps,
               const __grid_constant__ NodeBox b, const __grid_constant__ ProbeList probes, const __grid_constant__ StepIndex step) {
    grid_dependency_wait();
    grid_launch_dependents();
    if (kRows && probes.n > 0) sample_list(p, f, probes, false, step.at());
    if (kRows && p.fom_sample && p.fom_read >= 0 && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0)
        *p.fom_sample = f.ez[p.fom_read];  // an FoM probe outside the design region: every E is final here
    const int i = b.x0 + blockIdx.x * 32 + threadIdx.x, j = b.y0 + blockIdx.y * 8 + threadIdx.y, k = b.z0 + gridDim.z - 1 - blockIdx.z;
    if (i >= b.x1 || j >= b.y1) return;
    if constexpr (kRows) h_node_rows<Idx>(p, f, ps, i, j, k, step);
    else h_node_global<false, Idx>(p, f, f, f, ps, ps, i, j, k, kRel ? step.at() : step.m);
}

// After the E pass by class: E of the nodes of the design region's edge box [d0, d3] x [d1, d4] x [d2, d5] (node class
// kDesignNode, which the other E kernels do not store), with the per-cell eps_r of the design
// cells. Design nodes are interior: no CPML memory, no lumped edge.
__global__ void __launch_bounds__(256) k_design_e(const __grid_constant__ StepParams p, FieldPtrs fi, FieldPtrs fo,
                                                  const __grid_constant__ PsiSet pin,
                                                  const __grid_constant__ PsiSet pout, long long m) {
    const int* d = p.dbox;
    // an FoM probe outside the design region: its E is final once the other E kernels are done
    if (p.fom_sample && p.fom_read >= 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 &&
        threadIdx.y == 0)
        *p.fom_sample = fi.ez[p.fom_read];
    const int i = d[0] + blockIdx.x * 32 + threadIdx.x;
    const int j = d[1] + blockIdx.y * 8 + threadIdx.y;
    const int k = d[2] + blockIdx.z;
    if (i > d[3] || j > d[4]) return;
    if (design_row(p, p.rec[(long long)k * p.g.plane + (long long)j * p.g.pitch + i])) e_node_design<true>(p, fi, fo, i, j, k, m);
    else e_node_global<true>(p, fi, fo, pin, pout, i, j, k, m);
}

// E of the nodes with a plate-covered edge (node class kPlateNode, which the other E kernels leave
// alone): one thread per listed node, plate-aware coefficients. rows: k_update_e has done those that have
// a coefficient row (all but probes and lumped edges in a slab and rows beyond the table).
__global__ void __launch_bounds__(128) k_plate_e(const __grid_constant__ StepParams p, FieldPtrs fi, FieldPtrs fo,
                                                 const __grid_constant__ PsiSet pin,
                                                 const __grid_constant__ PsiSet pout, bool rows, long long m) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= p.n_plate_nodes) return;
    const int4 v = p.plate_nodes[q];
    if (rows && p.rec[(long long)v.z * p.g.plane + (long long)v.y * p.g.pitch + v.x] < kRecGeneral) return;
    e_node_global<false, false, true>(p, fi, fo, pin, pout, v.x, v.y, v.z, m);
}

cudaError_t launch_plate_e(const StepParams& p, const FieldPtrs& fi, const FieldPtrs& fo, const PsiSet& pin,
                           const PsiSet& pout, bool rows, long long m, cudaStream_t st) {
    if ((rows ? p.n_plate_general : p.n_plate_nodes) <= 0) return cudaSuccess;
    k_plate_e<<<(p.n_plate_nodes + 127) / 128, 128, 0, st>>>(p, fi, fo, pin, pout, rows, m);
    return cudaGetLastError();
}

cudaError_t launch_design_e(const StepParams& p, const FieldPtrs& fi, const FieldPtrs& fo, const PsiSet& pin,
                            const PsiSet& pout, long long m, cudaStream_t st) {
    if (!p.deps) return cudaSuccess;
    const int* d = p.dbox;
    const dim3 grid((d[3] - d[0] + 32) / 32, (d[4] - d[1] + 8) / 8, d[5] - d[2] + 1);
    k_design_e<<<grid, dim3(32, 8, 1), 0, st>>>(p, fi, fo, pin, pout, m);
    return cudaGetLastError();
}

template <typename Idx, bool kRows>
static cudaError_t two_pass(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const NodeBox& b, const ProbeList& probes,
                            const StepIndex& step, cudaStream_t st) {
    const dim3 grid((b.x1 - b.x0 + 31) / 32, (b.y1 - b.y0 + 7) / 8, b.z1 - b.z0), block(32, 8, 1);
    const bool rel = !kRows && step.base;
    cudaError_t e = launch_dependent(kRows && p.deps ? k_update_e<Idx, kRows, kRows> : rel ? k_update_e<Idx, kRows, false, !kRows> : k_update_e<Idx, kRows>,
                                     grid, block, 0, st, p, f, ps, b, probes, step);
    if (e == cudaSuccess && !kRows) e = launch_design_e(p, f, f, ps, ps, step.m, st);
    if (e == cudaSuccess) e = launch_plate_e(p, f, f, ps, ps, kRows, step.m, st);
    if (e == cudaSuccess) e = launch_dependent(rel ? k_update_h<Idx, kRows, !kRows> : k_update_h<Idx, kRows>, grid, block, 0, st, p, f, ps, b, probes, step);
    return e;
}

// One step over the nodes of b: E, the design region's and the plate nodes' E, H. By row the design
// region's E is the E pass's own (out of line): a launch between the passes, whose few nodes leave the
// device idle, took 14 us of an adjoint's 54 us forward step at 128^3.
static cudaError_t two_pass(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const NodeBox& b, const ProbeList& probes,
                            const StepIndex& step, cudaStream_t st) {
    const DeviceGrid& g = p.g;
    // 32-bit node offsets when every offset (plus one plane of lookahead) fits
    if (g.plane * (long long)(g.nz + 1) >= (1LL << 31)) return two_pass<long long, false>(p, f, ps, b, probes, step, st);
    if ((long long)g.nx * g.ny * g.nz > kRowsNodes) return two_pass<uint32_t, false>(p, f, ps, b, probes, step, st);
    return two_pass<uint32_t, true>(p, f, ps, b, probes, step, st);
}

cudaError_t launch_two_pass_rel(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const ProbeAt* probes, int n_probes,
                                const long long* base, int s, cudaStream_t st) {
    if (p.deps || p.n_plate_nodes > 0) return cudaErrorInvalidValue;  // no design region, no plates
    return two_pass(p, f, ps, NodeBox{0, 0, 0, p.g.nx, p.g.ny, p.g.nz}, ProbeList{probes, n_probes, s > 0}, StepIndex{base, s}, st);
}

// The nodes [b.x0, b.x1) x [b.y0, b.y1) x [b.z0, b.z1) only (the adjoint's segment recompute, whose
// nodes outside a shrinking box around the design region are never read again). Same per-node code, so
// the nodes inside give the same bits as a whole-grid step; the steps' probes stand in the ring already.
cudaError_t launch_two_pass_box(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const NodeBox& b, long long m,
                                cudaStream_t st) {
    const DeviceGrid& g = p.g;
    if (b.x0 < 0 || b.y0 < 0 || b.z0 < 0 || b.x1 > g.nx || b.y1 > g.ny || b.z1 > g.nz) return cudaErrorInvalidValue;
    if (b.x1 <= b.x0 || b.y1 <= b.y0 || b.z1 <= b.z0) return cudaSuccess;
    return two_pass(p, f, ps, b, ProbeList{}, StepIndex{nullptr, m}, st);
}

cudaError_t launch_two_pass(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, const ProbeAt* probes, int n_probes, bool late,
                            long long m, cudaStream_t st) {
    return two_pass(p, f, ps, NodeBox{0, 0, 0, p.g.nx, p.g.ny, p.g.nz}, ProbeList{probes, n_probes, late}, StepIndex{nullptr, m}, st);
}

}  // namespace fdtd
