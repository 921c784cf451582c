// Setup kernels: CPML profiles, per-material coefficient tables, lumped-edge coefficients,
// material painting and fills. They run once per simulation (fdtd_prepare).
//
// The CPML profile and lumped-element expressions are evaluated on the device with the same
// float/double mix and the same device powf/expf as the reference's setABCPML and defineSourceZ /
// defineResistor, so the resulting tables equal the reference's bit for bit.
#include "yee_common.cuh"
#include "yee_kernels.h"

namespace fdtd {

// Planes per CTA of the grid-sized setup kernels (one node per thread and plane).
constexpr int kSetupPlanes = 8;

// One axis of setABCPML (fdtdrav.h:1774-1891 for x_n, 1912-1941 for x_p, and the y / z mirrors).
// prof = {b_e, a_e, b_m, a_m, kappa_e, kappa_m}, each n entries. Nodes outside both slabs keep
// b = a = 1.2e-38 (setZero) and kappa = 1.
// r0 > 0 (not the reference's): sigma_max from the reflection coefficient r0 of a slab of P cells
// with grading order m, sigma_max = -(m + 1) ln(r0) / (2 eta0 P delta), eta0 = sqrt(mu0 / eps0)
// (Gedney's polynomial grading); kappa, alpha and the recurrences as the reference's.
__global__ void k_cpml_axis(float* be, float* ae, float* bm, float* am, float* ke, float* km, int n,
                            int pn_i, int pp_i, float delta, float dt, float eps_0, float mu_0, float pi, float r0) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    // parameters of fdtdrav.h:1774-1812, as float locals
    float npml = 3;
    float sigma_factor = 1.5;
    float kappa_max = 5;
    float alpha_max = 0.05;
    float alpha_min = 0.00;
    float sigma_opt = (npml + 1) / (150 * pi * 1 * delta);
    float sigma_max = sigma_factor * sigma_opt;
    const float pn = (float)pn_i, pp = (float)pp_i;
    float roe, rom;
    bool in = false;
    if (q < pn_i) {
        roe = (pn - q - 0.75) / pn;
        rom = (pn - q - 0.25) / pn;
        in = true;
        if (r0 > 0.f) sigma_max = -(npml + 1) * logf(r0) / (2.0f * sqrtf(mu_0 / eps_0) * pn * delta);
    } else if (q >= n - pp_i) {
        roe = (q - (n - pp - 1) - 0.75) / pp;
        rom = (q - (n - pp - 1) - 0.25) / pp;
        in = true;
        if (r0 > 0.f) sigma_max = -(npml + 1) * logf(r0) / (2.0f * sqrtf(mu_0 / eps_0) * pp * delta);
    }
    if (!in) {
        be[q] = kTiny; ae[q] = kTiny; bm[q] = kTiny; am[q] = kTiny; ke[q] = 1.0f; km[q] = 1.0f;
        return;
    }
    float sigma_pe = sigma_max * powf(roe, npml);
    float sigma_pm = sigma_max * powf(rom, npml);
    sigma_pm = sigma_pm * (mu_0 / eps_0);
    float kappa_e = 1 + (kappa_max - 1) * powf(roe, npml);
    float kappa_m = 1 + (kappa_max - 1) * powf(rom, npml);
    float alpha_e = alpha_min + (alpha_max - alpha_min) * (1 - roe);
    float alpha_m = alpha_min + (alpha_max - alpha_min) * (1 - rom);
    alpha_m = alpha_m * (mu_0 / eps_0);
    float b_e = expf((-dt / eps_0) * ((sigma_pe / kappa_e) + alpha_e));
    float a_e = (1 / delta) * (b_e - 1) * sigma_pe / (kappa_e * (sigma_pe + kappa_e * alpha_e));
    float b_m = expf((-dt / mu_0) * ((sigma_pm / kappa_m) + alpha_m));
    float a_m = (1 / delta) * (b_m - 1) * sigma_pm / (kappa_m * (sigma_pm + kappa_m * alpha_m));
    be[q] = b_e; ae[q] = a_e; bm[q] = b_m; am[q] = a_m; ke[q] = kappa_e; km[q] = kappa_m;
}

cudaError_t launch_cpml_profiles(const DeviceGrid& g, float pi, float r0, float* const prof[18], cudaStream_t st) {
    const int ns[3] = {g.nx, g.ny, g.nz};
    const int pn[3] = {g.pxn, g.pyn, g.pzn};
    const int pp[3] = {g.pxp, g.pyp, g.pzp};
    const float d[3] = {g.dx, g.dy, g.dz};
    for (int a = 0; a < 3; ++a) {
        float* const* P = prof + 6 * a;
        k_cpml_axis<<<(ns[a] + 127) / 128, 128, 0, st>>>(P[0], P[1], P[2], P[3], P[4], P[5], ns[a], pn[a], pp[a],
                                                         d[a], g.dt, g.eps0, g.mu0, pi, r0);
    }
    return cudaGetLastError();
}

// Coefficients of edges whose surrounding cells share material m (the averages of four / two equal
// values computed with the reference's formulas), plus the default entry for H faces on the low
// boundary of their axis (mu = 1, sigma_m = 1.2e-38).
__global__ void k_material_tables(const MatProps* props, int n, MatCoef* coef, DeviceGrid g) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > kMaxMaterials) return;
    MatCoef c;
    const float dp_e[3] = {g.dy, g.dz, g.dx}, dm_e[3] = {g.dz, g.dx, g.dy};
    const float dp_h[3] = {g.dz, g.dx, g.dy}, dm_h[3] = {g.dy, g.dz, g.dx};
    for (int q = 0; q < 3; ++q) {  // component q averages the values of axis q
        MatAxis a{1.0f, kTiny, 1.0f, kTiny};
        if (m < n && m != kDefaultEntry) a = props[m].a[q];
        const float eps = avg4(a.eps, a.eps, a.eps, a.eps);
        const float sig = avg4(a.sig, a.sig, a.sig, a.sig);
        const float mu = m == kDefaultEntry ? 1.0f : harm2(a.mu, a.mu);
        const float sm = m == kDefaultEntry ? kTiny : harm2(a.sigm, a.sigm);
        Coef3 e = coef3(eps, sig, g.dt, g.eps0, dp_e[q], dm_e[q]);
        c.e[q] = make_float4(e.a, e.bp, e.bm, 0.0f);
        Coef3 h = coef3(mu, sm, g.dt, g.mu0, dp_h[q], dm_h[q]);
        c.h[q] = make_float4(h.a, h.bp, h.bm, 0.0f);
    }
    coef[m] = c;
}

cudaError_t launch_material_tables(const DeviceGrid& g, const MatProps* props, int n, MatCoef* coef,
                                   cudaStream_t st) {
    k_material_tables<<<(kMaxMaterials + 1 + 127) / 128, 128, 0, st>>>(props, n, coef, g);
    return cudaGetLastError();
}

// Lumped-edge coefficient overrides (defineSourceZ fdtdrav.h:1368-1426 for sources,
// defineResistor fdtdrav.h:1429-1483 for resistors), from the edge-averaged eps_z / sigma_z; for
// Ex edges defineSourceX's (fdtdrav.h:1311-1365) from eps_x / sigma_x, with its per-component
// resistance (1 + je - js)(1 + ke - ks) / (ie - is) * rs and factor dt dx / (r dz dy).
// boxes: per owner {is,js,ks,ie,je,ke}; owner[e] = index of the element an edge belongs to.
__global__ void k_lumped_coefs(DeviceGrid g, const uint8_t* mat, const MatProps* props, LumpedEdge* edges,
                               const int* boxes, const float* resist, const int* owner, int n_edges) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_edges) return;
    LumpedEdge L = edges[e];
    const int* b = boxes + 6 * owner[e];
    float dt = g.dt, dx = g.dx, dy = g.dy, dz = g.dz, eps_0 = g.eps0;
    float rs = resist[owner[e]];
    float _is = (float)b[0], _js = (float)b[1], _ks = (float)b[2];
    float _ie = (float)b[3], _je = (float)b[4], _ke = (float)b[5];
    const long long n = (long long)L.k * g.plane + (long long)L.j * g.pitch + L.i;
    if (L.comp == 0) {
        float r_comp = (1 + _je - _js) * (1 + _ke - _ks) / (_ie - _is);
        r_comp = r_comp * rs;
        float rfactor = (dt * dx) / (r_comp * dz * dy);
        // eps_x / sigma_x of the edge: average of cells (i,j,k), (i,j-1,k), (i,j,k-1), (i,j-1,k-1)
        const MatAxis a = props[mat[n]].a[0], bb = props[mat[n - g.pitch]].a[0], c = props[mat[n - g.plane]].a[0],
                      d = props[mat[n - g.pitch - g.plane]].a[0];
        float eps_x = avg4(a.eps, bb.eps, c.eps, d.eps);
        float sig_x = avg4(a.sig, bb.sig, c.sig, d.sig);
        float den = __fadd_rn(__fmaf_rn(2.0f * eps_x, eps_0, __fmul_rn(dt, sig_x)), rfactor);
        float num = __fsub_rn(__fmaf_rn(2.0f * eps_x, eps_0, -__fmul_rn(dt, sig_x)), rfactor);
        L.ceze = __fdiv_rn(num, den);
        L.cezhy = __fdiv_rn(__fdiv_rn(2.0f * dt, dy), den);
        L.cezhx = __fdiv_rn(__fdiv_rn(-2.0f * dt, dz), den);
        L.cezj = 0.0f;  // the reference computes Cexj but never injects (calc_e, fdtdrav.h:681-685)
        edges[e] = L;
        return;
    }
    float r_comp = (1 + _ie - _is) * (1 + _je - _js) / (_ke - _ks);
    r_comp = r_comp * rs;
    float rfactor = (dt * dz) / (r_comp * dx * dy);
    float rfactor_aux = (r_comp * dx * dy);
    // eps_z / sigma_z of the edge: average of cells (i,j), (i-1,j), (i,j-1), (i-1,j-1) in plane k
    const MatAxis a = props[mat[n]].a[2], bb = props[mat[n - 1]].a[2], c = props[mat[n - g.pitch]].a[2],
                  d = props[mat[n - 1 - g.pitch]].a[2];
    float eps_z = avg4(a.eps, bb.eps, c.eps, d.eps);
    float sig_z = avg4(a.sig, bb.sig, c.sig, d.sig);
    float den = __fadd_rn(__fmaf_rn(2.0f * eps_z, eps_0, __fmul_rn(dt, sig_z)), rfactor);
    float num = __fsub_rn(__fmaf_rn(2.0f * eps_z, eps_0, -__fmul_rn(dt, sig_z)), rfactor);
    L.ceze = __fdiv_rn(num, den);
    L.cezhy = __fdiv_rn(__fdiv_rn(2.0f * dt, dx), den);
    L.cezhx = __fdiv_rn(__fdiv_rn(-2.0f * dt, dy), den);
    L.cezj = L.source >= 0 ? __fdiv_rn(__fdiv_rn(-2.0f * dt, rfactor_aux), den) : 0.0f;
    edges[e] = L;
}

cudaError_t launch_lumped_coefs(const DeviceGrid& g, const uint8_t* mat, const MatProps* props,
                                LumpedEdge* edges, const int* boxes, const float* resist, const int* owner,
                                int n_edges, cudaStream_t st) {
    if (n_edges == 0) return cudaSuccess;
    k_lumped_coefs<<<(n_edges + 127) / 128, 128, 0, st>>>(g, mat, props, edges, boxes, resist, owner, n_edges);
    return cudaGetLastError();
}

// Kappa-divided curl coefficients of material `bg` along each axis (the division setABCPML applies
// in its slabs, fdtdrav.h:1893-1906; kappa = 1 elsewhere leaves the coefficient unchanged).
// out[axis][slot]: E then H slots as documented on BgCurl.
__global__ void k_bg_curl(const MatCoef* coef, int bg, DeviceGrid g, const float* const* kappa, float* const* out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int a = blockIdx.y;
    const int n = a == 0 ? g.nx : a == 1 ? g.ny : g.nz;
    if (q >= n) return;
    const MatCoef c = coef[bg];
    const float ke = kappa[2 * a][q], km = kappa[2 * a + 1][q];
    // E slots: x {Ey minus, Ez plus}, y {Ex plus, Ez minus}, z {Ex minus, Ey plus}
    const float e0[3] = {c.e[1].z, c.e[0].y, c.e[0].z};
    const float e1[3] = {c.e[2].y, c.e[2].z, c.e[1].y};
    // H slots: x {Hy plus, Hz minus}, y {Hx minus, Hz plus}, z {Hx plus, Hy minus}
    const float h0[3] = {c.h[1].y, c.h[0].z, c.h[0].y};
    const float h1[3] = {c.h[2].z, c.h[2].y, c.h[1].z};
    out[4 * a + 0][q] = __fdiv_rn(e0[a], ke);
    out[4 * a + 1][q] = __fdiv_rn(e1[a], ke);
    out[4 * a + 2][q] = __fdiv_rn(h0[a], km);
    out[4 * a + 3][q] = __fdiv_rn(h1[a], km);
}

cudaError_t launch_bg_curl(const DeviceGrid& g, const MatCoef* coef, int bg, const float* const* kappa_dev,
                           float* const* out_dev, cudaStream_t st) {
    const int nmax = max(g.nx, max(g.ny, g.nz));
    k_bg_curl<<<dim3((nmax + 127) / 128, 3), 128, 0, st>>>(coef, bg, g, kappa_dev, out_dev);
    return cudaGetLastError();
}

// One axis of StepParams::te / th.
__global__ void k_axis_table(float4* te, float4* th, int n, const float* be, const float* ae, const float* bm,
                             const float* am, const float* e0, const float* e1, const float* h0, const float* h1) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    te[q] = make_float4(e0[q], e1[q], be[q], ae[q]);
    th[q] = make_float4(h0[q], h1[q], bm[q], am[q]);
}

// SlabRows: per axis the E entries of every row, then the H entries (rows of H on the low walls are
// the default entry's, so they need none of their own).
__global__ void k_slab_rows(const MatCoef* __restrict__ coef, DeviceGrid g, int n_rows, const float* kex, const float* key,
                            const float* kez, const float* kmx, const float* kmy, const float* kmz, float4* out) {
    const int lo[3] = {g.pxn, g.pyn, g.pzn}, hi[3] = {g.pxp, g.pyp, g.pzp}, n[3] = {g.nx, g.ny, g.nz};
    const float *ke[3] = {kex, key, kez}, *km[3] = {kmx, kmy, kmz};
    const int a = blockIdx.y, L = lo[a] + hi[a];
    for (int b = 0; b < a; ++b) out += 2LL * n_rows * (lo[b] + hi[b]);
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_rows * L) return;
    const int l = q % L, at = l < lo[a] ? l : n[a] - hi[a] + l - lo[a];
    const MatCoef& c = coef[q / L];
    const float size = a == 0 ? g.dx : a == 1 ? g.dy : g.dz;
    const float e0 = a == 0 ? c.e[1].z : a == 1 ? c.e[0].y : c.e[0].z, e1 = a == 0 ? c.e[2].y : a == 1 ? c.e[2].z : c.e[1].y;
    const float h0 = a == 0 ? c.h[1].y : a == 1 ? c.h[0].z : c.h[0].y, h1 = a == 0 ? c.h[2].z : a == 1 ? c.h[2].y : c.h[1].z;
    out[q] = make_float4(__fdiv_rn(e0, ke[a][at]), __fdiv_rn(e1, ke[a][at]), __fmul_rn(e0, size), __fmul_rn(e1, size));
    out[n_rows * L + q] = make_float4(__fdiv_rn(h0, km[a][at]), __fdiv_rn(h1, km[a][at]), __fmul_rn(h0, size), __fmul_rn(h1, size));
}

__global__ void k_rows_h(const MatCoef* __restrict__ coef, int n_rows, int bg, int* differ) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_rows) return;
    const uint32_t *a = reinterpret_cast<const uint32_t*>(coef[q].h), *b = reinterpret_cast<const uint32_t*>(coef[bg].h);
    for (int w = 0; w < (int)(sizeof(MatCoef::h) / 4); ++w)
        if (a[w] != b[w]) *differ = 1;
}

cudaError_t launch_rows_h(const MatCoef* coef, int n_rows, int bg, int* differ, cudaStream_t st) {
    const cudaError_t e = cudaMemsetAsync(differ, 0, sizeof(int), st);
    if (e != cudaSuccess || n_rows <= 0) return e;
    k_rows_h<<<(n_rows + 127) / 128, 128, 0, st>>>(coef, n_rows, bg, differ);
    return cudaGetLastError();
}

cudaError_t launch_slab_rows(const DeviceGrid& g, const MatCoef* coef, int n_rows, float* const kappa[6], float4* out,
                             cudaStream_t st) {
    const int L = max(g.pxn + g.pxp, max(g.pyn + g.pyp, g.pzn + g.pzp));
    if (n_rows <= 0 || L <= 0) return cudaSuccess;
    k_slab_rows<<<dim3((unsigned)((n_rows * L + 255) / 256), 3), 256, 0, st>>>(coef, g, n_rows, kappa[0], kappa[1], kappa[2], kappa[3],
                                                                              kappa[4], kappa[5], out);
    return cudaGetLastError();
}

cudaError_t launch_axis_tables(const DeviceGrid& g, float* const prof[18], float* const bg_curl[12], float4* const te[3],
                               float4* const th[3], cudaStream_t st) {
    const int ns[3] = {g.nx, g.ny, g.nz};
    for (int a = 0; a < 3; ++a) {
        float* const* P = prof + 6 * a;
        float* const* C = bg_curl + 4 * a;
        k_axis_table<<<(ns[a] + 127) / 128, 128, 0, st>>>(te[a], th[a], ns[a], P[0], P[1], P[2], P[3], C[0], C[1], C[2], C[3]);
    }
    return cudaGetLastError();
}

__global__ void k_fill(float* p, long long n, float v) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        p[q] = v;
}

cudaError_t launch_fill(float* p, long long n, float v, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    k_fill<<<(int)blocks, 256, 0, st>>>(p, n, v);
    return cudaGetLastError();
}

// The row padding of a field array (columns nx .. pitch-1 of every row) set to v.
__global__ void k_fill_padding(float* p, DeviceGrid g, float v) {
    const int w = g.pitch - g.nx;
    const long long n = (long long)w * g.ny * g.nz;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        p[(q / w) * g.pitch + g.nx + q % w] = v;
}

cudaError_t launch_fill_padding(float* p, const DeviceGrid& g, float v, cudaStream_t st) {
    const long long n = (long long)(g.pitch - g.nx) * g.ny * g.nz;
    if (n <= 0) return cudaSuccess;
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    k_fill_padding<<<(int)blocks, 256, 0, st>>>(p, g, v);
    return cudaGetLastError();
}

// setBrick (fdtdrav.h:1524-1571) on the material index: cells [is,ie) x [js,je) x [ks,ke).
__global__ void k_paint(uint8_t* mat, DeviceGrid g, int is, int js, int ks, int ie, int je, int ke, uint8_t v) {
    const int i = is + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = js + blockIdx.y * blockDim.y + threadIdx.y;
    const int k = ks + blockIdx.z;
    if (i < ie && j < je && k < ke) mat[(long long)k * g.plane + (long long)j * g.pitch + i] = v;
}

// Largest material index of the grid's cells (row padding excluded) into *out (atomicMax; *out
// starts at 0).
__global__ void k_index_max(const uint8_t* __restrict__ mat, DeviceGrid g, int* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    int v = 0;
    if (i < g.nx && j < g.ny)
        for (int k = blockIdx.z * kSetupPlanes, k1 = min(g.nz, k + kSetupPlanes); k < k1; ++k)
            v = max(v, (int)mat[(long long)k * g.plane + (long long)j * g.pitch + i]);
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0 && v > 0) atomicMax(out, v);
}

cudaError_t launch_index_max(const uint8_t* mat, const DeviceGrid& g, int* out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    const dim3 block(32, 8, 1), grid((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + kSetupPlanes - 1) / kSetupPlanes);
    k_index_max<<<grid, block, 0, st>>>(mat, g, out);
    return cudaGetLastError();
}

cudaError_t launch_paint(uint8_t* mat, const DeviceGrid& g, const int box[6], uint8_t value, cudaStream_t st) {
    const int is = box[0] < 0 ? 0 : box[0], js = box[1] < 0 ? 0 : box[1], ks = box[2] < 0 ? 0 : box[2];
    const int ie = box[3] > g.nx ? g.nx : box[3], je = box[4] > g.ny ? g.ny : box[4], ke = box[5] > g.nz ? g.nz : box[5];
    if (is >= ie || js >= je || ks >= ke) return cudaSuccess;
    dim3 block(32, 8, 1);
    dim3 grid((ie - is + 31) / 32, (je - js + 7) / 8, ke - ks);
    k_paint<<<grid, block, 0, st>>>(mat, g, is, js, ks, ie, je, ke, value);
    return cudaGetLastError();
}

}  // namespace fdtd

namespace fdtd {

// Node class (StepParams::cls): material id of nodes that take the fast path (interior, seven cells
// of one material below kUniformGeneral), kInterfaceNode for the other interior nodes,
// kUniformGeneral + m for the other nodes whose seven cells all hold material m, kGeneral
// otherwise. Lumped edges (k_class_lumped) and plates turn their nodes general afterwards.
// The seven cells are those the three E edge averages read, (i,j,k) (i-1,j,k) (i,j-1,k) (i,j,k-1)
// (i-1,j-1,k) (i-1,j,k-1) (i,j-1,k-1); the four cells of the H faces are among them.
// Nodes of the design region's edge box [dlo, dhi] get kDesignNode.
__device__ __forceinline__ void node_class(const uint8_t* __restrict__ mat, uint8_t* __restrict__ cls,
                                           const DeviceGrid& g, int4 dlo, int4 dhi, int i, int j, int k) {
    const long long n = (long long)k * g.plane + (long long)j * g.pitch + i;
    uint8_t c = kGeneral;
    // the seven cells as the general path reads them (cells outside the grid count as material 0)
    const long long R = g.pitch, P = g.plane;
    const int m0 = mat[n];
    const int mi = i > 0 ? mat[n - 1] : 0, mj = j > 0 ? mat[n - R] : 0, mk = k > 0 ? mat[n - P] : 0;
    const int mij = (i > 0 && j > 0) ? mat[n - 1 - R] : 0, mik = (i > 0 && k > 0) ? mat[n - 1 - P] : 0;
    const int mjk = (j > 0 && k > 0) ? mat[n - R - P] : 0;
    const bool uniform = mi == m0 && mj == m0 && mk == m0 && mij == m0 && mik == m0 && mjk == m0;
    const bool inner = interior(i, g.nx, g.pxn, g.pxp) && interior(j, g.ny, g.pyn, g.pyp) && interior(k, g.nz, g.pzn, g.pzp);
    if (uniform && inner && m0 < kUniformGeneral)
        c = (uint8_t)m0;  // fast path
    else if (inner)
        c = kInterfaceNode;  // table update with the coefficient row of its seven cells
    else if (uniform && m0 < kInterfaceNode - kUniformGeneral)
        c = (uint8_t)(kUniformGeneral + m0);  // general path without the cell-material loads
    if (i >= dlo.x && i <= dhi.x && j >= dlo.y && j <= dhi.y && k >= dlo.z && k <= dhi.z) c = kDesignNode;
    cls[n] = c;
}

// One CTA per 32 x 8 block of kSetupPlanes planes (one node per thread and plane): a CTA per
// block of one plane made the grid-sized setup kernels bound by launching CTAs.
__global__ void k_node_class(const uint8_t* __restrict__ mat, uint8_t* __restrict__ cls, DeviceGrid g, int4 dlo,
                             int4 dhi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.nx || j >= g.ny) return;
    for (int k = blockIdx.z * kSetupPlanes, k1 = min(g.nz, k + kSetupPlanes); k < k1; ++k)
        node_class(mat, cls, g, dlo, dhi, i, j, k);
}

// A node of the design edge box stays kDesignNode (an Ez lumped element may stand on the region's top
// face): its Ex and Ey take the design cells' eps_r, its Ez the lumped override, which the design kernels
// look for.
__global__ void k_class_lumped(uint8_t* cls, DeviceGrid g, const LumpedEdge* edges, int n_edges) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_edges) return;
    uint8_t& c = cls[(long long)edges[q].k * g.plane + (long long)edges[q].j * g.pitch + edges[q].i];
    if (c != kDesignNode) c = kGeneral;
}

__global__ void k_class_nodes(uint8_t* cls, DeviceGrid g, const int4* nodes, int n, uint8_t value) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) cls[(long long)nodes[q].z * g.plane + (long long)nodes[q].y * g.pitch + nodes[q].x] = value;
}

cudaError_t launch_class_nodes(const DeviceGrid& g, const int4* nodes, int n, int value, uint8_t* cls, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_class_nodes<<<(n + 127) / 128, 128, 0, st>>>(cls, g, nodes, n, (uint8_t)value);
    return cudaGetLastError();
}

cudaError_t launch_node_class(const DeviceGrid& g, const uint8_t* mat, const LumpedEdge* edges, int n_edges,
                              const int* design_box, uint8_t* cls, cudaStream_t st) {
    const int4 dlo = design_box ? make_int4(design_box[0], design_box[1], design_box[2], 0) : make_int4(1, 1, 1, 0);
    const int4 dhi = design_box ? make_int4(design_box[3], design_box[4], design_box[5], 0) : make_int4(0, 0, 0, 0);
    dim3 block(32, 8, 1);
    dim3 grid((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + kSetupPlanes - 1) / kSetupPlanes);
    k_node_class<<<grid, block, 0, st>>>(mat, cls, g, dlo, dhi);
    if (n_edges > 0) k_class_lumped<<<(n_edges + 127) / 128, 128, 0, st>>>(cls, g, edges, n_edges);
    return cudaGetLastError();
}

}  // namespace fdtd

namespace fdtd {

// Interface rows. Every kInterfaceNode and kGeneral node is keyed by its seven cell materials,
// packed one byte each in the order (i,j,k) (i-1,j,k) (i,j-1,k) (i,j,k-1) (i-1,j-1,k) (i-1,j,k-1)
// (i,j-1,k-1), cells outside the grid as material 0 (as the general path reads them). The
// distinct keys are collected in a hash set on the device (open addressing, linear probing), only
// they are sorted on the host, and each of the first kMaxInterfaceRows gets the coefficient row
// the general path would build for such a node (e_coef / h_coef: table entries where an edge's
// cells agree, the reference's averages otherwise), so an interior node's update is the table
// form with the same bits. Interior nodes whose key has no row take the general path, with the
// same bits too. The rows of nodes in CPML slabs or on boundary planes (classes kGeneral and
// kUniformGeneral + m) serve the kernels by row, which take the curl coefficients over kappa from
// the axis tables or SlabRows and apply the boundary rules themselves; the kernels by class keep their
// general path for those nodes. Lumped edges get rows of their own afterwards (special_row).
namespace {
__device__ __forceinline__ unsigned long long cell_key(const uint8_t* mat, const DeviceGrid& g, int i, int j, int k) {
    const long long R = g.pitch, P = g.plane, n = (long long)k * P + (long long)j * R + i;
    const unsigned long long m0 = mat[n], mi = i > 0 ? mat[n - 1] : 0, mj = j > 0 ? mat[n - R] : 0;
    const unsigned long long mk = k > 0 ? mat[n - P] : 0, mij = (i > 0 && j > 0) ? mat[n - 1 - R] : 0;
    const unsigned long long mik = (i > 0 && k > 0) ? mat[n - 1 - P] : 0, mjk = (j > 0 && k > 0) ? mat[n - R - P] : 0;
    return m0 | mi << 8 | mj << 16 | mk << 24 | mij << 32 | mik << 40 | mjk << 48;
}
constexpr unsigned long long kEmptyKey = ~0ull;  // keys use 56 bits
constexpr int kMaxProbes = 64;
__device__ __forceinline__ unsigned slot_of(unsigned long long key) {
    return (unsigned)((key * 0x9E3779B97F4A7C15ull) >> (64 - kIfaceTableBits));
}
// Slot of `key` in the set, or -1.
__device__ __forceinline__ int find_slot(const unsigned long long* __restrict__ table, unsigned long long key) {
    unsigned s = slot_of(key);
    for (int q = 0; q < kMaxProbes; ++q, s = (s + 1) & (kIfaceTableSize - 1)) {
        const unsigned long long v = table[s];
        if (v == key) return (int)s;
        if (v == kEmptyKey) return -1;
    }
    return -1;
}
}  // namespace

// Insert the key of every kInterfaceNode or kGeneral node into the set while it holds fewer than
// kIfaceTableSize / 2 keys (*filled counts them, a few more may land while it reaches that); a key
// that finds no room stays out (its nodes take the general path).
__device__ __forceinline__ void iface_insert(unsigned long long* table, int* filled, unsigned long long key) {
    unsigned s = slot_of(key);
    for (int q = 0; q < kMaxProbes; ++q, s = (s + 1) & (kIfaceTableSize - 1)) {
        const unsigned long long v = *(volatile unsigned long long*)(table + s);
        if (v == key) return;
        if (v != kEmptyKey) continue;
        if (*(volatile int*)filled >= kIfaceTableSize / 2) return;
        const unsigned long long old = atomicCAS(table + s, kEmptyKey, key);
        if (old == kEmptyKey) {
            atomicAdd(filled, 1);
            return;
        }
        if (old == key) return;
    }
}
__global__ void k_iface_insert(const uint8_t* __restrict__ cls, const uint8_t* __restrict__ mat, DeviceGrid g,
                               unsigned long long* table, int* filled) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.nx || j >= g.ny) return;
    for (int k = blockIdx.z * kSetupPlanes, k1 = min(g.nz, k + kSetupPlanes); k < k1; ++k) {
        const long long n = (long long)k * g.plane + (long long)j * g.pitch + i;
        if (cls[n] == kInterfaceNode || cls[n] == kGeneral) iface_insert(table, filled, cell_key(mat, g, i, j, k));
    }
}

// The keys held in the set, in slot order, to keys[atomicAdd(count)].
__global__ void k_iface_compact(const unsigned long long* __restrict__ table, unsigned long long* keys, int* count) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= kIfaceTableSize) return;
    const unsigned long long v = table[s];
    if (v != kEmptyKey) keys[atomicAdd(count, 1)] = v;
}

// slot_row[slot of sorted key q] = q for the rows kept.
__global__ void k_iface_slot_rows(const unsigned long long* __restrict__ table, const unsigned long long* __restrict__ keys,
                                  int n_keys, int* slot_row) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_keys) return;
    const int s = find_slot(table, keys[q]);
    if (s >= 0) slot_row[s] = q;
}

// Coefficient rows of every node (StepParams::rec): the material id of fast-path nodes and of
// kUniformGeneral + m nodes (m), the interface row of kInterfaceNode and kGeneral nodes whose key
// has one, and kRecGeneral | class for the rest. kInterfaceNode nodes without a row become
// kGeneral.
__device__ __forceinline__ void iface_row(uint8_t* __restrict__ cls, const uint8_t* __restrict__ mat, const DeviceGrid& g,
                                          const unsigned long long* __restrict__ table, const int* __restrict__ slot_row,
                                          uint16_t* __restrict__ rec, int i, int j, int k);
__global__ void k_iface_rows(uint8_t* __restrict__ cls, const uint8_t* __restrict__ mat, DeviceGrid g,
                             const unsigned long long* __restrict__ table, const int* __restrict__ slot_row,
                             uint16_t* __restrict__ rec, int* __restrict__ edge_mat) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (j >= g.ny) return;  // i < g.pitch: the blocks cover whole rows
    for (int k = blockIdx.z * kSetupPlanes, k1 = min(g.nz, k + kSetupPlanes); k < k1; ++k) {
        if (i < g.nx) {
            iface_row(cls, mat, g, table, slot_row, rec, i, j, k);
            const int r = rec[(long long)k * g.plane + (long long)j * g.pitch + i];
            if (r != 0 && r < kRecGeneral && (i == 0 || j == 0 || k == 0 || in_slab(i, g.nx, g.pxn, g.pxp) ||
                                              in_slab(j, g.ny, g.pyn, g.pyp) || in_slab(k, g.nz, g.pzn, g.pzp)))
                *edge_mat = 1;
        } else rec[(long long)k * g.plane + (long long)j * g.pitch + i] = 0;  // row padding: the sweep's tiles read it
    }
}
__device__ __forceinline__ void iface_row(uint8_t* __restrict__ cls, const uint8_t* __restrict__ mat, const DeviceGrid& g,
                                          const unsigned long long* __restrict__ table, const int* __restrict__ slot_row,
                                          uint16_t* __restrict__ rec, int i, int j, int k) {
    const long long n = (long long)k * g.plane + (long long)j * g.pitch + i;
    int c = cls[n];
    int r = kRecGeneral | c;
    if (c < kUniformGeneral) {
        r = c;
    } else if (c < kInterfaceNode) {
        r = c - kUniformGeneral;
    } else if (c == kInterfaceNode || c == kGeneral) {
        const int s = find_slot(table, cell_key(mat, g, i, j, k));
        const int row = s >= 0 ? slot_row[s] : -1;
        if (row >= 0) {
            r = kFirstInterfaceRow + row;
        } else if (c == kInterfaceNode) {
            cls[n] = kGeneral;
            r = kRecGeneral | kGeneral;
        }
    }
    rec[n] = (uint16_t)r;
}

// Lumped edges keep the general path in every schedule (their E update is the lumped override), in the
// design edge box as its nodes.
__global__ void k_rec_general(uint16_t* rec, DeviceGrid g, const LumpedEdge* edges, int n_edges, const uint8_t* cls) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_edges) return;
    const long long n = (long long)edges[q].k * g.plane + (long long)edges[q].j * g.pitch + edges[q].i;
    rec[n] = (uint16_t)(kRecGeneral | (cls[n] == kDesignNode ? kDesignNode : kGeneral));
}

// The nodes of probes inside a CPML slab too: the general path samples them before the CPML
// correction. The classes, which the per-node kernels go by, stay: those kernels sample themselves.
__global__ void k_rec_probes(uint16_t* rec, DeviceGrid g, const Probe* probes, int n) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const Probe& r = probes[q];
    if (!in_slab(r.i, g.nx, g.pxn, g.pxp) && !in_slab(r.j, g.ny, g.pyn, g.pyp) && !in_slab(r.k, g.nz, g.pzn, g.pzp)) return;
    const long long v = (long long)r.k * g.plane + (long long)r.j * g.pitch + r.i;
    if (rec[v] < kRecGeneral) rec[v] = (uint16_t)(kRecGeneral | kGeneral);
}

cudaError_t launch_rec_probes(const DeviceGrid& g, const Probe* probes, int n, uint16_t* rec, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_rec_probes<<<(n + 127) / 128, 128, 0, st>>>(rec, g, probes, n);
    return cudaGetLastError();
}

// The plate nodes inside a CPML slab, where the slab rows are missing: the kernels by row leave such a
// node's row alone then, and k_plate_e goes by the general mark.
__global__ void k_rec_slab_plates(uint16_t* rec, DeviceGrid g, const int4* nodes, int n) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int4 v = nodes[q];
    if (!in_slab(v.x, g.nx, g.pxn, g.pxp) && !in_slab(v.y, g.ny, g.pyn, g.pyp) && !in_slab(v.z, g.nz, g.pzn, g.pzp)) return;
    uint16_t& r = rec[(long long)v.z * g.plane + (long long)v.y * g.pitch + v.x];
    if (r < kRecGeneral) r = (uint16_t)(kRecGeneral | kPlateNode);
}

cudaError_t launch_rec_slab_plates(const DeviceGrid& g, const int4* nodes, int n, uint16_t* rec, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_rec_slab_plates<<<(n + 127) / 128, 128, 0, st>>>(rec, g, nodes, n);
    return cudaGetLastError();
}

// How many of the listed nodes take the general path.
__global__ void k_count_general(const uint16_t* rec, DeviceGrid g, const int4* nodes, int n, int* count) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n && rec[(long long)nodes[q].z * g.plane + (long long)nodes[q].y * g.pitch + nodes[q].x] >= kRecGeneral) atomicAdd(count, 1);
}

cudaError_t launch_count_general(const DeviceGrid& g, const uint16_t* rec, const int4* nodes, int n, int* count, cudaStream_t st) {
    const cudaError_t e = cudaMemsetAsync(count, 0, sizeof(int), st);
    if (e != cudaSuccess || n <= 0) return e;
    k_count_general<<<(n + 127) / 128, 128, 0, st>>>(rec, g, nodes, n, count);
    return cudaGetLastError();
}

cudaError_t launch_rec_general(const DeviceGrid& g, const LumpedEdge* edges, int n_edges, const uint8_t* cls, uint16_t* rec,
                               cudaStream_t st) {
    if (n_edges <= 0) return cudaSuccess;
    k_rec_general<<<(n_edges + 127) / 128, 128, 0, st>>>(rec, g, edges, n_edges, cls);
    return cudaGetLastError();
}

namespace {
struct DesignBox {
    int d[6];
    __host__ __device__ long long volume() const { return (long long)(d[3] - d[0] + 1) * (d[4] - d[1] + 1) * (d[5] - d[2] + 1); }
};
// Node e of the box, x fastest.
__device__ __forceinline__ int3 design_node(const DesignBox& b, long long e) {
    const int bx = b.d[3] - b.d[0] + 1, by = b.d[4] - b.d[1] + 1;
    return make_int3(b.d[0] + (int)(e % bx), b.d[1] + (int)((e / bx) % by), b.d[2] + (int)(e / ((long long)bx * by)));
}
DesignBox design_box(const int* d) { return DesignBox{{d[0], d[1], d[2], d[3], d[4], d[5]}}; }
}  // namespace

__global__ void k_design_insert(const uint8_t* __restrict__ cls, const uint8_t* __restrict__ mat, DeviceGrid g, DesignBox b,
                                unsigned long long* table, int* filled) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= b.volume()) return;
    const int3 v = design_node(b, e);
    if (cls[(long long)v.z * g.plane + (long long)v.y * g.pitch + v.x] == kDesignNode)
        iface_insert(table, filled, cell_key(mat, g, v.x, v.y, v.z));
}
__global__ void k_design_rows(const uint8_t* __restrict__ cls, const uint8_t* __restrict__ mat, DeviceGrid g, DesignBox b,
                              const unsigned long long* __restrict__ table, const int* __restrict__ slot_row, int first, uint16_t* rec) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= b.volume()) return;
    const int3 v = design_node(b, e);
    const long long n = (long long)v.z * g.plane + (long long)v.y * g.pitch + v.x;
    if (cls[n] != kDesignNode) return;
    const int s = find_slot(table, cell_key(mat, g, v.x, v.y, v.z)), row = s >= 0 ? slot_row[s] : -1;
    if (row >= 0) rec[n] = (uint16_t)(first + row);
}
// The general path's coefficients (e_coef with design cells), once instead of in every step.
__global__ void k_design_coefs(const __grid_constant__ StepParams p, DesignBox b, float4* out) {
    const long long ne = b.volume(), e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int3 v = design_node(b, e);
    const unsigned long long key = cell_key(p.mat, p.g, v.x, v.y, v.z);
    const int m0 = (int)(key & 0xff), mi = (int)((key >> 8) & 0xff), mj = (int)((key >> 16) & 0xff);
    const int mk = (int)((key >> 24) & 0xff), mij = (int)((key >> 32) & 0xff), mik = (int)((key >> 40) & 0xff);
    const int mjk = (int)((key >> 48) & 0xff);
    const Coef3 c[3] = {e_coef<true>(p, 0, m0 == mj && m0 == mk && m0 == mjk, m0, mj, mk, mjk, v.x, v.y, v.z),
                        e_coef<true>(p, 1, m0 == mi && m0 == mk && m0 == mik, m0, mi, mk, mik, v.x, v.y, v.z),
                        e_coef<true>(p, 2, m0 == mi && m0 == mj && m0 == mij, m0, mi, mj, mij, v.x, v.y, v.z)};
    for (int q = 0; q < 3; ++q) out[q * ne + e] = make_float4(c[q].a, c[q].bp, c[q].bm, 0.f);
}

cudaError_t launch_design_set(const DeviceGrid& g, const int* dbox, const uint8_t* cls, const uint8_t* mat, unsigned long long* table,
                              int* counters, unsigned long long* keys, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(table, 0xff, sizeof(unsigned long long) * kIfaceTableSize, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(counters, 0, 2 * sizeof(int), st);
    if (e != cudaSuccess) return e;
    const DesignBox b = design_box(dbox);
    k_design_insert<<<(unsigned)((b.volume() + 255) / 256), 256, 0, st>>>(cls, mat, g, b, table, counters);
    k_iface_compact<<<kIfaceTableSize / 256, 256, 0, st>>>(table, keys, counters + 1);
    return cudaGetLastError();
}

cudaError_t launch_design_rows(const DeviceGrid& g, const int* dbox, const uint8_t* cls, const uint8_t* mat,
                               const unsigned long long* table, const unsigned long long* keys, int n_keys, int first, int* slot_row,
                               uint16_t* rec, cudaStream_t st) {
    const cudaError_t e = cudaMemsetAsync(slot_row, 0xff, sizeof(int) * kIfaceTableSize, st);
    if (e != cudaSuccess || n_keys <= 0) return e;
    const DesignBox b = design_box(dbox);
    k_iface_slot_rows<<<(n_keys + 127) / 128, 128, 0, st>>>(table, keys, n_keys, slot_row);
    k_design_rows<<<(unsigned)((b.volume() + 255) / 256), 256, 0, st>>>(cls, mat, g, b, table, slot_row, first, rec);
    return cudaGetLastError();
}

__global__ void k_rec_design_general(const uint8_t* __restrict__ cls, DeviceGrid g, DesignBox b, uint16_t* rec) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= b.volume()) return;
    const int3 v = design_node(b, e);
    const long long n = (long long)v.z * g.plane + (long long)v.y * g.pitch + v.x;
    if (cls[n] == kDesignNode) rec[n] = (uint16_t)(kRecGeneral | kDesignNode);
}

cudaError_t launch_rec_design_general(const DeviceGrid& g, const int* dbox, const uint8_t* cls, uint16_t* rec, cudaStream_t st) {
    const DesignBox b = design_box(dbox);
    k_rec_design_general<<<(unsigned)((b.volume() + 255) / 256), 256, 0, st>>>(cls, g, b, rec);
    return cudaGetLastError();
}

cudaError_t launch_design_coefs(const StepParams& p, float4* dcoef, cudaStream_t st) {
    const DesignBox b = design_box(p.dbox);
    k_design_coefs<<<(unsigned)((b.volume() + 127) / 128), 128, 0, st>>>(p, b, dcoef);
    return cudaGetLastError();
}

// Coefficient row kFirstInterfaceRow + q of unique key q, from the material rows and properties.
__global__ void k_iface_coefs(const __grid_constant__ StepParams p, const unsigned long long* __restrict__ keys,
                              int n_keys, MatCoef* coef) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_keys) return;
    const unsigned long long key = keys[q];
    const int m0 = (int)(key & 0xff), mi = (int)((key >> 8) & 0xff), mj = (int)((key >> 16) & 0xff);
    const int mk = (int)((key >> 24) & 0xff), mij = (int)((key >> 32) & 0xff), mik = (int)((key >> 40) & 0xff);
    const int mjk = (int)((key >> 48) & 0xff);
    // position-free coefficients: no design cells (those nodes are kDesignNode); CPML kappa and
    // boundary faces are the kernels' own
    const Coef3 ex = e_coef(p, 0, m0 == mj && m0 == mk && m0 == mjk, m0, mj, mk, mjk, 1, 1, 1);
    const Coef3 ey = e_coef(p, 1, m0 == mi && m0 == mk && m0 == mik, m0, mi, mk, mik, 1, 1, 1);
    const Coef3 ez = e_coef(p, 2, m0 == mi && m0 == mj && m0 == mij, m0, mi, mj, mij, 1, 1, 1);
    const Coef3 hx = h_coef(p, 0, false, m0 == mi, m0, mi);
    const Coef3 hy = h_coef(p, 1, false, m0 == mj, m0, mj);
    const Coef3 hz = h_coef(p, 2, false, m0 == mk, m0, mk);
    MatCoef c;
    c.e[0] = make_float4(ex.a, ex.bp, ex.bm, 0.f);
    c.e[1] = make_float4(ey.a, ey.bp, ey.bm, 0.f);
    c.e[2] = make_float4(ez.a, ez.bp, ez.bm, 0.f);
    c.h[0] = make_float4(hx.a, hx.bp, hx.bm, 0.f);
    c.h[1] = make_float4(hy.a, hy.bp, hy.bm, 0.f);
    c.h[2] = make_float4(hz.a, hz.bp, hz.bm, 0.f);
    coef[kFirstInterfaceRow + q] = c;
}

cudaError_t launch_iface_set(const DeviceGrid& g, const uint8_t* cls, const uint8_t* mat, unsigned long long* table,
                             int* counters, unsigned long long* keys, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(table, 0xff, sizeof(unsigned long long) * kIfaceTableSize, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(counters, 0, 2 * sizeof(int), st);
    if (e != cudaSuccess) return e;
    const dim3 block(32, 8, 1), grid((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + kSetupPlanes - 1) / kSetupPlanes);
    k_iface_insert<<<grid, block, 0, st>>>(cls, mat, g, table, counters);
    k_iface_compact<<<kIfaceTableSize / 256, 256, 0, st>>>(table, keys, counters + 1);
    return cudaGetLastError();
}

cudaError_t launch_iface_rows(const DeviceGrid& g, uint8_t* cls, const uint8_t* mat, const unsigned long long* table,
                              const unsigned long long* keys, int n_keys, int* slot_row, uint16_t* rec, int* edge_mat,
                              cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(slot_row, 0xff, sizeof(int) * kIfaceTableSize, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(edge_mat, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    if (n_keys > 0) k_iface_slot_rows<<<(n_keys + 127) / 128, 128, 0, st>>>(table, keys, n_keys, slot_row);
    const dim3 block(32, 8, 1), grid((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + kSetupPlanes - 1) / kSetupPlanes);
    k_iface_rows<<<grid, block, 0, st>>>(cls, mat, g, table, slot_row, rec, edge_mat);
    return cudaGetLastError();
}

cudaError_t launch_iface_coefs(const StepParams& p, const unsigned long long* keys, int n_keys, MatCoef* coef,
                               cudaStream_t st) {
    if (n_keys <= 0) return cudaSuccess;
    k_iface_coefs<<<(n_keys + 127) / 128, 128, 0, st>>>(p, keys, n_keys, coef);
    return cudaGetLastError();
}

// The coefficient row of a node with plate-covered or lumped edges: as e_update builds its
// coefficients (cell averages, plate conductivity, lumped override), and its H faces'. Interior
// position rules (CPML kappa, default entries of the low walls) are the sweep's. cezj: the source's.
namespace {
__device__ __forceinline__ MatCoef special_row(const StepParams& p, int i, int j, int k, float& cezj) {
    const DeviceGrid& g = p.g;
    const unsigned long long key = cell_key(p.mat, g, i, j, k);
    const int m0 = (int)(key & 0xff), mi = (int)((key >> 8) & 0xff), mj = (int)((key >> 16) & 0xff);
    const int mk = (int)((key >> 24) & 0xff), mij = (int)((key >> 32) & 0xff), mik = (int)((key >> 40) & 0xff);
    const int mjk = (int)((key >> 48) & 0xff);
    Coef3 e[3] = {e_coef(p, 0, m0 == mj && m0 == mk && m0 == mjk, m0, mj, mk, mjk, i, j, k),
                  e_coef(p, 1, m0 == mi && m0 == mk && m0 == mik, m0, mi, mk, mik, i, j, k),
                  e_coef(p, 2, m0 == mi && m0 == mj && m0 == mij, m0, mi, mj, mij, i, j, k)};
    if (plane_has_plate(p, k)) {
        Coef3 pc[3];
        const int hit = e_plate(&p, i, j, k, m0, mi, mj, mk, mij, mik, mjk, pc);
        for (int c = 0; c < 3; ++c)
            if (hit >> c & 1) e[c] = pc[c];
    }
    const LumpedEdge* Lx = find_lumped(p, i, j, k, 0);
    const LumpedEdge* Lz = find_lumped(p, i, j, k, 2);
    if (Lx) e[0] = Coef3{Lx->ceze, Lx->cezhy, Lx->cezhx};
    if (Lz) e[2] = Coef3{Lz->ceze, Lz->cezhy, Lz->cezhx};
    cezj = Lz && Lz->source >= 0 ? Lz->cezj : 0.f;
    const Coef3 h[3] = {h_coef(p, 0, false, m0 == mi, m0, mi), h_coef(p, 1, false, m0 == mj, m0, mj),
                        h_coef(p, 2, false, m0 == mk, m0, mk)};
    MatCoef r;
    for (int c = 0; c < 3; ++c) {
        r.e[c] = make_float4(e[c].a, e[c].bp, e[c].bm, 0.f);
        r.h[c] = make_float4(h[c].a, h[c].bp, h[c].bm, 0.f);
    }
    return r;
}
__device__ __forceinline__ unsigned long long special_key(const MatCoef& r, float cezj, int source) {
    unsigned long long h = 0x9E3779B97F4A7C15ull * (unsigned)(source + 2);
    const unsigned* w = reinterpret_cast<const unsigned*>(&r);
    for (int q = 0; q < (int)(sizeof(MatCoef) / 4); ++q) {  // splitmix-style mixing of each word
        h = (h ^ w[q]) * 0xBF58476D1CE4E5B9ull;
        h ^= h >> 29;
    }
    h = (h ^ __float_as_uint(cezj)) * 0x94D049BB133111EBull;
    h ^= h >> 32;
    h &= ~(3ull << 62);  // bit 62 stays clear, so that no key equals kEmptyKey
    return source >= 0 ? h | 1ull << 63 : h;
}
}  // namespace

__global__ void k_special_set(const __grid_constant__ StepParams p, const int4* __restrict__ nodes, int n,
                              unsigned long long* table, int* filled) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int4 v = nodes[q];
    float cezj;
    const MatCoef r = special_row(p, v.x, v.y, v.z, cezj);
    iface_insert(table, filled, special_key(r, cezj, v.w));
}
// write: the rows; otherwise every node's entry of rec, checked against the row that was written
// (several nodes of a key write equal rows unless their hashes collide).
__global__ void k_special_rows(const __grid_constant__ StepParams p, const int4* __restrict__ nodes, int n,
                               const unsigned long long* __restrict__ table, const int* __restrict__ slot_row, int first,
                               int n_plain, MatCoef* coef, SrcRow* src, uint16_t* rec, bool write) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int4 v = nodes[q];
    float cezj;
    const MatCoef r = special_row(p, v.x, v.y, v.z, cezj);
    const int s = find_slot(table, special_key(r, cezj, v.w));
    const int row = s >= 0 ? slot_row[s] : -1;
    if (row < 0) return;  // no room: the node stays general
    if (write) {
        coef[first + row] = r;
        if (v.w >= 0) src[row - n_plain] = SrcRow{cezj, v.w};
        return;
    }
    const unsigned* a = reinterpret_cast<const unsigned*>(&r);
    const unsigned* b = reinterpret_cast<const unsigned*>(coef + first + row);
    bool same = v.w < 0 || (src[row - n_plain].source == v.w && __float_as_uint(src[row - n_plain].cezj) == __float_as_uint(cezj));
    for (int w = 0; w < (int)(sizeof(MatCoef) / 4); ++w) same = same && a[w] == b[w];
    if (same) rec[(long long)v.z * p.g.plane + (long long)v.y * p.g.pitch + v.x] = (uint16_t)(first + row);
}

// Row first + q for node q (nodes with a source from n_plain on).
__global__ void k_special_each(const __grid_constant__ StepParams p, const int4* __restrict__ nodes, int n, int n_plain,
                               int first, MatCoef* coef, SrcRow* src, uint16_t* rec) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int4 v = nodes[q];
    float cezj;
    coef[first + q] = special_row(p, v.x, v.y, v.z, cezj);
    if (q >= n_plain) src[q - n_plain] = SrcRow{cezj, v.w};
    rec[(long long)v.z * p.g.plane + (long long)v.y * p.g.pitch + v.x] = (uint16_t)(first + q);
}

cudaError_t launch_special_each(const StepParams& p, const int4* nodes, int n, int n_plain, int first, MatCoef* coef,
                                SrcRow* src, uint16_t* rec, cudaStream_t st) {
    k_special_each<<<(n + 127) / 128, 128, 0, st>>>(p, nodes, n, n_plain, first, coef, src, rec);
    return cudaGetLastError();
}

cudaError_t launch_special_set(const StepParams& p, const int4* nodes, int n, unsigned long long* table, int* counters,
                               unsigned long long* keys, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(table, 0xff, sizeof(unsigned long long) * kIfaceTableSize, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(counters, 0, 2 * sizeof(int), st);
    if (e != cudaSuccess) return e;
    k_special_set<<<(n + 127) / 128, 128, 0, st>>>(p, nodes, n, table, counters);
    k_iface_compact<<<kIfaceTableSize / 256, 256, 0, st>>>(table, keys, counters + 1);
    return cudaGetLastError();
}

cudaError_t launch_special_rows(const StepParams& p, const int4* nodes, int n, const unsigned long long* table,
                                const unsigned long long* keys, int n_keys, int n_plain, int first, int* slot_row,
                                MatCoef* coef, SrcRow* src, uint16_t* rec, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(slot_row, 0xff, sizeof(int) * kIfaceTableSize, st);
    if (e != cudaSuccess || n_keys <= 0) return e;
    k_iface_slot_rows<<<(n_keys + 127) / 128, 128, 0, st>>>(table, keys, n_keys, slot_row);
    for (bool write : {true, false})
        k_special_rows<<<(n + 127) / 128, 128, 0, st>>>(p, nodes, n, table, slot_row, first, n_plain, coef, src, rec, write);
    return cudaGetLastError();
}

}  // namespace fdtd
