// Discrete adjoint of the Yee step (no reference counterpart; the reference has no gradient).
//
// The forward step is linear in the state (E, H, CPML memory psi): calc_e maps (E, H, psi_E) to
// (E', psi_E'), then calc_h maps (H, E', psi_H) to (H', psi_H'). The adjoint state lambda holds
// dJ/d(state); one reverse step applies the transposes in reverse order:
//   k_adj_h  (transpose of calc_h) and then
//   k_adj_e  (transpose of calc_e, plus the figure-of-merit source and the design gradient).
// The curl operators are transposed in gather form: each kernel writes, per node and component,
// the two contributions its derivative terms send to the other field (arrays G_H and G_E, zero for
// components the update masks keep fixed), and the next kernel gathers them from the neighbours.
// No atomics; each node owns its lambda and its CPML adjoint memory. The coefficients are rebuilt
// exactly as e_update / h_update build them (material table, edge averages, design cells, CPML
// kappa division, lumped overrides), so the adjoint is the transpose of the FP32 update.
//
// Figure of merit J = sum_m dt * Ez(p)^2 with Ez sampled after step m's E update: its derivative
// 2 dt Ez_p(m) enters lambda_Ez(p) at reverse step m. The gradient with respect to the eps_r of a
// design cell collects, over the steps and the twelve E edges around the cell, lambda_e *
// dE_e'/d(eps_avg) / 4, where for an edge update E' = a E + c1 d1 + c2 d2 with
// den = 2 eps_avg eps0 + dt sigma_avg:
//   da/deps = 4 eps0 dt sigma / den^2,  d(c1, c2)/deps = -(2 eps0 / den) (c1, c2),
// so dE'/deps = da/deps * E - (2 eps0 / den) * (E' - a E), from the saved design-region E of the
// step (edges of the design region carry no CPML term and no lumped element).
#include "yee_common.cuh"
#include "adjoint.h"
#include "tma.cuh"

namespace fdtd {

namespace {

// One CPML term of an adjoint component: memory slot, profile values and psi coefficient.
struct PsiTerm {
    float* mem;  // adjoint psi entry, NULL when the node is outside the slab
    float b, a, cpsi;
    float old;   // its value before this step
};
// The term of adjoint psi entry `mem`, its old value read here: where the term is built, not
// where it is applied (3-4 % off the reverse step at 128^3).
__device__ __forceinline__ PsiTerm psi_term(float* mem, float b, float a, float cpsi) {
    return PsiTerm{mem, b, a, cpsi, *mem};
}

// Transpose of one component update v' = a v + c1 d1 + c2 d2 (+ psi terms t1 on d1, t2 on d2):
// returns the new lambda of the component and the contributions g1, g2 to the fields of d1, d2.
__device__ __forceinline__ float adj_comp(float L, float a, float c1, float c2, const PsiTerm& t1, const PsiTerm& t2,
                                          float& g1, float& g2) {
    g1 = c1 * L;
    g2 = c2 * L;
    if (t1.mem) {
        const float mm = __fmaf_rn(t1.cpsi, L, t1.old);
        *t1.mem = t1.b * mm;
        g1 = __fmaf_rn(t1.a, mm, g1);
    }
    if (t2.mem) {
        const float mm = __fmaf_rn(t2.cpsi, L, t2.old);
        *t2.mem = t2.b * mm;
        g2 = __fmaf_rn(t2.a, mm, g2);
    }
    return a * L;
}

__device__ __forceinline__ long long node(const DeviceGrid& g, int i, int j, int k) {
    return (long long)k * g.plane + (long long)j * g.pitch + i;
}

}  // namespace

// ---- transpose of calc_h (h_update) -------------------------------------------------------
// G_E slots (written by k_adj_e): 0 Ex->Hz, 1 Ex->Hy, 2 Ey->Hx, 3 Ey->Hz, 4 Ez->Hy, 5 Ez->Hx.
// G_H slots (written here):        0 Hx->Ey, 1 Hx->Ez, 2 Hy->Ez, 3 Hy->Ex, 4 Hz->Ex, 5 Hz->Ey.
// CTAs of 256 per SM: at 128^3 the 192-step gradient took 30.1 ms with 4 (64 registers, no spills), 30.7 with
// 5 and 31.1 with 6.
constexpr int kAdjCtas = 4;
// General path of k_adj_h, out of line.
__device__ __noinline__ void adj_h_general(const StepParams* pp, const AdjState* pa, const PsiSet* pps, int i, int j, int k, float lx,
                                           float ly, float lz) {
    const StepParams& p = *pp;
    const AdjState& a = *pa;
    const PsiSet& psa = *pps;
    const DeviceGrid& g = p.g;
    const long long P = g.plane, R = g.pitch, n = node(g, i, j, k);
    const int c = p.cls[n];
    const bool kp = k < g.nz - 1, jp = j < g.ny - 1, ip = i < g.nx - 1;
    const uint8_t* mat = p.mat;
    const bool one = c >= kUniformGeneral && c < kInterfaceNode;  // seven cells of one material, given by the class
    const int m0 = one ? c - kUniformGeneral : mat[n];
    const int mi = one ? m0 : i > 0 ? mat[n - 1] : 0, mj = one ? m0 : j > 0 ? mat[n - R] : 0;
    const int mk = one ? m0 : k > 0 ? mat[n - P] : 0;
    const bool hx_m = jp && kp, hy_m = ip && kp, hz_m = ip && jp;
    const bool xs = in_slab(i, g.nx, g.pxn, g.pxp), ys = in_slab(j, g.ny, g.pyn, g.pyp), zs = in_slab(k, g.nz, g.pzn, g.pzp);
    const int bg = p.bg.mat;
    const bool ux = m0 == mi, uy = m0 == mj, uz = m0 == mk;
    const bool on_bg = m0 == bg;
    const Coef3 cx = h_coef(p, 0, i == 0, ux, m0, mi);
    const Coef3 cy = h_coef(p, 1, j == 0, uy, m0, mj);
    const Coef3 cz = h_coef(p, 2, k == 0, uz, m0, mk);
    const bool bx = i != 0 && ux && on_bg, by = j != 0 && uy && on_bg, bz = k != 0 && uz && on_bg;
    const BgCurl& B = p.bg;
    int side;
    float g0 = 0.f, g1 = 0.f, g2 = 0.f, g3 = 0.f, g4 = 0.f, g5 = 0.f;
    if (hx_m) {  // Hx: c1 on dEy_k (z CPML), c2 on dEz_j (y CPML)
        PsiTerm t1{nullptr, 0, 0, 0, 0}, t2{nullptr, 0, 0, 0, 0};
        if (zs) { const int q = psi_off_z(g, i, j, k, side); t1 = psi_term(psa.f[4 + side].h[0] + q, p.bmz[k], p.amz[k], __fmul_rn(cx.bp, g.dz)); }
        if (ys) { const int q = psi_off_y(g, i, j, k, side); t2 = psi_term(psa.f[2 + side].h[0] + q, p.bmy[j], p.amy[j], __fmul_rn(cx.bm, g.dy)); }
        const float c1 = zs ? kdiv(cx.bp, bx, B.h[2][0], p.kmz, k) : cx.bp;
        const float c2 = ys ? kdiv(cx.bm, bx, B.h[1][0], p.kmy, j) : cx.bm;
        lx = adj_comp(lx, cx.a, c1, c2, t1, t2, g0, g1);
    }
    if (hy_m) {  // Hy: c1 on dEz_i (x CPML), c2 on dEx_k (z CPML)
        PsiTerm t1{nullptr, 0, 0, 0, 0}, t2{nullptr, 0, 0, 0, 0};
        if (xs) { const int q = psi_off_x(g, i, j, k, side); t1 = psi_term(psa.f[side].h[0] + q, p.bmx[i], p.amx[i], __fmul_rn(cy.bp, g.dx)); }
        if (zs) { const int q = psi_off_z(g, i, j, k, side); t2 = psi_term(psa.f[4 + side].h[1] + q, p.bmz[k], p.amz[k], __fmul_rn(cy.bm, g.dz)); }
        const float c1 = xs ? kdiv(cy.bp, by, B.h[0][0], p.kmx, i) : cy.bp;
        const float c2 = zs ? kdiv(cy.bm, by, B.h[2][1], p.kmz, k) : cy.bm;
        ly = adj_comp(ly, cy.a, c1, c2, t1, t2, g2, g3);
    }
    if (hz_m) {  // Hz: c1 on dEx_j (y CPML), c2 on dEy_i (x CPML)
        PsiTerm t1{nullptr, 0, 0, 0, 0}, t2{nullptr, 0, 0, 0, 0};
        if (ys) { const int q = psi_off_y(g, i, j, k, side); t1 = psi_term(psa.f[2 + side].h[1] + q, p.bmy[j], p.amy[j], __fmul_rn(cz.bp, g.dy)); }
        if (xs) { const int q = psi_off_x(g, i, j, k, side); t2 = psi_term(psa.f[side].h[1] + q, p.bmx[i], p.amx[i], __fmul_rn(cz.bm, g.dx)); }
        const float c1 = ys ? kdiv(cz.bp, bz, B.h[1][1], p.kmy, j) : cz.bp;
        const float c2 = xs ? kdiv(cz.bm, bz, B.h[0][1], p.kmx, i) : cz.bm;
        lz = adj_comp(lz, cz.a, c1, c2, t1, t2, g4, g5);
    }
    a.l[3][n] = lx; a.l[4][n] = ly; a.l[5][n] = lz;
    a.gh[0][n] = g0; a.gh[1][n] = g1; a.gh[2][n] = g2; a.gh[3][n] = g3; a.gh[4][n] = g4; a.gh[5][n] = g5;
}

// The CPML terms of a node on one axis: its face and offset there, the two old values.
struct AdjSlab {
    int face, q, l;  // l: the slab plane (SlabRows)
    float old0, old1;
};
template <bool kE>
__device__ __forceinline__ AdjSlab adj_slab(const DeviceGrid& g, const PsiSet& psa, int axis, int i, int j, int k) {
    AdjSlab s;
    int side;
    s.q = axis == 0 ? psi_off_x(g, i, j, k, side) : axis == 1 ? psi_off_y(g, i, j, k, side) : psi_off_z(g, i, j, k, side);
    s.face = 2 * axis + side;
    const int at = axis == 0 ? i : axis == 1 ? j : k, n = axis == 0 ? g.nx : axis == 1 ? g.ny : g.nz;
    const int pn = axis == 0 ? g.pxn : axis == 1 ? g.pyn : g.pzn, pp = axis == 0 ? g.pxp : axis == 1 ? g.pyp : g.pzp;
    s.l = side ? at - (n - pp) + pn : at;
    const PsiFace& f = psa.f[s.face];
    s.old0 = (kE ? f.e[0] : f.h[0])[s.q];
    s.old1 = (kE ? f.e[1] : f.h[1])[s.q];
    return s;
}
// One term of adj_comp: memory v' = b (v + f L), contribution g + a (v + f L). t: {b, a}; f: the factor.
__device__ __forceinline__ float adj_psi(float* mem, const float2& t, float f, float old, float L, float g) {
    const float mm = __fmaf_rn(f, L, old);
    *mem = t.x * mm;
    return __fmaf_rn(t.y, mm, g);
}
__device__ __forceinline__ float2 lo2(const float4* t) { return __ldg(reinterpret_cast<const float2*>(t)); }
__device__ __forceinline__ float2 hi2(const float4* t) { return __ldg(reinterpret_cast<const float2*>(t) + 1); }

// By coefficient row like the two-pass kernels (node_rows.cuh): the background's coefficients are constants,
// a slab's come from its axis' table or the slab row table, other rows' from the row table; the rest
// is called out of line. At 128^3 bound by L2: a pass moves 18 floats a node and the gathers' neighbours,
// 300 MB in 33 us, of a 151 MB state that does not quite stay there.
template <typename Idx>
__global__ void __launch_bounds__(256, kAdjCtas) k_adj_h(const __grid_constant__ StepParams p, const __grid_constant__ AdjState a,
                                               const __grid_constant__ PsiSet psa) {
    grid_dependency_wait();
    grid_launch_dependents();
    const DeviceGrid& g = p.g;
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= g.nx || j >= g.ny) return;
    const Idx P = (Idx)g.plane, R = (Idx)g.pitch, n = (Idx)k * P + (Idx)j * R + (Idx)i;
    const bool kp = k < g.nz - 1, jp = j < g.ny - 1, ip = i < g.nx - 1;
    const int c = p.rec[n];
    // finish the transpose of the previous reverse step's calc_e: gather G_E
    float lx = a.l[3][n] + a.ge[2][n] - (kp ? a.ge[2][n + P] : 0.f) + a.ge[5][n] - (jp ? a.ge[5][n + R] : 0.f);
    float ly = a.l[4][n] + a.ge[1][n] - (kp ? a.ge[1][n + P] : 0.f) + a.ge[4][n] - (ip ? a.ge[4][n + 1] : 0.f);
    float lz = a.l[5][n] + a.ge[0][n] - (jp ? a.ge[0][n + R] : 0.f) + a.ge[3][n] - (ip ? a.ge[3][n + 1] : 0.f);
    const bool xs = in_slab(i, g.nx, g.pxn, g.pxp), ys = in_slab(j, g.ny, g.pyn, g.pyp), zs = in_slab(k, g.nz, g.pzn, g.pzp);
    AdjSlab X{}, Y{}, Z{};
    if (xs) X = adj_slab<false>(g, psa, 0, i, j, k);
    if (ys) Y = adj_slab<false>(g, psa, 1, i, j, k);
    if (zs) Z = adj_slab<false>(g, psa, 2, i, j, k);
    const BgNode& B = p.bgn;
    const bool own = c != p.bg.mat, low = (own || !B.low_ok) && (i == 0 || j == 0 || k == 0);
    if (c >= kRecGeneral || low || (own && (xs || ys || zs) && !p.rows.h[0])) {
        adj_h_general(&p, &a, &psa, i, j, k, lx, ly, lz);
        return;
    }
    float ax = B.ha[0], ay = B.ha[1], az = B.ha[2];
    float cx0 = B.hc[0], cx1 = B.hc[1], cy0 = B.hc[2], cy1 = B.hc[3], cz0 = B.hc[4], cz1 = B.hc[5];
    if (own) {
        const float4 x = __ldg(&p.coef[c].h[0]), y = __ldg(&p.coef[c].h[1]), z = __ldg(&p.coef[c].h[2]);
        ax = x.x; cx0 = x.y; cx1 = x.z; ay = y.x; cy0 = y.y; cy1 = y.z; az = z.x; cz0 = z.y; cz1 = z.z;
    }
    const int rx = c * (g.pxn + g.pxp) + X.l, ry = c * (g.pyn + g.pyp) + Y.l, rz = c * (g.pzn + g.pzp) + Z.l;
    if (xs) { const float2 t = lo2(own ? p.rows.h[0] + rx : p.th[0] + i); cy0 = t.x; cz1 = t.y; }
    if (ys) { const float2 t = lo2(own ? p.rows.h[1] + ry : p.th[1] + j); cx1 = t.x; cz0 = t.y; }
    if (zs) { const float2 t = lo2(own ? p.rows.h[2] + rz : p.th[2] + k); cx0 = t.x; cy1 = t.y; }
    const bool mx = jp && kp, my = ip && kp, mz = ip && jp;
    float g0 = mx ? cx0 * lx : 0.f, g1 = mx ? cx1 * lx : 0.f, g2 = my ? cy0 * ly : 0.f, g3 = my ? cy1 * ly : 0.f;
    float g4 = mz ? cz0 * lz : 0.f, g5 = mz ? cz1 * lz : 0.f;
    if (xs) {
        const float2 t = hi2(p.th[0] + i), f = own ? hi2(p.rows.h[0] + rx) : make_float2(B.ch[0], B.ch[1]);
        if (my) g2 = adj_psi(psa.f[X.face].h[0] + X.q, t, f.x, X.old0, ly, g2);
        if (mz) g5 = adj_psi(psa.f[X.face].h[1] + X.q, t, f.y, X.old1, lz, g5);
    }
    if (ys) {
        const float2 t = hi2(p.th[1] + j), f = own ? hi2(p.rows.h[1] + ry) : make_float2(B.ch[2], B.ch[3]);
        if (mx) g1 = adj_psi(psa.f[Y.face].h[0] + Y.q, t, f.x, Y.old0, lx, g1);
        if (mz) g4 = adj_psi(psa.f[Y.face].h[1] + Y.q, t, f.y, Y.old1, lz, g4);
    }
    if (zs) {
        const float2 t = hi2(p.th[2] + k), f = own ? hi2(p.rows.h[2] + rz) : make_float2(B.ch[4], B.ch[5]);
        if (mx) g0 = adj_psi(psa.f[Z.face].h[0] + Z.q, t, f.x, Z.old0, lx, g0);
        if (my) g3 = adj_psi(psa.f[Z.face].h[1] + Z.q, t, f.y, Z.old1, ly, g3);
    }
    a.l[3][n] = mx ? ax * lx : lx; a.l[4][n] = my ? ay * ly : ly; a.l[5][n] = mz ? az * lz : lz;
    a.gh[0][n] = g0; a.gh[1][n] = g1; a.gh[2][n] = g2; a.gh[3][n] = g3; a.gh[4][n] = g4; a.gh[5][n] = g5;
}

// ---- transpose of calc_e (e_update), FoM source and design gradient ------------------------
// General path of k_adj_e, out of line.
__device__ __noinline__ void adj_e_general(const StepParams* pp, const AdjState* pa, const PsiSet* pps, const AdjStep* pst, int i,
                                           int j, int k, float lx, float ly, float lz) {
    const StepParams& p = *pp;
    const AdjState& a = *pa;
    const PsiSet& psa = *pps;
    const AdjStep& st = *pst;
    const DeviceGrid& g = p.g;
    const long long P = g.plane, R = g.pitch, n = node(g, i, j, k);
    const int c = p.cls[n];
    const uint8_t* mat = p.mat;
    const bool one = c >= kUniformGeneral && c < kInterfaceNode;  // seven cells of one material, given by the class
    const int m0 = one ? c - kUniformGeneral : mat[n];
    const int mi = one ? m0 : i > 0 ? mat[n - 1] : 0, mj = one ? m0 : j > 0 ? mat[n - R] : 0;
    const int mk = one ? m0 : k > 0 ? mat[n - P] : 0;
    const int mij = one ? m0 : (i > 0 && j > 0) ? mat[n - 1 - R] : 0;
    const int mik = one ? m0 : (i > 0 && k > 0) ? mat[n - 1 - P] : 0;
    const int mjk = one ? m0 : (j > 0 && k > 0) ? mat[n - R - P] : 0;
    const bool in_x = i > 0 && i < g.nx - 1, in_y = j > 0 && j < g.ny - 1, in_z = k > 0 && k < g.nz - 1;
    const bool ex_m = i < g.nx - 1 && in_y && in_z, ey_m = in_x && j < g.ny - 1 && in_z, ez_m = in_x && in_y && k < g.nz - 1;
    const bool xs = in_slab(i, g.nx, g.pxn, g.pxp), ys = in_slab(j, g.ny, g.pyn, g.pyp), zs = in_slab(k, g.nz, g.pzn, g.pzp);
    const int bg = p.bg.mat;
    const bool ux = m0 == mj && m0 == mk && m0 == mjk;
    const bool uy = m0 == mi && m0 == mk && m0 == mik;
    const bool uz = m0 == mi && m0 == mj && m0 == mij;
    const bool on_bg = m0 == bg;
    const Coef3 cx = e_coef<true>(p, 0, ux, m0, mj, mk, mjk, i, j, k);
    const Coef3 cy = e_coef<true>(p, 1, uy, m0, mi, mk, mik, i, j, k);
    const Coef3 cz = e_coef<true>(p, 2, uz, m0, mi, mj, mij, i, j, k);

    // design gradient: lambda here is dJ/dE^{m+1}; E^m and E^{m+1} come from the saved design E
    if (st.acc) {
        const int* d = p.dbox;
        const int ei = i - d[0], ej = j - d[1], ek = k - d[2];
        const int bx = d[3] - d[0] + 1, by = d[4] - d[1] + 1, bzz = d[5] - d[2] + 1;
        if (ei >= 0 && ej >= 0 && ek >= 0 && ei < bx && ej < by && ek < bzz) {
            const long long e = ((long long)ek * by + ej) * bx + ei, ne = (long long)bx * by * bzz;
            const float lam[3] = {lx, ly, lz};
            const Coef3 cc[3] = {cx, cy, cz};
            const bool on[3] = {ex_m, ey_m, ez_m};
            const int mm[3][4] = {{m0, mj, mk, mjk}, {m0, mi, mk, mik}, {m0, mi, mj, mij}};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (!on[c] || !has_design(p, mm[c][0], mm[c][1], mm[c][2], mm[c][3])) continue;
                const double2 w = st.weight[c * ne + e];
                const double em = st.e_old[c * ne + e], ep = st.e_new[c * ne + e];
                const double v = (double)lam[c] * (w.x * em - w.y * (ep - (double)cc[c].a * em));
                st.acc[c * ne + e] += v;
            }
        }
    }

    const BgCurl& B = p.bg;
    int side;
    float g0 = 0.f, g1 = 0.f, g2 = 0.f, g3 = 0.f, g4 = 0.f, g5 = 0.f;
    if (ex_m) {  // Ex: c1 on dHz_j (y CPML), c2 on dHy_k (z CPML)
        PsiTerm t1{nullptr, 0, 0, 0, 0}, t2{nullptr, 0, 0, 0, 0};
        if (ys) { const int q = psi_off_y(g, i, j, k, side); t1 = psi_term(psa.f[2 + side].e[0] + q, p.bey[j], p.aey[j], __fmul_rn(cx.bp, g.dy)); }
        if (zs) { const int q = psi_off_z(g, i, j, k, side); t2 = psi_term(psa.f[4 + side].e[0] + q, p.bez[k], p.aez[k], __fmul_rn(cx.bm, g.dz)); }
        const float c1 = ys ? kdiv(cx.bp, ux && on_bg, B.e[1][0], p.key, j) : cx.bp;
        const float c2 = zs ? kdiv(cx.bm, ux && on_bg, B.e[2][0], p.kez, k) : cx.bm;
        lx = adj_comp(lx, cx.a, c1, c2, t1, t2, g0, g1);
    }
    if (ey_m) {  // Ey: c1 on dHx_k (z CPML), c2 on dHz_i (x CPML)
        PsiTerm t1{nullptr, 0, 0, 0, 0}, t2{nullptr, 0, 0, 0, 0};
        if (zs) { const int q = psi_off_z(g, i, j, k, side); t1 = psi_term(psa.f[4 + side].e[1] + q, p.bez[k], p.aez[k], __fmul_rn(cy.bp, g.dz)); }
        if (xs) { const int q = psi_off_x(g, i, j, k, side); t2 = psi_term(psa.f[side].e[0] + q, p.bex[i], p.aex[i], __fmul_rn(cy.bm, g.dx)); }
        const float c1 = zs ? kdiv(cy.bp, uy && on_bg, B.e[2][1], p.kez, k) : cy.bp;
        const float c2 = xs ? kdiv(cy.bm, uy && on_bg, B.e[0][0], p.kex, i) : cy.bm;
        ly = adj_comp(ly, cy.a, c1, c2, t1, t2, g2, g3);
    }
    if (ez_m) {  // Ez: c1 on dHy_i (x CPML), c2 on dHx_j (y CPML); lumped edges override a, c1, c2
        PsiTerm t1{nullptr, 0, 0, 0, 0}, t2{nullptr, 0, 0, 0, 0};
        if (xs) { const int q = psi_off_x(g, i, j, k, side); t1 = psi_term(psa.f[side].e[1] + q, p.bex[i], p.aex[i], __fmul_rn(cz.bp, g.dx)); }
        if (ys) { const int q = psi_off_y(g, i, j, k, side); t2 = psi_term(psa.f[2 + side].e[1] + q, p.bey[j], p.aey[j], __fmul_rn(cz.bm, g.dy)); }
        const bool plane_lumped = p.lumped_k[k] < p.lumped_k[k + 1];
        const LumpedEdge* L = plane_lumped ? find_lumped(p, i, j, k, 2) : nullptr;  // design handles have no Ex edges
        float aa, c1, c2;
        if (L) { aa = L->ceze; c1 = L->cezhy; c2 = L->cezhx; }
        else {
            aa = cz.a;
            c1 = xs ? kdiv(cz.bp, uz && on_bg, B.e[0][1], p.kex, i) : cz.bp;
            c2 = ys ? kdiv(cz.bm, uz && on_bg, B.e[1][1], p.key, j) : cz.bm;
        }
        lz = adj_comp(lz, aa, c1, c2, t1, t2, g4, g5);
    }
    a.l[0][n] = lx; a.l[1][n] = ly; a.l[2][n] = lz;
    a.ge[0][n] = g0; a.ge[1][n] = g1; a.ge[2][n] = g2; a.ge[3][n] = g3; a.ge[4][n] = g4; a.ge[5][n] = g5;
}

// By coefficient row, as k_adj_h. The planes from the top down: it begins with what k_adj_h wrote last, which
// is still in L2 (the 192-step gradient 26.8 -> 25.9 ms).
template <typename Idx>
__global__ void __launch_bounds__(256, kAdjCtas) k_adj_e(const __grid_constant__ StepParams p, const __grid_constant__ AdjState a,
                                               const __grid_constant__ PsiSet psa, const __grid_constant__ AdjStep st) {
    grid_dependency_wait();
    grid_launch_dependents();
    const DeviceGrid& g = p.g;
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int k = gridDim.z - 1 - blockIdx.z;
    if (i >= g.nx || j >= g.ny) return;
    const Idx P = (Idx)g.plane, R = (Idx)g.pitch, n = (Idx)k * P + (Idx)j * R + (Idx)i;
    const int c = p.rec[n];
    // finish the transpose of calc_h: gather G_H
    float lx = a.l[0][n] + (k > 0 ? a.gh[3][n - P] : 0.f) - a.gh[3][n] + (j > 0 ? a.gh[4][n - R] : 0.f) - a.gh[4][n];
    float ly = a.l[1][n] + (k > 0 ? a.gh[0][n - P] : 0.f) - a.gh[0][n] + (i > 0 ? a.gh[5][n - 1] : 0.f) - a.gh[5][n];
    float lz = a.l[2][n] + (j > 0 ? a.gh[1][n - R] : 0.f) - a.gh[1][n] + (i > 0 ? a.gh[2][n - 1] : 0.f) - a.gh[2][n];
    if ((long long)n == st.probe) lz += st.source;  // dJ/dEz(p) of the sample taken in this step
    const bool xs = in_slab(i, g.nx, g.pxn, g.pxp), ys = in_slab(j, g.ny, g.pyn, g.pyp), zs = in_slab(k, g.nz, g.pzn, g.pzp);
    AdjSlab X{}, Y{}, Z{};
    if (xs) X = adj_slab<true>(g, psa, 0, i, j, k);
    if (ys) Y = adj_slab<true>(g, psa, 1, i, j, k);
    if (zs) Z = adj_slab<true>(g, psa, 2, i, j, k);
    const BgNode& B = p.bgn;
    const bool own = c != p.bg.mat;
    if (c >= kRecGeneral || (c >= p.des_row0 && c < p.des_row1) || (own && (xs || ys || zs) && !p.rows.e[0])) {  // the design edge box among them
        adj_e_general(&p, &a, &psa, &st, i, j, k, lx, ly, lz);
        return;
    }
    float ax = B.ea[0], ay = B.ea[1], az = B.ea[2];
    float cx0 = B.ec[0], cx1 = B.ec[1], cy0 = B.ec[2], cy1 = B.ec[3], cz0 = B.ec[4], cz1 = B.ec[5];
    if (own) {
        const float4 x = __ldg(&p.coef[c].e[0]), y = __ldg(&p.coef[c].e[1]), z = __ldg(&p.coef[c].e[2]);
        ax = x.x; cx0 = x.y; cx1 = x.z; ay = y.x; cy0 = y.y; cy1 = y.z; az = z.x; cz0 = z.y; cz1 = z.z;
    }
    const int rx = c * (g.pxn + g.pxp) + X.l, ry = c * (g.pyn + g.pyp) + Y.l, rz = c * (g.pzn + g.pzp) + Z.l;
    if (xs) { const float2 t = lo2(own ? p.rows.e[0] + rx : p.te[0] + i); cy1 = t.x; cz0 = t.y; }
    if (ys) { const float2 t = lo2(own ? p.rows.e[1] + ry : p.te[1] + j); cx0 = t.x; cz1 = t.y; }
    if (zs) { const float2 t = lo2(own ? p.rows.e[2] + rz : p.te[2] + k); cx1 = t.x; cy0 = t.y; }
    bool mx, my, mz;
    e_masks(g, i, j, k, mx, my, mz);
    float g0 = mx ? cx0 * lx : 0.f, g1 = mx ? cx1 * lx : 0.f, g2 = my ? cy0 * ly : 0.f, g3 = my ? cy1 * ly : 0.f;
    float g4 = mz ? cz0 * lz : 0.f, g5 = mz ? cz1 * lz : 0.f;
    if (xs) {
        const float2 t = hi2(p.te[0] + i), f = own ? hi2(p.rows.e[0] + rx) : make_float2(B.ce[0], B.ce[1]);
        if (my) g3 = adj_psi(psa.f[X.face].e[0] + X.q, t, f.x, X.old0, ly, g3);
        if (mz) g4 = adj_psi(psa.f[X.face].e[1] + X.q, t, f.y, X.old1, lz, g4);
    }
    if (ys) {
        const float2 t = hi2(p.te[1] + j), f = own ? hi2(p.rows.e[1] + ry) : make_float2(B.ce[2], B.ce[3]);
        if (mx) g0 = adj_psi(psa.f[Y.face].e[0] + Y.q, t, f.x, Y.old0, lx, g0);
        if (mz) g5 = adj_psi(psa.f[Y.face].e[1] + Y.q, t, f.y, Y.old1, lz, g5);
    }
    if (zs) {
        const float2 t = hi2(p.te[2] + k), f = own ? hi2(p.rows.e[2] + rz) : make_float2(B.ce[4], B.ce[5]);
        if (mx) g1 = adj_psi(psa.f[Z.face].e[0] + Z.q, t, f.x, Z.old0, lx, g1);
        if (my) g2 = adj_psi(psa.f[Z.face].e[1] + Z.q, t, f.y, Z.old1, ly, g2);
    }
    a.l[0][n] = mx ? ax * lx : lx; a.l[1][n] = my ? ay * ly : ly; a.l[2][n] = mz ? az * lz : lz;
    a.ge[0][n] = g0; a.ge[1][n] = g1; a.ge[2][n] = g2; a.ge[3][n] = g3; a.ge[4][n] = g4; a.ge[5][n] = g5;
}

// AdjStep::weight of the edges of the design edge box with a design cell: {da/deps, 2 eps0 / den} (the
// head of this file), the same in every step. Their FP64 divisions in every reverse step held the
// design region's CTAs back: k_adj_e 49 us against k_adj_h's 32 at 128^3 with a 32 x 32 x 16 region.
__global__ void k_adj_weights(const __grid_constant__ StepParams p, double2* out) {
    const DeviceGrid& g = p.g;
    const int* d = p.dbox;
    const int bx = d[3] - d[0] + 1, by = d[4] - d[1] + 1, bz = d[5] - d[2] + 1;
    const long long ne = (long long)bx * by * bz, e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int i = d[0] + (int)(e % bx), j = d[1] + (int)((e / bx) % by), k = d[2] + (int)(e / ((long long)bx * by));
    const long long P = g.plane, R = g.pitch, n = node(g, i, j, k);  // an interior node (fdtd_set_design_region)
    const uint8_t* mat = p.mat;
    const int m0 = mat[n], mi = mat[n - 1], mj = mat[n - R], mk = mat[n - P];
    const int mij = mat[n - 1 - R], mik = mat[n - 1 - P], mjk = mat[n - R - P];
    const int mm[3][4] = {{m0, mj, mk, mjk}, {m0, mi, mk, mik}, {m0, mi, mj, mij}};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double2 w = make_double2(0.0, 0.0);
        if (has_design(p, mm[c][0], mm[c][1], mm[c][2], mm[c][3])) {
            float eps, sig;
            edge_material(p, c, i, j, k, mm[c][0], mm[c][1], mm[c][2], mm[c][3], eps, sig);
            const double e0 = g.eps0, dt = g.dt;
            const double den = 2.0 * (double)eps * e0 + dt * (double)sig;
            w = make_double2(4.0 * e0 * dt * (double)sig / (den * den), 2.0 * e0 / den);
        }
        out[c * ne + e] = w;
    }
}

cudaError_t launch_adj_weights(const StepParams& p, double2* out, cudaStream_t s) {
    const int* d = p.dbox;
    const long long ne = (long long)(d[3] - d[0] + 1) * (d[4] - d[1] + 1) * (d[5] - d[2] + 1);
    k_adj_weights<<<(unsigned)((ne + 127) / 128), 128, 0, s>>>(p, out);
    return cudaGetLastError();
}

// After a forward step: the FoM sample Ez(p) and, when `snap` is set, the E components over the
// design edge box [d0, d3] x [d1, d4] x [d2, d5] (three arrays of the box volume).
__global__ void k_after_step(const float* ex, const float* ey, const float* ez, DeviceGrid g, long long probe,
                             float* sample, int d0, int d1, int d2, int bx, int by, int bz, float* snap) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q == 0 && sample) *sample = ez[probe];
    if (!snap) return;
    const long long ne = (long long)bx * by * bz;
    if (q >= ne) return;
    const int ei = (int)(q % bx), ej = (int)((q / bx) % by), ek = (int)(q / ((long long)bx * by));
    const int i = d0 + ei, j = d1 + ej, k = d2 + ek;
    if (i >= g.nx || j >= g.ny || k >= g.nz) { snap[q] = 0.f; snap[ne + q] = 0.f; snap[2 * ne + q] = 0.f; return; }
    const long long n = (long long)k * g.plane + (long long)j * g.pitch + i;
    snap[q] = ex[n];
    snap[ne + q] = ey[n];
    snap[2 * ne + q] = ez[n];
}

// dJ/deps_r of each design cell: a quarter of the accumulated edge terms of its twelve E edges.
__global__ void k_grad_finalize(const double* acc, int dx, int dy, int dz, double* grad) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= (long long)dx * dy * dz) return;
    const int ci = (int)(q % dx), cj = (int)((q / dx) % dy), ck = (int)(q / ((long long)dx * dy));
    const int bx = dx + 1, by = dy + 1, bz = dz + 1;
    const long long ne = (long long)bx * by * bz;
    auto at = [&](int c, int i, int j, int k) { return acc[c * ne + ((long long)k * by + j) * bx + i]; };
    double s = 0.0;
    // Ex edges (ci, cj..cj+1, ck..ck+1); Ey edges (ci..ci+1, cj, ck..ck+1); Ez (ci..ci+1, cj..cj+1, ck)
    for (int b = 0; b < 2; ++b)
        for (int c = 0; c < 2; ++c) {
            s += at(0, ci, cj + b, ck + c);
            s += at(1, ci + b, cj, ck + c);
            s += at(2, ci + b, cj + c, ck);
        }
    grad[q] = 0.25 * s;
}

cudaError_t launch_adj_step(const StepParams& p, const AdjState& a, const PsiSet& psa, const AdjStep& st,
                            cudaStream_t s) {
    const dim3 block(32, 8, 1), grid((p.g.nx + 31) / 32, (p.g.ny + 7) / 8, p.g.nz);
    const bool idx32 = p.g.plane * (long long)(p.g.nz + 1) < (1LL << 31);
    const cudaError_t e = launch_dependent(idx32 ? k_adj_h<uint32_t> : k_adj_h<unsigned long long>, grid, block, 0, s, p, a, psa);
    if (e != cudaSuccess) return e;
    return launch_dependent(idx32 ? k_adj_e<uint32_t> : k_adj_e<unsigned long long>, grid, block, 0, s, p, a, psa, st);
}

cudaError_t launch_after_step(const float* ex, const float* ey, const float* ez, const DeviceGrid& g, long long probe,
                              float* sample, const int dbox[6], float* snap, cudaStream_t s) {
    const int bx = dbox[3] - dbox[0] + 1, by = dbox[4] - dbox[1] + 1, bz = dbox[5] - dbox[2] + 1;
    const long long ne = snap ? (long long)bx * by * bz : 1;
    k_after_step<<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(ex, ey, ez, g, probe, sample, dbox[0], dbox[1], dbox[2],
                                                             bx, by, bz, snap);
    return cudaGetLastError();
}

// The six field components over node box b, to (save) or from a packed buffer of 6 x box volume
// floats (component-major, x fastest).
__global__ void k_box_state(FieldPtrs f, DeviceGrid g, NodeBox b, float* buf, bool save) {
    const int bx = b.x1 - b.x0, by = b.y1 - b.y0;
    const long long nb = (long long)bx * by * (b.z1 - b.z0);
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= nb) return;
    const int i = b.x0 + (int)(q % bx), j = b.y0 + (int)((q / bx) % by), k = b.z0 + (int)(q / ((long long)bx * by));
    const long long n = (long long)k * g.plane + (long long)j * g.pitch + i;
    float* c[6] = {f.ex, f.ey, f.ez, f.hx, f.hy, f.hz};
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        if (save) buf[r * nb + q] = c[r][n];
        else c[r][n] = buf[r * nb + q];
    }
}

cudaError_t launch_box_state(const FieldPtrs& f, const DeviceGrid& g, const NodeBox& b, float* buf, bool save,
                             cudaStream_t s) {
    if (b.x0 < 0 || b.y0 < 0 || b.z0 < 0 || b.x1 > g.nx || b.y1 > g.ny || b.z1 > g.nz) return cudaErrorInvalidValue;
    const long long nb = (long long)(b.x1 - b.x0) * (b.y1 - b.y0) * (b.z1 - b.z0);
    if (nb <= 0) return cudaSuccess;
    k_box_state<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>(f, g, b, buf, save);
    return cudaGetLastError();
}

cudaError_t launch_grad_finalize(const double* acc, const int dbox[6], double* grad, cudaStream_t s) {
    const int dx = dbox[3] - dbox[0], dy = dbox[4] - dbox[1], dz = dbox[5] - dbox[2];
    const long long n = (long long)dx * dy * dz;
    k_grad_finalize<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(acc, dx, dy, dz, grad);
    return cudaGetLastError();
}

}  // namespace fdtd
