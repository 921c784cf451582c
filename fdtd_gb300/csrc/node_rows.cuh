// Per-node E and H updates by coefficient row (StepParams::rec): the two-pass kernels. Same results as
// node_global.cuh, which serves the nodes on the general path here and the kernels that keep to the
// node classes (batch.cu, k_design_e, k_plate_e).
//
// One node per thread is bound by its instructions and one round of loads, so the common node does
// little: the row, twelve field values and the CPML memory load together (their addresses depend on
// the position only), the background's coefficients are constants, a slab's curl coefficients and
// recurrence factors come from its axis' table in one 16-byte load, and other rows' from the row
// tables. Nodes on the general path call out of line, so that their code costs the others neither
// registers nor instruction cache. Probes are not looked for here: see ProbeList. At
// 128^3 a step takes 41.4 us against 45.7 by class, at 64^3 11.5 against 15.0.
#pragma once

#include "node_global.cuh"

namespace fdtd {

// The step: m, or *base + m where base is given (a CUDA graph captured once replays those while a counter
// on the device advances: the batched chain form).
struct StepIndex {
    const long long* base;
    long long m;
    __device__ __forceinline__ long long at() const { return base ? *base + m : m; }
};

// kDesign: the grid has a design region (the other grids' pass is kept free of its code, which cost 5 % at 128^3).
template <typename Idx, bool kDesign>
static __device__ __noinline__ void e_node_general(const StepParams* p, const FieldPtrs* f, const PsiSet* ps, const StepIndex* step,
                                                   int i, int j, int k) {
    const int c = kDesign ? p->rec[(Idx)k * (Idx)p->g.plane + (Idx)j * (Idx)p->g.pitch + (Idx)i] : 0;
    if (kDesign && design_row(*p, c))
        e_node_design<false, Idx>(*p, *f, *f, i, j, k, 0);
    else if (kDesign && c == (kRecGeneral | kDesignNode))
        e_node_global<true>(*p, *f, *f, *ps, *ps, i, j, k, step->at());
    else
        e_node_global<false, false, false, Idx>(*p, *f, *f, *ps, *ps, i, j, k, step->at());
}
template <typename Idx>
static __device__ __noinline__ void h_node_general(const StepParams* p, const FieldPtrs* f, const PsiSet* ps, const StepIndex* step,
                                                   int i, int j, int k) {
    h_node_global<false, Idx>(*p, *f, *f, *f, *ps, *ps, i, j, k, step->at());
}

// The CPML memory of a node on one axis: offsets of E array 0 and the arrays' stride from PsiSet::base,
// and the node's slab plane (SlabRows).
template <typename Idx>
struct PsiSlot {
    Idx at, stride;
    int l;
};
// face: 0 x, 2 y, 4 z; q: the node's index on the axis; plane: elements per slab plane, or for x per
// node; rest: offset within the plane.
template <typename Idx>
__device__ __forceinline__ PsiSlot<Idx> psi_slot(const StepParams& p, int face, int q, int n, int pn, int pp, Idx unit, Idx rest) {
    const bool lo = q < pn;
    const int t = lo ? q : q - (n - pp);
    return PsiSlot<Idx>{(Idx)p.psi_off[face + !lo] + (Idx)t * unit + rest, (Idx)p.psi_stride[face + !lo], lo ? t : t + pn};
}
template <typename Idx>
__device__ __forceinline__ PsiSlot<Idx> psi_slot_x(const StepParams& p, int i, int j, int k) {
    const DeviceGrid& g = p.g;
    return psi_slot<Idx>(p, 0, i, g.nx, g.pxn, g.pxp, 1, ((Idx)k * (Idx)g.ny + (Idx)j) * (Idx)(i < g.pxn ? g.pxn : g.pxp));
}
template <typename Idx>
__device__ __forceinline__ PsiSlot<Idx> psi_slot_y(const StepParams& p, int i, int j, int k) {
    const DeviceGrid& g = p.g;
    return psi_slot<Idx>(p, 2, j, g.ny, g.pyn, g.pyp, (Idx)g.pitch, (Idx)k * (Idx)(j < g.pyn ? g.pyn : g.pyp) * (Idx)g.pitch + (Idx)i);
}
template <typename Idx>
__device__ __forceinline__ PsiSlot<Idx> psi_slot_z(const StepParams& p, int i, int j, int k) {
    const DeviceGrid& g = p.g;
    return psi_slot<Idx>(p, 4, k, g.nz, g.pzn, g.pzp, (Idx)g.plane, (Idx)j * (Idx)g.pitch + (Idx)i);
}

// The halves of an axis table's or SlabRows' entry: curl coefficients; recurrence factors (axis tables) or
// factors of the CPML memory (SlabRows).
__device__ __forceinline__ float2 curl_pair(const float4* t) { return __ldg(reinterpret_cast<const float2*>(t)); }
__device__ __forceinline__ float2 psi_pair(const float4* t) { return __ldg(reinterpret_cast<const float2*>(t) + 1); }

template <typename Idx, bool kDesign>
__device__ __forceinline__ void e_node_rows(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, int i, int j, int k,
                                            const StepIndex& step) {
    const DeviceGrid& g = p.g;
    const Idx P = (Idx)g.plane, R = (Idx)g.pitch, n = (Idx)k * P + (Idx)j * R + (Idx)i;
    const int c = p.rec[n];
    const float ex = f.ex[n], ey = f.ey[n], ez = f.ez[n], hx = f.hx[n], hy = f.hy[n], hz = f.hz[n];
    const float hx_jm = j > 0 ? f.hx[n - R] : 0.f, hx_km = k > 0 ? f.hx[n - P] : 0.f;
    const float hy_im = i > 0 ? f.hy[n - 1] : 0.f, hy_km = k > 0 ? f.hy[n - P] : 0.f;
    const float hz_im = i > 0 ? f.hz[n - 1] : 0.f, hz_jm = j > 0 ? f.hz[n - R] : 0.f;
    const bool xs = in_slab(i, g.nx, g.pxn, g.pxp), ys = in_slab(j, g.ny, g.pyn, g.pyp), zs = in_slab(k, g.nz, g.pzn, g.pzp);
    const bool slab = xs || ys || zs;
    PsiSlot<Idx> X{}, Y{}, Z{};
    float x0, x1, y0, y1, z0, z1;
    if (xs) { X = psi_slot_x<Idx>(p, i, j, k); }
    if (ys) { Y = psi_slot_y<Idx>(p, i, j, k); }
    if (zs) { Z = psi_slot_z<Idx>(p, i, j, k); }
    const BgNode& B = p.bgn;
    const bool own = c != p.bg.mat;
    if (c >= kRecGeneral || (kDesign && design_row(p, c)) || (own && slab && !p.rows.e[0])) {
        e_node_general<Idx, kDesign>(&p, &f, &ps, &step, i, j, k);
        return;
    }
    float ax = B.ea[0], ay = B.ea[1], az = B.ea[2];
    float cx0 = B.ec[0], cx1 = B.ec[1], cy0 = B.ec[2], cy1 = B.ec[3], cz0 = B.ec[4], cz1 = B.ec[5];
    if (own) {
        const float4 a = __ldg(&p.coef[c].e[0]), b = __ldg(&p.coef[c].e[1]), d = __ldg(&p.coef[c].e[2]);
        ax = a.x; cx0 = a.y; cx1 = a.z; ay = b.x; cy0 = b.y; cy1 = b.z; az = d.x; cz0 = d.y; cz1 = d.z;
    }
    const int rx = c * (g.pxn + g.pxp) + X.l, ry = c * (g.pyn + g.pyp) + Y.l, rz = c * (g.pzn + g.pzp) + Z.l;
    if (slab) {  // the curl coefficients along a slab's axis, over kappa
        if (xs) { const float2 t = curl_pair(own ? p.rows.e[0] + rx : p.te[0] + i); cy1 = t.x; cz0 = t.y; }
        if (ys) { const float2 t = curl_pair(own ? p.rows.e[1] + ry : p.te[1] + j); cx0 = t.x; cz1 = t.y; }
        if (zs) { const float2 t = curl_pair(own ? p.rows.e[2] + rz : p.te[2] + k); cx1 = t.x; cy0 = t.y; }
    }
    const float dHz_j = __fsub_rn(hz, hz_jm), dHy_k = __fsub_rn(hy, hy_km), dHx_k = __fsub_rn(hx, hx_km);
    const float dHz_i = __fsub_rn(hz, hz_im), dHy_i = __fsub_rn(hy, hy_im), dHx_j = __fsub_rn(hx, hx_jm);
    float vx = upd3(ax, ex, cx0, dHz_j, cx1, dHy_k);
    float vy = upd3(ay, ey, cy0, dHx_k, cy1, dHz_i);
    float vz = upd3(az, ez, cz0, dHy_i, cz1, dHx_j);
    if (c >= p.src_row0) {  // lumped source edge (fdtdrav.h:728)
        const SrcRow sr = p.src_rows[c - p.src_row0];
        const long long m = step.at();
        vz = __fmaf_rn(sr.cezj, m < p.wave_len[sr.source] ? p.waves[sr.source][m] : 0.f, vz);
    }
    bool mx, my, mz;
    e_masks(g, i, j, k, mx, my, mz);
    if (xs) {  // fdtdrav.h:752-785
        x0 = ps.base[X.at]; x1 = ps.base[X.at + X.stride];
        const float2 t = psi_pair(p.te[0] + i), u = own ? psi_pair(p.rows.e[0] + rx) : make_float2(B.ce[0], B.ce[1]);
        x0 = psi_upd(t.x, x0, t.y, dHz_i); x1 = psi_upd(t.x, x1, t.y, dHy_i);
        if (my) ps.base[X.at] = x0;
        if (mz) ps.base[X.at + X.stride] = x1;
        vy = psi_add(vy, u.x, x0); vz = psi_add(vz, u.y, x1);
    }
    if (ys) {  // fdtdrav.h:790-827
        y0 = ps.base[Y.at]; y1 = ps.base[Y.at + Y.stride];
        const float2 t = psi_pair(p.te[1] + j), u = own ? psi_pair(p.rows.e[1] + ry) : make_float2(B.ce[2], B.ce[3]);
        y0 = psi_upd(t.x, y0, t.y, dHz_j); y1 = psi_upd(t.x, y1, t.y, dHx_j);
        if (mx) ps.base[Y.at] = y0;
        if (mz) ps.base[Y.at + Y.stride] = y1;
        vx = psi_add(vx, u.x, y0); vz = psi_add(vz, u.y, y1);
    }
    if (zs) {  // fdtdrav.h:829-911
        z0 = ps.base[Z.at]; z1 = ps.base[Z.at + Z.stride];
        const float2 t = psi_pair(p.te[2] + k), u = own ? psi_pair(p.rows.e[2] + rz) : make_float2(B.ce[4], B.ce[5]);
        z0 = psi_upd(t.x, z0, t.y, dHy_k); z1 = psi_upd(t.x, z1, t.y, dHx_k);
        if (mx) ps.base[Z.at] = z0;
        if (my) ps.base[Z.at + Z.stride] = z1;
        vx = psi_add(vx, u.x, z0); vy = psi_add(vy, u.y, z1);
    }
    if (mx) f.ex[n] = vx;
    if (my) f.ey[n] = vy;
    if (mz) f.ez[n] = vz;
}

template <typename Idx>
__device__ __forceinline__ void h_node_rows(const StepParams& p, const FieldPtrs& f, const PsiSet& ps, int i, int j, int k,
                                            const StepIndex& step) {
    const DeviceGrid& g = p.g;
    const Idx P = (Idx)g.plane, R = (Idx)g.pitch, n = (Idx)k * P + (Idx)j * R + (Idx)i;
    const int c = p.rec[n];
    const float hx = f.hx[n], hy = f.hy[n], hz = f.hz[n], ex = f.ex[n], ey = f.ey[n], ez = f.ez[n];
    const bool ix = i < g.nx - 1, iy = j < g.ny - 1, iz = k < g.nz - 1;
    const float ey_kp = iz ? f.ey[n + P] : 0.f, ex_kp = iz ? f.ex[n + P] : 0.f;
    const float ez_jp = iy ? f.ez[n + R] : 0.f, ex_jp = iy ? f.ex[n + R] : 0.f;
    const float ez_ip = ix ? f.ez[n + 1] : 0.f, ey_ip = ix ? f.ey[n + 1] : 0.f;
    const bool xs = in_slab(i, g.nx, g.pxn, g.pxp), ys = in_slab(j, g.ny, g.pyn, g.pyp), zs = in_slab(k, g.nz, g.pzn, g.pzp);
    const bool slab = xs || ys || zs;
    PsiSlot<Idx> X{}, Y{}, Z{};
    float x0, x1, y0, y1, z0, z1;
    if (xs) { X = psi_slot_x<Idx>(p, i, j, k); X.at += 2 * X.stride; }
    if (ys) { Y = psi_slot_y<Idx>(p, i, j, k); Y.at += 2 * Y.stride; }
    if (zs) { Z = psi_slot_z<Idx>(p, i, j, k); Z.at += 2 * Z.stride; }
    const BgNode& B = p.bgn;
    const bool own = c != p.bg.mat, low = (own || !B.low_ok) && (i == 0 || j == 0 || k == 0);
    if (c >= kRecGeneral || low || (own && slab && !p.rows.h[0])) {  // (faces on a low wall take the default entry)
        h_node_general<Idx>(&p, &f, &ps, &step, i, j, k);
        return;
    }
    float ax = B.ha[0], ay = B.ha[1], az = B.ha[2];
    float cx0 = B.hc[0], cx1 = B.hc[1], cy0 = B.hc[2], cy1 = B.hc[3], cz0 = B.hc[4], cz1 = B.hc[5];
    if (own) {
        const float4 a = __ldg(&p.coef[c].h[0]), b = __ldg(&p.coef[c].h[1]), d = __ldg(&p.coef[c].h[2]);
        ax = a.x; cx0 = a.y; cx1 = a.z; ay = b.x; cy0 = b.y; cy1 = b.z; az = d.x; cz0 = d.y; cz1 = d.z;
    }
    const int rx = c * (g.pxn + g.pxp) + X.l, ry = c * (g.pyn + g.pyp) + Y.l, rz = c * (g.pzn + g.pzp) + Z.l;
    if (slab) {
        if (xs) { const float2 t = curl_pair(own ? p.rows.h[0] + rx : p.th[0] + i); cy0 = t.x; cz1 = t.y; }
        if (ys) { const float2 t = curl_pair(own ? p.rows.h[1] + ry : p.th[1] + j); cx1 = t.x; cz0 = t.y; }
        if (zs) { const float2 t = curl_pair(own ? p.rows.h[2] + rz : p.th[2] + k); cx0 = t.x; cy1 = t.y; }
    }
    const float dEy_k = __fsub_rn(ey_kp, ey), dEz_j = __fsub_rn(ez_jp, ez), dEz_i = __fsub_rn(ez_ip, ez);
    const float dEx_k = __fsub_rn(ex_kp, ex), dEx_j = __fsub_rn(ex_jp, ex), dEy_i = __fsub_rn(ey_ip, ey);
    float vx = upd3_hx(ax, hx, cx0, dEy_k, cx1, dEz_j);
    float vy = upd3(ay, hy, cy0, dEz_i, cy1, dEx_k);
    float vz = upd3(az, hz, cz0, dEx_j, cz1, dEy_i);
    const bool mx = iy && iz, my = ix && iz, mz = ix && iy;
    if (xs) {  // fdtdrav.h:401-442
        x0 = ps.base[X.at]; x1 = ps.base[X.at + X.stride];
        const float2 t = psi_pair(p.th[0] + i), u = own ? psi_pair(p.rows.h[0] + rx) : make_float2(B.ch[0], B.ch[1]);
        x0 = psi_upd(t.x, x0, t.y, dEz_i); x1 = psi_upd(t.x, x1, t.y, dEy_i);
        if (my) ps.base[X.at] = x0;
        if (mz) ps.base[X.at + X.stride] = x1;
        vy = psi_add(vy, u.x, x0); vz = psi_add(vz, u.y, x1);
    }
    if (ys) {  // fdtdrav.h:445-486
        y0 = ps.base[Y.at]; y1 = ps.base[Y.at + Y.stride];
        const float2 t = psi_pair(p.th[1] + j), u = own ? psi_pair(p.rows.h[1] + ry) : make_float2(B.ch[2], B.ch[3]);
        y0 = psi_upd(t.x, y0, t.y, dEz_j); y1 = psi_upd(t.x, y1, t.y, dEx_j);
        if (mx) ps.base[Y.at] = y0;
        if (mz) ps.base[Y.at + Y.stride] = y1;
        vx = psi_add(vx, u.x, y0); vz = psi_add(vz, u.y, y1);
    }
    if (zs) {  // fdtdrav.h:489-562
        z0 = ps.base[Z.at]; z1 = ps.base[Z.at + Z.stride];
        const float2 t = psi_pair(p.th[2] + k), u = own ? psi_pair(p.rows.h[2] + rz) : make_float2(B.ch[4], B.ch[5]);
        z0 = psi_upd(t.x, z0, t.y, dEy_k); z1 = psi_upd_hyz(t.x, z1, t.y, dEx_k);
        if (mx) ps.base[Z.at] = z0;
        if (my) ps.base[Z.at + Z.stride] = z1;
        vx = psi_add(vx, u.x, z0); vy = psi_add(vy, u.y, z1);
    }
    if (mx) f.hx[n] = vx;
    if (my) f.hy[n] = vy;
    if (mz) f.hz[n] = vz;
}

}  // namespace fdtd
