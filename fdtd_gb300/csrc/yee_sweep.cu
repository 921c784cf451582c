// Fused schedule: one kernel per time step sweeps the whole grid, fields A -> B and CPML memory
// psi_in -> psi_out.
//
// A CTA owns a column of 32 x kSweepRows nodes and a chunk of planes [k0, k1) and marches along z, a
// quad of four x-neighbours per thread: the addresses, tests and parameter loads, which outnumber
// the arithmetic several times in a kernel of one node per thread, are shared by the quad, and its
// values move as 16-byte words. Planes stream through a shared-memory ring filled by TMA
// (cp.async.bulk.tensor, 3-D tiles, the next plane in flight while one is computed): H with a
// one-node halo, old E, and the 16-bit coefficient row of each node (StepParams::rec). At plane k a
// thread computes E(k) of its quad and then H(k-1), whose neighbours' E(k-1) lie in shared memory
// since the step before: one barrier per plane. What it needs of its own nodes at plane k-1 stays
// in registers. One more warp computes E on the row above the tile and the column beside it, which
// the H update needs (recomputed from the old fields, not exchanged).
//
// Coefficients. A quad whose four nodes share a coefficient row loads it once (the background's comes
// with the kernel parameters); in a CPML slab the curl coefficients along the slab's axis come from
// the axis' table for background nodes (StepParams::te, th: divided by kappa) and from SlabRows for
// other rows. Quads of several rows load them component by component, or node by node where the registers
// do not allow that. With materials in the slabs of which none is magnetic (StepParams::h_bg), H looks at no
// rows. What is left (lumped edges and probes in a slab, design nodes with a lumped edge, keys beyond the table)
// runs e_update_diff / h_update_diff (slow_node).
// Old CPML memory of the y and z faces is fetched a plane ahead with cp.async into slots of the
// thread's own.
//
// What bounds it: on grids beyond L2, HBM and the latency of a plane step; on smaller ones the latency
// of a plane step alone (15 warps an SM, about 650 instructions per quad and step, a third of the
// issue slots) and, with materials in the slabs, the tiles that hold them. Measured per step with boxes clear of
// the CPML, against the schedule it replaced (a sweep of the interior tiles, then one-node-per-thread passes over
// the CPML shell): 512^3 1.59 -> 1.30 ms, 256^3 0.279 -> 0.226, 1024 x 1024 x 896 10.4 -> 8.3; against the two passes
// of that time, 64^3 18.3 -> 11.5 us. One node per thread in the same march ran 2.0 ms at 512^3
// (352 instructions per node against about 165). 3 CTAs an SM (128 registers) against 2: 512^3 1.39 /
// 1.55 ms, 128^3 52 / 61 us. Registers decide much: spills of 100 bytes in the march cost 5 % at 512^3 and
// 20 % at 64^3, so old H of a plane is read again from its stage at the end of the step rather than
// kept through it (of the kernels here, those of materials in the slabs spill 40 to 72 bytes in the two-CTA
// and the 64-bit form, the others none); and code, as the march should fit the instruction cache: rows other than
// the background's have their slab coefficients in a table (SlabRows), since divisions in line made grids
// with materials in the slabs 10-20 % slower.
// All arithmetic is that of yee_common.cuh, so the results equal the two-pass schedule's bits.
// Every wait on a TMA barrier is bounded: on timeout the kernel uses nothing of that plane, records an
// error in the status word, drains its own copies (again bounded) and exits.
#define FDTD_RARE __forceinline__  // calls in the slow path would spill the march's state (512^3: 31.0 -> 28.6 ms for 20 steps)
#include <cuda.h>

#include <algorithm>

#include "planner.h"
#include "tma.cuh"
#include "yee_common.cuh"
#include "yee_kernels.h"

namespace fdtd {

namespace {

// Stages of the ring: a third one left less of the SM's memory to L1 and was 12-20 % slower.
constexpr int TX = kTileX, TY = kSweepRows;
constexpr int QX = TX / 4;                // quads per row
constexpr int NOWN = QX * TY;             // threads with a quad of the tile; then the halo row and column
constexpr int NTH = NOWN + (QX + TY + 31) / 32 * 32;
static_assert(NOWN % 32 == 0, "own quads fill whole warps");
constexpr int NST = 2;                    // planes in the ring
// A grid swept alone of up to this many CTAs: two of 168 registers an SM run the grid at once (kWide) instead of three of 128:
// a plane step is shorter with the registers to have the loads of a quad of several rows in flight
// together (64^3: vacuum 11.0 -> 10.4 us a step, boxes 12.5 -> 10.5, boxes that touch a CPML slab 16.7 -> 12.6).
constexpr unsigned kSweepWideCtas = 2 * 152;
constexpr int round128(int b) { return (b + 127) / 128 * 128; }
// Tiles in shared memory. H and coefficient rows, with rows of W: x in [x0-4, x0+36), y in
// [y0-1, y0+TY] and x in [x0, x0+40), y in [y0, y0+TY]; old and new E, with rows of WE: x in
// [x0, x0+36), y in [y0, y0+TY].
constexpr int W = TX + 8, WE = TX + 4, HR = TY + 2, ER = TY + 1;
constexpr int H_BYTES = round128(W * HR * 4), E_BYTES = round128(WE * ER * 4), M_BYTES = round128(W * ER * 2);
constexpr int STAGE_BYTES = 3 * H_BYTES + 3 * E_BYTES + M_BYTES;
constexpr unsigned H_TX = W * HR * 4, E_TX = WE * ER * 4, M_TX = W * ER * 2;  // bytes the boxes carry
constexpr int HF = H_BYTES / 4, EF = E_BYTES / 4;
constexpr int H_OFF = W + 4, E_OFF = 3 * HF;  // float offsets in a stage of a tile node 0's Hx and Ex
constexpr int NF = WE * ER;               // floats of one new-E component plane
// CPML memory of a thread's quad on its y face, or its z face where it lies in no y slab, fetched one
// plane ahead (cp.async): E arrays 0 and 1, H arrays 0 and 1
enum { kPsiE = 0, kPsiH = 2, kPsiSlots = 4 };

// Where the CPML memory of a plane of a z face begins: E array 0 of node (0, 0) at base, the face's
// other arrays `stride` apart (E1, H0, H1). on = 0: the plane lies in no z slab.
template <typename Idx>
struct __align__(16) PsiAt {
    Idx base, stride, on, pad;
};

template <typename Idx>
struct SweepSmem {
    unsigned char stage[NST][STAGE_BYTES];  // H (3), old E (3), rows of a plane
    float enew[2][3][NF];                   // new E of planes k - 1, k
    float4 psi[kPsiSlots][NTH];
    float xe[4][W], xh[4][W];               // curl 0, curl 1, b, a of each column, E and H
    float4 ye[ER], yh[ER];                  // {curl 0, curl 1, b, a} of each row / plane
    float4 ze[kMaxSweepPlanes], zh[kMaxSweepPlanes];
    PsiAt<Idx> zo[kMaxSweepPlanes];
    uint64_t bar[NST];
    long long m;                            // the step
};

__device__ __forceinline__ const float* f32(const unsigned char* b) { return reinterpret_cast<const float*>(b); }

// The kernel's parameters, in constant memory.
struct SweepArgs {
    FusedMaps maps;
    StepParams p;
    FieldPtrs fo;
    PsiSet pin, pout;
    SweepPlan sg;
    long long m;            // the step, or its offset from *base
    const long long* base;  // device step counter (launches captured in a graph), or NULL
    FieldPtrs fi;
    const ProbeAt* probes;  // probes outside the CPML slabs (n of them), sampled one step late: see k_sweep
    int n_probes_at;
    int late;               // the step before this one belongs to the same call
    float sig[kSweepSources];  // this step's signal of each source
};

__device__ __forceinline__ long long sweep_m(const SweepArgs& A) { return A.base ? *A.base + A.m : A.m; }
__device__ __forceinline__ float sweep_sig(const SweepArgs& A, int source) {
    if (!A.base) return A.sig[source];
    const long long m = sweep_m(A);
    return m < A.p.wave_len[source] ? A.p.waves[source][m] : 0.f;
}

// Slow path, one node at a time (in line: a call would spill the march's state): nodes on the general path
// (lumped edges and probes in a slab, design nodes with a lumped edge, keys beyond the table), nodes of another
// material than the background in a CPML slab where there is no SlabRows table, and H faces of such nodes on
// the low walls. bits: 1 E(k), 2 H(k-1), 4 a node of the tile (stored, probes
// sampled), 8 E(k) is this chunk's. Old H of plane k - 1 and the node's row there come with the
// call, the rest from the shared-memory tiles.
template <typename Idx>
__device__ __forceinline__ void slow_node(const SweepArgs* pa, SweepSmem<Idx>* ps, int bits, int k, int stage, int i, int j,
                                       int t, int te, float hxp, float hyp, float hzp, int cp) {
    const StepParams& p = pa->p;
    const FieldPtrs& fo = pa->fo;
    SweepSmem<Idx>& S = *ps;
    const float* T = f32(S.stage[stage]) + t;
    const float* TE = f32(S.stage[stage]) + E_OFF + te;
    float* en = &S.enew[k & 1][0][te];
    const float* ep = &S.enew[(k - 1) & 1][0][te];
    const long long R = p.g.pitch, PL = p.g.plane, m = S.m, rr = m % p.ring_cap;
    const bool own = bits & 4, store_e = bits & 8;
    float out[3], pre[3];
    if (bits & 1) {
        const float *H0 = T + H_OFF, *H1 = H0 + HF, *H2 = H1 + HF;
        EDiff d;
        d.dHz_j = __fsub_rn(H2[0], H2[-W]);
        d.dHx_j = __fsub_rn(H0[0], H0[-W]);
        d.dHy_k = __fsub_rn(H1[0], hyp);
        d.dHx_k = __fsub_rn(H0[0], hxp);
        d.dHz_i = __fsub_rn(H2[0], H2[-1]);
        d.dHy_i = __fsub_rn(H1[0], H1[-1]);
        const int c = reinterpret_cast<const uint16_t*>(S.stage[stage] + 3 * H_BYTES + 3 * E_BYTES)[t];
        const long long n = (long long)k * PL + (long long)j * R + i;
        ENbr nb{};
        nb.ex = TE[0]; nb.ey = TE[EF]; nb.ez = TE[2 * EF];
        const PsiIO io{pa->pin.f, pa->pout.f, own && store_e};
        if (c < kRecGeneral) {
            e_update_diff<false, false, false, false, true>(p, nb, d, i, j, k, m, false, io, out, pre, c);
        } else {
            const uint8_t* mat = p.mat;
            nb.m0 = mat[n];
            nb.mi = i > 0 ? mat[n - 1] : 0;
            nb.mj = j > 0 ? mat[n - R] : 0;
            nb.mk = k > 0 ? mat[n - PL] : 0;
            nb.mij = (i > 0 && j > 0) ? mat[n - 1 - R] : 0;
            nb.mik = (i > 0 && k > 0) ? mat[n - 1 - PL] : 0;
            nb.mjk = (j > 0 && k > 0) ? mat[n - R - PL] : 0;
            const bool lumped = p.lumped_k[k] < p.lumped_k[k + 1];
            e_update_diff<true, false, true, false>(p, nb, d, i, j, k, m, lumped, io, out, pre);
            if (own && store_e && p.probe_k[k] < p.probe_k[k + 1])
                for (int a = 0; a < 3; ++a) sample(p, rr, a, i, j, k, pre[a]);
        }
        en[0] = out[0]; en[NF] = out[1]; en[2 * NF] = out[2];
        if (own && store_e) { fo.ex[n] = out[0]; fo.ey[n] = out[1]; fo.ez[n] = out[2]; }
    }
    if (!(bits & 2)) return;
    const int kh = k - 1;
    HNbr nb{};
    nb.hx = hxp; nb.hy = hyp; nb.hz = hzp;
    HDiff f;
    f.dEy_k = __fsub_rn(en[NF], ep[NF]);
    f.dEx_k = __fsub_rn(en[0], ep[0]);
    f.dEz_j = __fsub_rn(ep[2 * NF + WE], ep[2 * NF]);
    f.dEx_j = __fsub_rn(ep[WE], ep[0]);
    f.dEz_i = __fsub_rn(ep[2 * NF + 1], ep[2 * NF]);
    f.dEy_i = __fsub_rn(ep[NF + 1], ep[NF]);
    const long long n = (long long)kh * PL + (long long)j * R + i;
    const PsiIO io{pa->pin.f, pa->pout.f, true};
    if (cp < kRecGeneral) {
        h_update_diff<false, false, true>(p, nb, f, i, j, kh, io, out, pre, cp);
    } else {
        const uint8_t* mat = p.mat;
        nb.m0 = mat[n];
        nb.mi = i > 0 ? mat[n - 1] : 0;
        nb.mj = j > 0 ? mat[n - R] : 0;
        nb.mk = kh > 0 ? mat[n - PL] : 0;
        h_update_diff<false, false>(p, nb, f, i, j, kh, io, out, pre);
        if (p.probe_k[kh] < p.probe_k[kh + 1])
            for (int a = 0; a < 3; ++a) sample(p, rr, 3 + a, i, j, kh, pre[a]);
    }
    fo.hx[n] = out[0]; fo.hy[n] = out[1]; fo.hz[n] = out[2];
}

struct Quad {
    float v[4];
};
__device__ __forceinline__ Quad lds4(const float* a) {
    const float4 f = *reinterpret_cast<const float4*>(a);
    return Quad{f.x, f.y, f.z, f.w};
}
__device__ __forceinline__ Quad ldg4(const float* a) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(a));
    return Quad{f.x, f.y, f.z, f.w};
}
__device__ __forceinline__ void st4(float* a, const Quad& q) {
    *reinterpret_cast<float4*>(a) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
// The nodes of a mask (bit r: node r) to a[0 .. 3] (and b, c).
__device__ __forceinline__ void st_mask3(float* a, float* b, float* c, const Quad& x, const Quad& y, const Quad& z, int mask) {
    if (mask == 15) {
        st4(a, x); st4(b, y); st4(c, z);
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (mask >> r & 1) { a[r] = x.v[r]; b[r] = y.v[r]; c[r] = z.v[r]; }
    }
}
__device__ __forceinline__ void st_mask2(float* a, float* b, const Quad& x, const Quad& y, int ma, int mb) {
    if ((ma & mb) == 15) {
        st4(a, x); st4(b, y);
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (ma >> r & 1) a[r] = x.v[r];
            if (mb >> r & 1) b[r] = y.v[r];
        }
    }
}
// The halves of an entry of SlabRows: curl coefficients, factors of the CPML memory.
__device__ __forceinline__ float2 curl2(const float4* t) { return __ldg(reinterpret_cast<const float2*>(t)); }
__device__ __forceinline__ float2 psi2(const float4* t) { return __ldg(reinterpret_cast<const float2*>(t) + 1); }
// The curl coefficients along x of the nodes of a mask, entry r for node r.
__device__ __forceinline__ void curl_x(Quad& c0, Quad& c1, const float4* t, int mask) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
        if (mask >> r & 1) {
            const float2 f = curl2(t + r);
            c0.v[r] = f.x; c1.v[r] = f.y;
        }
}
// The row of node r of a quad.
__device__ __forceinline__ int row_at(const uint2& c, int r) { return (int)((r < 2 ? c.x : c.y) >> (16 * (r & 1)) & 0xffffu); }
__device__ __forceinline__ float pick(const Quad& q, int r) { return r == 0 ? q.v[0] : r == 1 ? q.v[1] : r == 2 ? q.v[2] : q.v[3]; }

__device__ __forceinline__ void prefetch_l1(const void* a) { asm volatile("prefetch.global.L1 [%0];" ::"l"(a)); }
__device__ __forceinline__ void cp_async16(float4* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ Quad quad_of(const float4& f) { return Quad{f.x, f.y, f.z, f.w}; }

// The march of one thread's quad at tile row `row`, first column `col`. kEdge: the tile (halo
// included) meets a CPML slab or a wall in x (wx) or y (wy), or the chunk one in z; without it no
// node does. kMat: rows other than the background's lie in a slab or on a low wall (without it the
// few that may, beside general nodes, take the slow path). Their quads of one row take the background's
// way through the step, with coefficients from the tables: node by node, a load waiting for the one
// before it, they held their tiles up (a half space and boxes through the slabs, us a step: 225^3 300 -> 244,
// 320^3 567 -> 444; with the chunks of plan_sweep 237 and 419). kDesign (with kMat): the grid has a design
// region, whose rows' E coefficients are each node's own (StepParams::dcoef): on the slow path a region of
// 256^3 cells in 512^3 cost 2.4 ms of a step's 3.7, now 0.14 of 1.49. A kernel of their own, as the test for
// such rows cost the others 1 to 8 %.
template <typename Idx, bool kEdge, int kKind, bool kWide>
__device__ __forceinline__ void march(const SweepArgs& A, SweepSmem<Idx>& S, int x0, int y0, int k0, int k1, int row,
                                      int col, bool own, bool wx, bool wy) {
    constexpr bool kMat = kKind != kSweepPlain, kDesign = kKind == kSweepDesign;
    const StepParams& p = A.p;
    const DeviceGrid& g = p.g;
    const FieldPtrs& fo = A.fo;
    const BgNode& B = p.bgn;
    const float* const pin = A.pin.base;
    float* const pout = A.pout.base;
    const int i = x0 + col, j = y0 + row, t = row * W + col, te = row * WE + col, kfirst = k0 - 1;
    // nodes of the quad (bit r) in the grid, below the high x wall, off both x walls, in an x slab
    int in4 = 15, lt4 = 15, in_x = 15, xs = 0, xslow = 0;
    bool ylt = true, yin = true, ys = false;
    Idx qx = 0, sx = 0, dx = 0, qy = 0, sy = 0, dy = 0;  // CPML memory of the x and y faces at plane k (advanced with it):
                                                       // E array 0 of the first node, the arrays' stride, the planes'
    if (kEdge) {
        if (wx) {
            in4 = i + 4 <= g.nx ? 15 : i < g.nx ? (1 << (g.nx - i)) - 1 : 0;
            lt4 = i + 4 <= g.nx - 1 ? 15 : i < g.nx - 1 ? (1 << (g.nx - 1 - i)) - 1 : 0;
            in_x = i > 0 ? lt4 : lt4 & 14;
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (in_slab(i + r, g.nx, g.pxn, g.pxp)) xs |= 1 << r;
        }
        if (j >= g.ny) in4 = 0;
        xs &= in4;
        // a quad that meets both x slabs: the high side's nodes take the slow path
        if (xs && i < g.pxn && i + 3 >= g.nx - g.pxp) {
            xslow = xs & ~((1 << max(0, min(4, g.pxn - i))) - 1);
            xs &= ~xslow;
        }
        ylt = j < g.ny - 1;
        yin = j > 0 && ylt;
        ys = wy && in4 && in_slab(j, g.ny, g.pyn, g.pyp);
        if (xs) {
            const bool lo = i < g.pxn;
            const int w = lo ? g.pxn : g.pxp;
            sx = (Idx)p.psi_stride[lo ? 0 : 1];
            dx = (Idx)g.ny * (Idx)w;
            qx = (Idx)p.psi_off[lo ? 0 : 1] + (Idx)k0 * dx + (Idx)j * (Idx)w + (Idx)(lo ? i : i - (g.nx - g.pxp));
        }
        if (ys) {
            const bool lo = j < g.pyn;
            const int w = lo ? g.pyn : g.pyp;
            sy = (Idx)p.psi_stride[lo ? 2 : 3];
            dy = (Idx)w * (Idx)g.pitch;
            qy = (Idx)p.psi_off[lo ? 2 : 3] + (Idx)k0 * dy + (Idx)(lo ? j : j - (g.ny - g.pyp)) * (Idx)g.pitch + (Idx)i;
        }
    }
    own = own && in4;
    // kMat: the slab coefficients of row c (SlabRows); lx, ly, lz(k): the slab planes of the quad's first
    // node, its row and plane k
    const int Lx = g.pxn + g.pxp, Ly = g.pyn + g.pyp, Lz = g.pzn + g.pzp;
    const int lx = i < g.pxn ? i : i - (g.nx - Lx), ly = j < g.pyn ? j : j - (g.ny - Ly);
    auto lz = [&](int k) { return k < g.pzn ? k : k - (g.nz - Lz); };
    const SlabRows& SR = p.rows;
    const Idx nij = (Idx)j * (Idx)g.pitch + (Idx)i;
    Idx n = (Idx)k0 * (Idx)g.plane + nij;
    const int bgm = p.bg.mat;
    float4* const ps = &S.psi[0][threadIdx.x];

    auto issue = [&](int k, int s) {
        unsigned char* d = S.stage[s];
        mbar_expect_tx(&S.bar[s], 3 * H_TX + 3 * E_TX + M_TX);
        for (int c = 0; c < 3; ++c) tma_load_3d(d + c * H_BYTES, &A.maps.h[c], &S.bar[s], x0 - 4, y0 - 1, k);
        for (int c = 0; c < 3; ++c) tma_load_3d(d + 3 * H_BYTES + c * E_BYTES, &A.maps.e[c], &S.bar[s], x0, y0, k);
        tma_load_3d(d + 3 * H_BYTES + 3 * E_BYTES, &A.maps.rec, &S.bar[s], x0, y0, k);
    };
    // Fetch the old CPML memory of E(k) and H(k-1) into the thread's slots (qk: its y face's offset at plane k).
    auto fetch_psi = [&](int k, Idx qk) {
        if (ys) {
            cp_async16(ps + kPsiE * NTH, pin + qk);
            cp_async16(ps + (kPsiE + 1) * NTH, pin + qk + sy);
            if (own && k > k0) {
                cp_async16(ps + kPsiH * NTH, pin + qk - dy + 2 * sy);
                cp_async16(ps + (kPsiH + 1) * NTH, pin + qk - dy + 3 * sy);
            }
        } else {
            const PsiAt<Idx> z = S.zo[k - kfirst], zh = S.zo[k - 1 - kfirst];
            if (z.on && in4) {
                cp_async16(ps + kPsiE * NTH, pin + z.base + nij);
                cp_async16(ps + (kPsiE + 1) * NTH, pin + z.base + nij + z.stride);
            }
            if (zh.on && own && k > k0) {
                cp_async16(ps + kPsiH * NTH, pin + zh.base + nij + 2 * zh.stride);
                cp_async16(ps + (kPsiH + 1) * NTH, pin + zh.base + nij + 3 * zh.stride);
            }
        }
        cp_async_commit();
    };
    if (kEdge) fetch_psi(k0, qy);
    // plane k0 - 1: only its Hx and Hy are needed (loaded by the kernel into stage 0)
    bool ok = mbar_wait(&S.bar[0], 0);
    Quad hxp = lds4(f32(S.stage[0]) + t + H_OFF), hyp = lds4(f32(S.stage[0]) + t + H_OFF + HF);  // old H of plane k - 1
    Quad hzp{};
    uint2 cp = make_uint2(0, 0);  // the nodes' rows there
    int s = 1;
    uint32_t parity = 0;  // of stage s
#pragma unroll 1
    for (int k = k0;; ++k) {
        if (__syncthreads_or(!ok)) {
            // a plane never arrived: record it, wait (bounded) for the copies that may still be in flight, exit
            if (kEdge) cp_async_wait_all();
            if (threadIdx.x == 0) {
                atomic_flag(p.status, 1);
                for (int q = SweepRing::drain_begin(k); q < SweepRing::drain_end(k, k1, NST); ++q)
                    mbar_wait(&S.bar[SweepRing::stage(q - kfirst, NST)], SweepRing::parity(q - kfirst, NST));
            }
            __syncthreads();
            return;
        }
        if (k > k1) return;
        if (threadIdx.x == 0 && k + NST - 1 <= k1) {
            fence_proxy_async();  // generic reads of the recycled stage precede the async writes
            issue(k + NST - 1, s == 0 ? NST - 1 : s - 1);
        }
        const int q = k - kfirst;
        const bool store_e = own && k < k1;
        bool zs = false, zsh = false, kin = true, klt = true, klh = true;
        if (kEdge) {
            zs = S.zo[q].on && in4;
            zsh = S.zo[q - 1].on;
            klt = k < g.nz - 1;
            klh = k - 1 < g.nz - 1;
            kin = k > 0 && klt;
        }
        const float* T = f32(S.stage[s]) + t;
        const float* TE = f32(S.stage[s]) + E_OFF + te;
        float* en = &S.enew[k & 1][0][te];
        const float* ep = &S.enew[(k - 1) & 1][0][te];
        Quad xq0, xq1;
        if (kEdge && xs) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (xs >> r & 1) {
                    xq0.v[r] = __ldg(pin + (qx + r));
                    xq1.v[r] = __ldg(pin + (qx + sx + r));
                }
        }
        ok = mbar_wait(&S.bar[s], parity);
        if (!ok) continue;  // the stage holds anything: no row of it may index a table, nothing is stored
        const Quad hx = lds4(T + H_OFF), hy = lds4(T + H_OFF + HF), hz = lds4(T + H_OFF + 2 * HF);
        const uint2 cw = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(S.stage[s] + 3 * H_BYTES + 3 * E_BYTES) + t);
        Quad vx, vy, vz;
        int slow = 0;  // nodes on the slow path: bits 0-3 E(k), bits 4-7 H(k-1)
        // ---- E(k) ----
        {
            const Quad hzj = lds4(T + H_OFF + 2 * HF - W), hxj = lds4(T + H_OFF - W);
            const float hzi = T[H_OFF + 2 * HF - 1], hyi = T[H_OFF + HF - 1];
            vx = lds4(TE); vy = lds4(TE + EF); vz = lds4(TE + 2 * EF);
            const int c0 = (int)(cw.x & 0xffffu);
            bool mixed = false;
            const bool bg = kEdge && !kMat ? true : c0 == bgm;
            if (cw.x == cw.y && cw.x == (uint32_t)c0 * 0x10001u &&
                (kEdge ? (kMat ? c0 < (kDesign ? p.des_row0 : p.src_row0) : c0 == bgm) && !xslow : c0 < (kDesign ? p.des_row0 : p.src_row0))) {
                // one row for the quad (in tiles at the edge without kMat, the background's)
                float4 a = make_float4(B.ea[0], B.ec[0], B.ec[1], 0.f), b = make_float4(B.ea[1], B.ec[2], B.ec[3], 0.f);
                float4 d = make_float4(B.ea[2], B.ec[4], B.ec[5], 0.f);
                if (!bg) {
                    const MatCoef* mc = p.coef + c0;
                    a = __ldg(&mc->e[0]); b = __ldg(&mc->e[1]); d = __ldg(&mc->e[2]);
                }
                Quad x0c = {b.z, b.z, b.z, b.z}, x1c = {d.y, d.y, d.y, d.y};
                if (kEdge && bg) {  // curl coefficients along a slab's axis, over kappa
                    if (ys) { a.y = S.ye[row].x; d.z = S.ye[row].y; }
                    if (zs) { a.z = S.ze[q].x; b.y = S.ze[q].y; }
                    if (xs) { x0c = lds4(&S.xe[0][col]); x1c = lds4(&S.xe[1][col]); }
                } else if (kEdge) {
                    if (ys) { const float2 f = curl2(SR.e[1] + c0 * Ly + ly); a.y = f.x; d.z = f.y; }
                    if (zs) { const float2 f = curl2(SR.e[2] + c0 * Lz + lz(k)); a.z = f.x; b.y = f.y; }
                    if (xs) curl_x(x0c, x1c, SR.e[0] + c0 * Lx + lx, xs);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    vx.v[r] = upd3(a.x, vx.v[r], a.y, __fsub_rn(hz.v[r], hzj.v[r]), a.z, __fsub_rn(hy.v[r], hyp.v[r]));
                    vy.v[r] = upd3(b.x, vy.v[r], b.y, __fsub_rn(hx.v[r], hxp.v[r]), x0c.v[r], __fsub_rn(hz.v[r], r ? hz.v[r - 1] : hzi));
                    vz.v[r] = upd3(d.x, vz.v[r], x1c.v[r], __fsub_rn(hy.v[r], r ? hy.v[r - 1] : hyi), d.z, __fsub_rn(hx.v[r], hxj.v[r]));
                }
            } else {
                // rows per node; in a slab background nodes take the tabulated curl coefficients, and
                // without kMat the others the slow path
                mixed = true;
                // where a component's E coefficients of node r (row c) lie
                long long dq = 0, dn = 0;
                if (kDesign) {
                    const int* d = p.dbox;
                    const long long bx = d[3] - d[0] + 1, by = d[4] - d[1] + 1;
                    dn = bx * by * (d[5] - d[2] + 1);
                    dq = ((k - d[2]) * by + (j - d[1])) * bx + (i - d[0]);
                }
                auto e_row = [&](int c, int r, int comp) {
                    return kDesign && c >= p.des_row0 && c < p.des_row1 ? p.dcoef + (comp * dn + dq + r) : &p.coef[c].e[comp];
                };
                if constexpr (kWide || !kEdge) {
                    // (component by component, so that the four nodes' loads are in flight together: the quads
                    // of a material's surface decide how long the plane takes. Tiles at the edge have no
                    // registers left for it with three CTAs an SM, and spills cost more: 512^3 28.4 -> 28.1 ms for
                    // 20 steps with it in the interior tiles)
                    int c[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        c[r] = row_at(cw, r);
                        if (c[r] >= kRecGeneral || (kEdge && ((!kMat && c[r] != bgm && (ys || zs || (xs >> r & 1))) || (xslow >> r & 1)))) {
                            slow |= 1 << r;
                            c[r] = bgm;
                        }
                    }
                    // the curl coefficients along the axes whose slab the nodes lie in, over kappa
                    auto slab_e = [&](Quad& f, bool in, const float4* T, int L, int l, int w, float bg) {
                        if (kEdge && in)
#pragma unroll
                            for (int r = 0; r < 4; ++r) f.v[r] = kMat ? __ldg(&T[c[r] * L + l].x + w) : bg;
                    };
                    auto slab_ex = [&](Quad& f, int w) {
                        if (kEdge && xs)
#pragma unroll
                            for (int r = 0; r < 4; ++r)
                                if (xs >> r & 1) f.v[r] = kMat ? __ldg(&SR.e[0][c[r] * Lx + lx + r].x + w) : S.xe[w][col + r];
                    };
                    Quad f0, f1, f2;
                    auto rows = [&](int comp) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const float4 f = __ldg(e_row(c[r], r, comp));
                            f0.v[r] = f.x; f1.v[r] = f.y; f2.v[r] = f.z;
                        }
                    };
                    rows(0);
                    slab_e(f1, ys, SR.e[1], Ly, ly, 0, S.ye[row].x);
                    slab_e(f2, zs, SR.e[2], Lz, lz(k), 0, S.ze[q].x);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        vx.v[r] = upd3(f0.v[r], vx.v[r], f1.v[r], __fsub_rn(hz.v[r], hzj.v[r]), f2.v[r], __fsub_rn(hy.v[r], hyp.v[r]));
                    rows(1);
                    slab_e(f1, zs, SR.e[2], Lz, lz(k), 1, S.ze[q].y);
                    slab_ex(f2, 0);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        vy.v[r] = upd3(f0.v[r], vy.v[r], f1.v[r], __fsub_rn(hx.v[r], hxp.v[r]), f2.v[r],
                                       __fsub_rn(hz.v[r], r ? hz.v[r - 1] : hzi));
                    rows(2);
                    slab_ex(f1, 1);
                    slab_e(f2, ys, SR.e[1], Ly, ly, 1, S.ye[row].y);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        vz.v[r] = upd3(f0.v[r], vz.v[r], f1.v[r], __fsub_rn(hy.v[r], r ? hy.v[r - 1] : hyi), f2.v[r],
                                       __fsub_rn(hx.v[r], hxj.v[r]));
                        if (c[r] >= p.src_row0) {  // lumped source edge (fdtdrav.h:728)
                            const SrcRow sr = p.src_rows[c[r] - p.src_row0];
                            vz.v[r] = __fmaf_rn(sr.cezj, sweep_sig(A, sr.source), vz.v[r]);
                        }
                    }
                } else {
                    // (their rows on the way to L1 together, E's and H's, which the next plane step wants: the loads
                    // below come one row after the other)
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const char* a = reinterpret_cast<const char*>(p.coef + (row_at(cw, r) < kRecGeneral ? row_at(cw, r) : 0));
                        prefetch_l1(a);
                        prefetch_l1(a + 32);
                        prefetch_l1(a + 64);
                    }
                    int cur = -1;
                    float4 a{}, b{}, d{};
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int c = row_at(cw, r);
                        const bool x = kEdge && (xs >> r & 1);
                        if (c >= kRecGeneral || (kEdge && ((!kMat && c != bgm && (ys || zs || x)) || (xslow >> r & 1)))) {
                            slow |= 1 << r;
                            continue;
                        }
                        if (c != cur) {
                            a = __ldg(e_row(c, r, 0)); b = __ldg(e_row(c, r, 1)); d = __ldg(e_row(c, r, 2));
                            cur = kDesign && c >= p.des_row0 && c < p.des_row1 ? -1 : c;  // (a design row's are the node's own)
                            if (!kMat || c == bgm) {
                                if (kEdge && ys) { a.y = S.ye[row].x; d.z = S.ye[row].y; }
                                if (kEdge && zs) { a.z = S.ze[q].x; b.y = S.ze[q].y; }
                            } else if (kEdge) {
                                if (ys) { const float4 f = __ldg(SR.e[1] + c * Ly + ly); a.y = f.x; d.z = f.y; }
                                if (zs) { const float4 f = __ldg(SR.e[2] + c * Lz + lz(k)); a.z = f.x; b.y = f.y; }
                            }
                        }
                        float xb = b.z, xd = d.y;
                        if (x) {
                            if (!kMat || c == bgm) {
                                xb = S.xe[0][col + r]; xd = S.xe[1][col + r];
                            } else {
                                const float4 f = __ldg(SR.e[0] + c * Lx + lx + r);
                                xb = f.x; xd = f.y;
                            }
                        }
                        vx.v[r] = upd3(a.x, vx.v[r], a.y, __fsub_rn(hz.v[r], hzj.v[r]), a.z, __fsub_rn(hy.v[r], hyp.v[r]));
                        vy.v[r] = upd3(b.x, vy.v[r], b.y, __fsub_rn(hx.v[r], hxp.v[r]), xb, __fsub_rn(hz.v[r], r ? hz.v[r - 1] : hzi));
                        vz.v[r] = upd3(d.x, vz.v[r], xd, __fsub_rn(hy.v[r], r ? hy.v[r - 1] : hyi), d.z, __fsub_rn(hx.v[r], hxj.v[r]));
                        if (c >= p.src_row0) {  // lumped source edge (fdtdrav.h:728)
                            const SrcRow sr = p.src_rows[c - p.src_row0];
                            vz.v[r] = __fmaf_rn(sr.cezj, sweep_sig(A, sr.source), vz.v[r]);
                        }
                    }
                }
                slow &= in4;
                if (kEdge && k >= g.nz) slow = 0;
            }
            if (kEdge) {
                cp_async_wait_all();
                const bool wall = in_x != 15 || !yin || !kin;
                int mx = 15, my = 15, mz = 15;
                if (wall) {
                    mx = yin && kin ? lt4 : 0;
                    my = ylt && kin ? in_x : 0;
                    mz = yin && klt ? in_x : 0;
                }
                const int st = store_e ? in4 & ~slow : 0;
                // v0 and v1 plus the quad's CPML memory u0, u1 along an axis (factors b0, b1, or its rows')
                auto add = [&](Quad& v0, Quad& v1, const Quad& u0, const Quad& u1, float b0, float b1, const float4* T, int L, int l,
                               int dl, int nodes) {
                    if (kMat && !mixed && !bg) {  // the quad's row's (the same on every plane of the slabs)
                        const float2 f = psi2(T + c0 * L);
                        b0 = f.x; b1 = f.y;
                    }
                    if (kMat && mixed) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const int c = row_at(cw, r);
                            if (c < kRecGeneral && (nodes >> r & 1)) {
                                const float4 f = __ldg(T + c * L + l + r * dl);
                                v0.v[r] = psi_add(v0.v[r], f.z, u0.v[r]);
                                v1.v[r] = psi_add(v1.v[r], f.w, u1.v[r]);
                            }
                        }
                        return;
                    }
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (nodes >> r & 1) {
                            v0.v[r] = psi_add(v0.v[r], b0, u0.v[r]);
                            v1.v[r] = psi_add(v1.v[r], b1, u1.v[r]);
                        }
                };
                if (xs) {  // fdtdrav.h:752-785
                    const Quad b = lds4(&S.xe[2][col]), c = lds4(&S.xe[3][col]);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (xs >> r & 1) {
                            xq0.v[r] = psi_upd(b.v[r], xq0.v[r], c.v[r], __fsub_rn(hz.v[r], r ? hz.v[r - 1] : hzi));
                            xq1.v[r] = psi_upd(b.v[r], xq1.v[r], c.v[r], __fsub_rn(hy.v[r], r ? hy.v[r - 1] : hyi));
                            if (st & my & (1 << r)) pout[qx + r] = xq0.v[r];
                            if (st & mz & (1 << r)) pout[qx + sx + r] = xq1.v[r];
                        }
                    add(vy, vz, xq0, xq1, B.ce[0], B.ce[1], SR.e[0], Lx, lx, 1, xs);
                }
                if (ys) {  // fdtdrav.h:790-827
                    const float b = S.ye[row].z, c = S.ye[row].w;
                    Quad u = quad_of(ps[kPsiE * NTH]), w = quad_of(ps[(kPsiE + 1) * NTH]);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        u.v[r] = psi_upd(b, u.v[r], c, __fsub_rn(hz.v[r], hzj.v[r]));
                        w.v[r] = psi_upd(b, w.v[r], c, __fsub_rn(hx.v[r], hxj.v[r]));
                    }
                    st_mask2(pout + qy, pout + qy + sy, u, w, st & mx, st & mz);
                    add(vx, vz, u, w, B.ce[2], B.ce[3], SR.e[1], Ly, ly, 0, 15);
                }
                if (zs) {  // fdtdrav.h:829-911
                    const float b = S.ze[q].z, c = S.ze[q].w;
                    const Idx at = S.zo[q].base + nij;
                    Quad u, w;
                    if (ys) { u = ldg4(pin + at); w = ldg4(pin + at + S.zo[q].stride); }
                    else { u = quad_of(ps[kPsiE * NTH]); w = quad_of(ps[(kPsiE + 1) * NTH]); }
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        u.v[r] = psi_upd(b, u.v[r], c, __fsub_rn(hy.v[r], hyp.v[r]));
                        w.v[r] = psi_upd(b, w.v[r], c, __fsub_rn(hx.v[r], hxp.v[r]));
                    }
                    st_mask2(pout + at, pout + at + S.zo[q].stride, u, w, st & mx, st & my);
                    add(vx, vy, u, w, B.ce[4], B.ce[5], SR.e[2], Lz, lz(k), 0, 15);
                }
                if (wall) {  // components the walls keep
                    const Quad ex = lds4(TE), ey = lds4(TE + EF), ez = lds4(TE + 2 * EF);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (!(mx >> r & 1)) vx.v[r] = ex.v[r];
                        if (!(my >> r & 1)) vy.v[r] = ey.v[r];
                        if (!(mz >> r & 1)) vz.v[r] = ez.v[r];
                    }
                }
            }
        }
        st4(en, vx);
        st4(en + NF, vy);
        st4(en + 2 * NF, vz);
        if (store_e) {
            const int st = in4 & ~slow;
            st_mask3(fo.ex + n, fo.ey + n, fo.ez + n, vx, vy, vz, st);
        }
        // ---- H(k-1) ----
        if (k > k0 && own) {
            const int kh = k - 1;
            const Idx gx = qx - dx + 2 * sx;
            if (kEdge && xs) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (xs >> r & 1) {
                        xq0.v[r] = __ldg(pin + (gx + r));
                        xq1.v[r] = __ldg(pin + (gx + sx + r));
                    }
            }
            // differences of E: along z, y and x
            const Quad ex = lds4(ep), ey = lds4(ep + NF), ez = lds4(ep + 2 * NF);
            const Quad ezj = lds4(ep + 2 * NF + WE), exj = lds4(ep + WE);
            const float ezi = ep[2 * NF + 4], eyi = ep[NF + 4];
            const bool low_jk = kEdge && (j == 0 || kh == 0);  // faces on a low wall take the default entry
            Quad ux = hxp, uy = hyp, uz = hzp;
            bool one = cp.x == cp.y && cp.x == (cp.x & 0xffffu) * 0x10001u, mixed = false;  // one row for the quad
            int c0 = (int)(cp.x & 0xffffu);
            if (kMat && p.h_bg && !((cp.x | cp.y) & kRecGeneral * 0x10001u)) { c0 = bgm; one = true; }
            // the row that component `comp` of node r (row c) takes: the default entry's on a low wall
            auto hrow = [&](int c, int r, int comp) {
                if (!kEdge || !kMat) return c;
                return (comp == 0 ? i + r == 0 : comp == 1 ? j == 0 : kh == 0) ? kDefaultEntry : c;
            };
            // entry (row of component p, row of component q) of an axis's slab coefficients
            auto slab_h = [&](const float4* T, int L, int l, int rp, int rq) {
                float4 f = __ldg(T + rp * L + l);
                if (rq != rp) { const float4 o = __ldg(T + rq * L + l); f.y = o.y; f.w = o.w; }
                return f;
            };
            const bool table = c0 == bgm && (!low_jk || B.low_ok);  // the tabulated coefficients apply
            const bool bg = kEdge && !kMat ? true : c0 == bgm;
            // one row for the quad: the background's where its tabulated coefficients apply, with kMat another
            // one off the low walls
            if (one && (kEdge ? (kMat && !bg ? c0 < kRecGeneral && !low_jk && i > 0 : table && (i > 0 || B.low_ok)) && !xslow : c0 < kRecGeneral)) {
                float4 a = make_float4(B.ha[0], B.hc[0], B.hc[1], 0.f), b = make_float4(B.ha[1], B.hc[2], B.hc[3], 0.f);
                float4 d = make_float4(B.ha[2], B.hc[4], B.hc[5], 0.f);
                if (!bg) {
                    a = __ldg(&p.coef[c0].h[0]); b = __ldg(&p.coef[c0].h[1]); d = __ldg(&p.coef[c0].h[2]);
                }
                Quad x0c = {b.y, b.y, b.y, b.y}, x1c = {d.z, d.z, d.z, d.z};
                if (kEdge && bg) {
                    if (ys) { a.z = S.yh[row].x; d.y = S.yh[row].y; }
                    if (zsh) { a.y = S.zh[q - 1].x; b.z = S.zh[q - 1].y; }
                    if (xs) { x0c = lds4(&S.xh[0][col]); x1c = lds4(&S.xh[1][col]); }
                } else if (kEdge) {
                    if (ys) { const float2 f = curl2(SR.h[1] + c0 * Ly + ly); a.z = f.x; d.y = f.y; }
                    if (zsh) { const float2 f = curl2(SR.h[2] + c0 * Lz + lz(kh)); a.y = f.x; b.z = f.y; }
                    if (xs) curl_x(x0c, x1c, SR.h[0] + c0 * Lx + lx, xs);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    ux.v[r] = upd3_hx(a.x, ux.v[r], a.y, __fsub_rn(vy.v[r], ey.v[r]), a.z, __fsub_rn(ezj.v[r], ez.v[r]));
                    uy.v[r] = upd3(b.x, uy.v[r], x0c.v[r], __fsub_rn(r < 3 ? ez.v[r + 1] : ezi, ez.v[r]), b.z, __fsub_rn(vx.v[r], ex.v[r]));
                    uz.v[r] = upd3(d.x, uz.v[r], d.y, __fsub_rn(exj.v[r], ex.v[r]), x1c.v[r], __fsub_rn(r < 3 ? ey.v[r + 1] : eyi, ey.v[r]));
                }
            } else {
                mixed = true;
                if constexpr (kWide || !kEdge) {
                    int c[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        c[r] = row_at(cp, r);
                        const bool lw = kEdge && (low_jk || i + r == 0);
                        if (c[r] >= kRecGeneral || (kEdge && ((!kMat && ((c[r] != bgm && (ys || zsh || (xs >> r & 1) || lw)) || (lw && !B.low_ok))) ||
                                                              (xslow >> r & 1)))) {
                            slow |= 16 << r;
                            c[r] = bgm;
                        }
                    }
                    auto slab_q = [&](Quad& f, bool in, const float4* T, int L, int l, int w, int comp, float bg) {
                        if (kEdge && in)
#pragma unroll
                            for (int r = 0; r < 4; ++r) f.v[r] = kMat ? __ldg(&T[hrow(c[r], r, comp) * L + l].x + w) : bg;
                    };
                    auto slab_qx = [&](Quad& f, int w, int comp) {
                        if (kEdge && xs)
#pragma unroll
                            for (int r = 0; r < 4; ++r)
                                if (xs >> r & 1) f.v[r] = kMat ? __ldg(&SR.h[0][hrow(c[r], r, comp) * Lx + lx + r].x + w) : S.xh[w][col + r];
                    };
                    Quad f0, f1, f2;
                    auto rows = [&](int comp) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const float4 f = __ldg(&p.coef[hrow(c[r], r, comp)].h[comp]);
                            f0.v[r] = f.x; f1.v[r] = f.y; f2.v[r] = f.z;
                        }
                    };
                    rows(0);
                    slab_q(f1, zsh, SR.h[2], Lz, lz(kh), 0, 0, S.zh[q - 1].x);
                    slab_q(f2, ys, SR.h[1], Ly, ly, 0, 0, S.yh[row].x);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        ux.v[r] = upd3_hx(f0.v[r], ux.v[r], f1.v[r], __fsub_rn(vy.v[r], ey.v[r]), f2.v[r], __fsub_rn(ezj.v[r], ez.v[r]));
                    rows(1);
                    slab_qx(f1, 0, 1);
                    slab_q(f2, zsh, SR.h[2], Lz, lz(kh), 1, 1, S.zh[q - 1].y);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        uy.v[r] = upd3(f0.v[r], uy.v[r], f1.v[r], __fsub_rn(r < 3 ? ez.v[r + 1] : ezi, ez.v[r]), f2.v[r],
                                       __fsub_rn(vx.v[r], ex.v[r]));
                    rows(2);
                    slab_q(f1, ys, SR.h[1], Ly, ly, 1, 2, S.yh[row].y);
                    slab_qx(f2, 1, 2);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        uz.v[r] = upd3(f0.v[r], uz.v[r], f1.v[r], __fsub_rn(exj.v[r], ex.v[r]), f2.v[r],
                                       __fsub_rn(r < 3 ? ey.v[r + 1] : eyi, ey.v[r]));
                } else {
                    int cur = -1;
                    float4 a{}, b{}, d{};
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int c = row_at(cp, r);
                        const bool x = kEdge && (xs >> r & 1), lw = kEdge && (low_jk || (r == 0 && i == 0));
                        if (c >= kRecGeneral || (kEdge && ((!kMat && ((c != bgm && (ys || zsh || x || lw)) || (lw && !B.low_ok))) ||
                                                           (xslow >> r & 1)))) {
                            slow |= 16 << r;
                            continue;
                        }
                        const bool tab = !kMat || (c == bgm && (!lw || B.low_ok));
                        if (c != cur) {
                            a = __ldg(&p.coef[hrow(c, r, 0)].h[0]); b = __ldg(&p.coef[hrow(c, r, 1)].h[1]);
                            d = __ldg(&p.coef[hrow(c, r, 2)].h[2]);
                            cur = kEdge && kMat && r == 0 && i == 0 ? -1 : c;
                            if (tab) {
                                if (kEdge && ys) { a.z = S.yh[row].x; d.y = S.yh[row].y; }
                                if (kEdge && zsh) { a.y = S.zh[q - 1].x; b.z = S.zh[q - 1].y; }
                            } else if (kEdge) {
                                if (ys) { const float4 f = slab_h(SR.h[1], Ly, ly, hrow(c, r, 0), hrow(c, r, 2)); a.z = f.x; d.y = f.y; }
                                if (zsh) { const float4 f = slab_h(SR.h[2], Lz, lz(kh), hrow(c, r, 0), hrow(c, r, 1)); a.y = f.x; b.z = f.y; }
                            }
                        }
                        float xb = b.y, xd = d.z;
                        if (x) {
                            if (tab) {
                                xb = S.xh[0][col + r]; xd = S.xh[1][col + r];
                            } else {
                                const float4 f = slab_h(SR.h[0], Lx, lx + r, hrow(c, r, 1), hrow(c, r, 2));
                                xb = f.x; xd = f.y;
                            }
                        }
                        ux.v[r] = upd3_hx(a.x, ux.v[r], a.y, __fsub_rn(vy.v[r], ey.v[r]), a.z, __fsub_rn(ezj.v[r], ez.v[r]));
                        uy.v[r] = upd3(b.x, uy.v[r], xb, __fsub_rn(r < 3 ? ez.v[r + 1] : ezi, ez.v[r]), b.z, __fsub_rn(vx.v[r], ex.v[r]));
                        uz.v[r] = upd3(d.x, uz.v[r], d.y, __fsub_rn(exj.v[r], ex.v[r]), xd, __fsub_rn(r < 3 ? ey.v[r + 1] : eyi, ey.v[r]));
                    }
                }
                slow &= in4 | in4 << 4;
            }
            slow |= (slow & 15) << 4;  // H(k-1) of a node whose E(k) is still to come
            const int st = in4 & ~(slow >> 4);
            if (kEdge) {
                int mx = 15, my = 15, mz = 15;
                const bool wall = lt4 != 15 || !ylt || !klh;
                if (wall) {
                    mx = ylt && klh ? 15 : 0;
                    my = klh ? lt4 : 0;
                    mz = ylt ? lt4 : 0;
                }
                auto add = [&](Quad& v0, Quad& v1, const Quad& u0, const Quad& u1, float b0, float b1, const float4* T, int L, int l,
                               int dl, int nodes, int p0, int p1) {
                    if (kMat && !mixed && !bg) {
                        const float2 f = psi2(T + c0 * L);
                        b0 = f.x; b1 = f.y;
                    }
                    if (kMat && mixed) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const int c = row_at(cp, r);
                            if (c < kRecGeneral && (nodes >> r & 1)) {
                                const float4 f = slab_h(T, L, l + r * dl, hrow(c, r, p0), hrow(c, r, p1));
                                v0.v[r] = psi_add(v0.v[r], f.z, u0.v[r]);
                                v1.v[r] = psi_add(v1.v[r], f.w, u1.v[r]);
                            }
                        }
                        return;
                    }
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (nodes >> r & 1) {
                            v0.v[r] = psi_add(v0.v[r], b0, u0.v[r]);
                            v1.v[r] = psi_add(v1.v[r], b1, u1.v[r]);
                        }
                };
                if (xs) {  // fdtdrav.h:401-442
                    const Quad b = lds4(&S.xh[2][col]), c = lds4(&S.xh[3][col]);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (xs >> r & 1) {
                            xq0.v[r] = psi_upd(b.v[r], xq0.v[r], c.v[r], __fsub_rn(r < 3 ? ez.v[r + 1] : ezi, ez.v[r]));
                            xq1.v[r] = psi_upd(b.v[r], xq1.v[r], c.v[r], __fsub_rn(r < 3 ? ey.v[r + 1] : eyi, ey.v[r]));
                            if (st & my & (1 << r)) pout[gx + r] = xq0.v[r];
                            if (st & mz & (1 << r)) pout[gx + sx + r] = xq1.v[r];
                        }
                    add(uy, uz, xq0, xq1, B.ch[0], B.ch[1], SR.h[0], Lx, lx, 1, xs, 1, 2);
                }
                if (ys) {  // fdtdrav.h:445-486
                    const float b = S.yh[row].z, c = S.yh[row].w;
                    Quad u = quad_of(ps[kPsiH * NTH]), w = quad_of(ps[(kPsiH + 1) * NTH]);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        u.v[r] = psi_upd(b, u.v[r], c, __fsub_rn(ezj.v[r], ez.v[r]));
                        w.v[r] = psi_upd(b, w.v[r], c, __fsub_rn(exj.v[r], ex.v[r]));
                    }
                    const Idx at = qy - dy + 2 * sy;
                    st_mask2(pout + at, pout + at + sy, u, w, st & mx, st & mz);
                    add(ux, uz, u, w, B.ch[2], B.ch[3], SR.h[1], Ly, ly, 0, 15, 0, 2);
                }
                if (zsh) {  // fdtdrav.h:489-562
                    const float b = S.zh[q - 1].z, c = S.zh[q - 1].w;
                    const Idx sz = S.zo[q - 1].stride, at = S.zo[q - 1].base + nij + 2 * sz;
                    Quad u, w;
                    if (ys) { u = ldg4(pin + at); w = ldg4(pin + at + sz); }
                    else { u = quad_of(ps[kPsiH * NTH]); w = quad_of(ps[(kPsiH + 1) * NTH]); }
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        u.v[r] = psi_upd(b, u.v[r], c, __fsub_rn(vy.v[r], ey.v[r]));
                        w.v[r] = psi_upd_hyz(b, w.v[r], c, __fsub_rn(vx.v[r], ex.v[r]));
                    }
                    st_mask2(pout + at, pout + at + sz, u, w, st & mx, st & my);
                    add(ux, uy, u, w, B.ch[4], B.ch[5], SR.h[2], Lz, lz(kh), 0, 15, 0, 1);
                }
                if (wall) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (!(mx >> r & 1)) ux.v[r] = hxp.v[r];
                        if (!(my >> r & 1)) uy.v[r] = hyp.v[r];
                        if (!(mz >> r & 1)) uz.v[r] = hzp.v[r];
                    }
                }
            }
            const Idx nh = n - (Idx)g.plane;
            st_mask3(fo.hx + nh, fo.hy + nh, fo.hz + nh, ux, uy, uz, st);
        }
        if (slow) {
#pragma unroll 1
            for (int r = 0; r < 4; ++r) {
                const int bits = (slow >> r & 1) | (slow >> (3 + r) & 2);
                if (!bits) continue;
                const uint32_t c = (r < 2 ? cp.x : cp.y) >> (16 * (r & 1)) & 0xffffu;
                slow_node<Idx>(&A, &S, bits | (own ? 4 : 0) | (store_e ? 8 : 0), k, s, i + r, j, t + r, te + r, pick(hxp, r), pick(hyp, r),
                               pick(hzp, r), (int)c);
            }
        }
        hxp = lds4(T + H_OFF); hyp = lds4(T + H_OFF + HF); hzp = lds4(T + H_OFF + 2 * HF);  // (again: not kept in registers)
        cp = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(S.stage[s] + 3 * H_BYTES + 3 * E_BYTES) + t);
        n += (Idx)g.plane;
        if (kEdge) {
            qx += dx;
            qy += dy;
            if (k < k1) fetch_psi(k + 1, qy);
        }
        if (++s == NST) { s = 0; parity ^= 1u; }
    }
}

}  // namespace

template <typename Idx, int kKind, bool kWide>
__global__ void __launch_bounds__(NTH, kWide ? 2 : 3) k_sweep(const __grid_constant__ SweepArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SweepSmem<Idx>& S = *reinterpret_cast<SweepSmem<Idx>*>(smem_raw);
    const StepParams& p = A.p;
    const DeviceGrid& g = p.g;
    const int tid = threadIdx.x;
    // item: chunk outer, tiles inner (x fastest), so the CTAs in flight work on neighbouring planes; every
    // other step from the top down, beginning with what the step before wrote last and L2 still holds
    // (225 x 190 x 163 3.27 -> 3.24 ms for 24 steps)
    int b = blockIdx.x;
    const int bx = b % A.sg.nbx;
    b /= A.sg.nbx;
    const int by = b % A.sg.nby, ch = A.m & 1 ? A.sg.chunks() - 1 - b / A.sg.nby : b / A.sg.nby;
    const int x0 = bx * TX, y0 = by * TY;
    const int k0 = A.sg.chunk(ch), k1 = A.sg.chunk(ch + 1);
    const int kfirst = k0 - 1;  // the planes k0 - 1 .. k1, at most kMaxSweepPlanes (plan_sweep)

    // ---- per-column, per-row and per-plane tables ----
    if (tid == 0) {
        S.m = sweep_m(A);
        for (int q = 0; q < NST; ++q) mbar_init(&S.bar[q], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = tid; q < W; q += NTH) {
        const bool in = x0 + q < g.nx;
        const float4 e = in ? __ldg(p.te[0] + x0 + q) : none, h = in ? __ldg(p.th[0] + x0 + q) : none;
        S.xe[0][q] = e.x; S.xe[1][q] = e.y; S.xe[2][q] = e.z; S.xe[3][q] = e.w;
        S.xh[0][q] = h.x; S.xh[1][q] = h.y; S.xh[2][q] = h.z; S.xh[3][q] = h.w;
    }
    // (other threads than the ones above where there are enough)
    for (int r = NTH - 1 - tid; r < ER; r += NTH) {
        const bool in = y0 + r < g.ny;
        S.ye[r] = in ? __ldg(p.te[1] + y0 + r) : none;
        S.yh[r] = in ? __ldg(p.th[1] + y0 + r) : none;
    }
    for (int r = (tid + NTH - W) % NTH; r <= k1 - kfirst; r += NTH) {
        const int q = kfirst + r;
        const bool in = q >= 0 && q < g.nz;
        S.ze[r] = in ? __ldg(p.te[2] + q) : none;
        S.zh[r] = in ? __ldg(p.th[2] + q) : none;
        PsiAt<Idx> o{0, 0, 0, 0};
        if (in && in_slab(q, g.nz, g.pzn, g.pzp)) {
            const bool lo = q < g.pzn;
            o.base = (Idx)p.psi_off[lo ? 4 : 5] + (Idx)(lo ? q : q - (g.nz - g.pzp)) * (Idx)g.plane;
            o.stride = (Idx)p.psi_stride[lo ? 4 : 5];
            o.on = 1;
        }
        S.zo[r] = o;
    }
    __syncthreads();
    grid_dependency_wait();  // the previous step wrote what this one reads
    grid_launch_dependents();
    if (tid == 0) {
        mbar_expect_tx(&S.bar[0], 2 * H_TX);
        for (int c = 0; c < 2; ++c) tma_load_3d(S.stage[0] + c * H_BYTES, &A.maps.h[c], &S.bar[0], x0 - 4, y0 - 1, kfirst);
        for (int k = k0; k <= min(k1, k0 + NST - 2); ++k) {
            const int s = 1 + k - k0;
            unsigned char* d = S.stage[s];
            mbar_expect_tx(&S.bar[s], 3 * H_TX + 3 * E_TX + M_TX);
            for (int c = 0; c < 3; ++c) tma_load_3d(d + c * H_BYTES, &A.maps.h[c], &S.bar[s], x0 - 4, y0 - 1, k);
            for (int c = 0; c < 3; ++c) tma_load_3d(d + 3 * H_BYTES + c * E_BYTES, &A.maps.e[c], &S.bar[s], x0, y0, k);
            tma_load_3d(d + 3 * H_BYTES + 3 * E_BYTES, &A.maps.rec, &S.bar[s], x0, y0, k);
        }
    }
    // Probes outside the CPML slabs hold the step's final values, so they are read from the finished
    // fields: here the step before (its fields are this step's input), and after a call's last step by
    // k_sample_probes. Probes inside a slab are sampled by the slow path, before the CPML correction.
    if (A.late)
        for (long long q = (long long)blockIdx.x * NTH + tid; q < A.n_probes_at; q += (long long)gridDim.x * NTH)
            sample_at(A.probes[q], A.fi, p, S.m - 1);
    // own quads, then those of the halo row and the halo column (spare threads repeat the last one)
    const bool own = tid < NOWN;
    const int h = min(tid - NOWN, QX + TY - 1);
    const int row = own ? tid / QX : h < QX ? TY : h - QX, col = own ? tid % QX * 4 : h < QX ? h * 4 : TX;
    const bool wx = x0 < max(g.pxn, 1) || x0 + TX >= min(g.nx - g.pxp, g.nx - 1);
    const bool wy = y0 < max(g.pyn, 1) || y0 + TY >= min(g.ny - g.pyp, g.ny - 1);
    const bool wz = k0 < max(g.pzn, 1) || k1 >= min(g.nz - g.pzp, g.nz - 1);  // E(k0) .. E(k1), H(k0) .. H(k1 - 1)
    if (wx || wy || wz) march<Idx, true, kKind, kWide>(A, S, x0, y0, k0, k1, row, col, own, wx, wy);
    else march<Idx, false, kKind, kWide>(A, S, x0, y0, k0, k1, row, col, own, false, false);
}

template <typename Idx>
constexpr int sweep_smem() { return (int)sizeof(SweepSmem<Idx>); }

// The kernel for a grid's kind; 64-bit offsets have no two-CTA form (such grids fill the device).
using SweepKernel = void (*)(const SweepArgs);
template <typename Idx, bool kWide>
SweepKernel sweep_kernel(int kind) {
    return kind == kSweepPlain ? SweepKernel(k_sweep<Idx, kSweepPlain, kWide>)
           : kind == kSweepMat ? SweepKernel(k_sweep<Idx, kSweepMat, kWide>)
                               : SweepKernel(k_sweep<Idx, kSweepDesign, kWide>);
}
cudaError_t sweep_configure() {
    cudaError_t e = cudaSuccess;
    auto configure = [&](SweepKernel k, int smem) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    };
    for (int kind : {kSweepPlain, kSweepMat, kSweepDesign}) {
        configure(sweep_kernel<uint32_t, false>(kind), sweep_smem<uint32_t>());
        configure(sweep_kernel<uint32_t, true>(kind), sweep_smem<uint32_t>());
        configure(sweep_kernel<unsigned long long, false>(kind), sweep_smem<unsigned long long>());
    }
    return e;
}

__global__ void k_sample_probes(const __grid_constant__ StepParams p, const __grid_constant__ FieldPtrs f,
                                const ProbeAt* __restrict__ probes, int n, const long long* base, long long m) {
    grid_dependency_wait();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) sample_at(probes[q], f, p, base ? *base + m : m);
}

cudaError_t launch_sample_probes(const StepParams& p, const FieldPtrs& f, const ProbeAt* probes, int n, const long long* base,
                                 long long m, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    return launch_dependent(k_sample_probes, dim3((unsigned)(n + 127) / 128), dim3(128), 0, st, p, f, probes, n, base, m);
}

cudaError_t launch_sweep(const FusedMaps& maps, const StepParams& p, const FieldPtrs& fi, const FieldPtrs& fo,
                         const PsiSet& pin, const PsiSet& pout, const SweepPlan& sg, const SweepStep& ss, long long m,
                         cudaStream_t st) {
    SweepArgs args{maps, p, fo, pin, pout, sg, m, ss.base, fi, ss.probes, ss.n_probes, ss.late, {}};
    std::copy(ss.sig, ss.sig + kSweepSources, args.sig);
    const bool idx32 = p.g.plane * (long long)(p.g.nz + 1) < (1LL << 31) && p.psi_total < (1LL << 31);
    const unsigned ctas = (unsigned)(sg.nbx * sg.nby * sg.chunks());
    const bool wide = !ss.base && ctas <= kSweepWideCtas;
    const SweepKernel k = !idx32 ? sweep_kernel<unsigned long long, false>(ss.kind)
                          : wide ? sweep_kernel<uint32_t, true>(ss.kind)
                                 : sweep_kernel<uint32_t, false>(ss.kind);
    return launch_dependent(k, dim3(ctas), dim3(NTH), idx32 ? sweep_smem<uint32_t>() : sweep_smem<unsigned long long>(), st, args);
}

// Tensor maps of the sweep: H tiles with a one-node halo (x from 4 nodes before the tile: a TMA box
// starts on a 16-byte boundary), old-E and coefficient-row tiles. Coordinates outside the arrays
// load as zeros.
int encode_sweep_maps(FusedMaps* out, const DeviceGrid& g, float* const h[3], float* const e[3], const uint16_t* rec,
                      void* encode_fn) {
    using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    const EncodeFn encode = reinterpret_cast<EncodeFn>(encode_fn);
    const cuuint64_t dims[3] = {(cuuint64_t)g.pitch, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
    const cuuint64_t fstr[2] = {(cuuint64_t)g.pitch * 4, (cuuint64_t)g.plane * 4};
    const cuuint64_t mstr[2] = {(cuuint64_t)g.pitch * 2, (cuuint64_t)g.plane * 2};
    const cuuint32_t hbox[3] = {W, HR, 1}, ebox[3] = {WE, ER, 1}, mbox[3] = {W, ER, 1}, es[3] = {1, 1, 1};
    auto map = [&](CUtensorMap* mp, CUtensorMapDataType t, void* base, const cuuint64_t* str, const cuuint32_t* box) {
        return encode(mp, t, 3, base, dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    for (int c = 0; c < 3; ++c)
        if (!map(&out->h[c], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, h[c], fstr, hbox) ||
            !map(&out->e[c], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, e[c], fstr, ebox))
            return -1;
    return map(&out->rec, CU_TENSOR_MAP_DATA_TYPE_UINT16, const_cast<uint16_t*>(rec), mstr, mbox) ? 0 : -1;
}

}  // namespace fdtd
