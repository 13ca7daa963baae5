// sweep_cells.cuh -- per-cell pieces of the fused sweeps that do not depend
// on how the field values reached the thread (registers or a TMA-staged
// shared-memory tile): CPML psi corrections and the Drude-Lorentz / gain
// updates looked up on their compacted lists.
#pragma once

#include "cells.cuh"

namespace cps {

// Rounding written out: one product, one sum or one fused multiply-add each, so
// that every kernel that holds an update computes the same bits, whatever the
// compiler would contract around it.
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }

// a F + b d1 c1 - b d2 c2 (bulk E and H updates, BasicFDTD.cpp:25-84)
template <typename T>
__device__ __forceinline__ T yee(T a, T F, T b, T d1, T c1, T d2, T c2)
{
    return rfma(-rmul(b, d2), c2, rfma(a, F, rmul(rmul(b, d1), c1)));
}
// the same in the Hz update's order of rounding
template <typename T>
__device__ __forceinline__ T yee_z(T a, T F, T b, T d1, T c1, T d2, T c2)
{
    return rfma(-rmul(b, d2), c2, rfma(rmul(b, d1), c1, rmul(a, F)));
}
// a F - b d1 c1 + b d2 c2
template <typename T>
__device__ __forceinline__ T yee_n(T a, T F, T b, T d1, T c1, T d2, T c2)
{
    return rfma(rmul(b, d2), c2, rfma(a, F, -rmul(rmul(b, d1), c1)));
}
// b psi + c d, and a component with +/- psi times its curl coefficient
template <typename T>
__device__ __forceinline__ T psi_new(T b, T psi, T c, T d) { return rfma(b, psi, rmul(c, d)); }
template <typename T>
__device__ __forceinline__ T psi_add(T F, T a, T cc) { return rfma(a, cc, F); }
template <typename T>
__device__ __forceinline__ T psi_sub(T F, T a, T cc) { return rfma(-a, cc, F); }

__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// CPML slab membership of a column, fixed along the k march
template <typename T>
struct ColPml {
    int fx, sxl, fy, syl;
    T bx, cx, by, cy;
};

// E side: x slabs cover i in [1, np] and [nx-np, nx-1] (CPML.cpp:534-556)
template <typename T>
__device__ __forceinline__ ColPml<T> col_pml_e(const PmlView<T> &p, const Dims &d, int i, int j, bool act)
{
    ColPml<T> c{-1, 0, -1, 0, T(0), T(0), T(0), T(0)};
    if (act && i <= p.np[kFX1]) { c.fx = kFX1; c.sxl = i; }
    else if (act && i >= d.nx - p.np[kFX2]) { c.fx = kFX2; c.sxl = i - (d.nx - p.np[kFX2]); }
    if (j <= p.np[kFY1]) { c.fy = kFY1; c.syl = j; }
    else if (j >= d.ny - p.np[kFY2]) { c.fy = kFY2; c.syl = j - (d.ny - p.np[kFY2]); }
    if (c.fx >= 0) { c.bx = p.bE[c.fx][c.sxl]; c.cx = p.cE[c.fx][c.sxl]; }
    if (c.fy >= 0) { c.by = p.bE[c.fy][c.syl]; c.cy = p.cE[c.fy][c.syl]; }
    return c;
}

// H side: x slabs cover i in [0, np-1] and [nx-np, nx-1] (CPML.cpp:614-636)
template <typename T>
__device__ __forceinline__ ColPml<T> col_pml_h(const PmlView<T> &p, const Dims &d, int i, int j, bool act)
{
    ColPml<T> c{-1, 0, -1, 0, T(0), T(0), T(0), T(0)};
    if (act && i < p.np[kFX1]) { c.fx = kFX1; c.sxl = i; }
    else if (act && i >= d.nx - p.np[kFX2]) { c.fx = kFX2; c.sxl = i - (d.nx - p.np[kFX2]); }
    if (j < p.np[kFY1]) { c.fy = kFY1; c.syl = j; }
    else if (j >= d.ny - p.np[kFY2]) { c.fy = kFY2; c.syl = j - (d.ny - p.np[kFY2]); }
    if (c.fx >= 0) { c.bx = p.bH[c.fx][c.sxl]; c.cx = p.cH[c.fx][c.sxl]; }
    if (c.fy >= 0) { c.by = p.bH[c.fy][c.syl]; c.cy = p.cH[c.fy][c.syl]; }
    return c;
}

// CPML E corrections at one cell (CPML.cpp:537-602), x then y then z slabs
template <typename T>
__device__ __forceinline__ void pml_e_cell(const PmlView<T> &p, const Dims &d, const ColPml<T> &c, T ce, int i,
                                           int j, int k, T dHz_i, T dHy_i, T dHx_j, T dHz_j, T dHy_k, T dHx_k, T &ex,
                                           T &ey, T &ez)
{
    if (c.fx >= 0) {
        const int np = p.np[c.fx];
        const int64_t q = ((int64_t)k * (d.ny + 1) + j) * psi_xw(np) + c.sxl;
        T *q0 = p.qe[c.fx][0], *q1 = p.qe[c.fx][1];
        const T a0 = psi_new(c.bx, q0[q], c.cx, dHz_i), a1 = psi_new(c.bx, q1[q], c.cx, dHy_i);
        q0[q] = a0; q1[q] = a1;
        ey = psi_sub(ey, a0, ce);
        ez = psi_add(ez, a1, ce);
    }
    if (c.fy >= 0) {
        const int np = p.np[c.fy];
        const int64_t q = ((int64_t)k * (np + 1) + c.syl) * d.px + i;
        T *q0 = p.qe[c.fy][0], *q1 = p.qe[c.fy][1];
        const T a0 = psi_new(c.by, q0[q], c.cy, dHx_j), a1 = psi_new(c.by, q1[q], c.cy, dHz_j);
        q0[q] = a0; q1[q] = a1;
        ez = psi_sub(ez, a0, ce);
        ex = psi_add(ex, a1, ce);
    }
    int fz = -1, szl = 0;
    if (k <= p.np[kFZ1]) { fz = kFZ1; szl = k; }
    else if (k >= d.nz - p.np[kFZ2]) { fz = kFZ2; szl = k - (d.nz - p.np[kFZ2]); }
    if (fz >= 0) {
        const int64_t q = ((int64_t)szl * (d.ny + 1) + j) * d.px + i;
        T *q0 = p.qe[fz][0], *q1 = p.qe[fz][1];
        const T b = p.bE[fz][szl], cc = p.cE[fz][szl];
        const T a0 = psi_new(b, q0[q], cc, dHy_k), a1 = psi_new(b, q1[q], cc, dHx_k);
        q0[q] = a0; q1[q] = a1;
        ex = psi_sub(ex, a0, ce);
        ey = psi_add(ey, a1, ce);
    }
}

// psi words of one cell, loaded a plane ahead of their use
template <typename T>
struct PsiRegs {
    T x0, x1, y0, y1, z0, z1;
};

// E-side psi of plane k for a column (slab membership as in pml_e_cell).  Plain
// loads here and in psi_load_h: a sweep is launched while its predecessor still
// writes these words, and only plain loads stay behind its wait (pdl.cuh).
template <typename T>
__device__ __forceinline__ void psi_load_e(const PmlView<T> &p, const Dims &d, const ColPml<T> &c, int i, int j, int k,
                                           PsiRegs<T> &r)
{
    if (c.fx >= 0) {
        const int64_t q = ((int64_t)k * (d.ny + 1) + j) * psi_xw(p.np[c.fx]) + c.sxl;
        r.x0 = p.qe[c.fx][0][q]; r.x1 = p.qe[c.fx][1][q];
    }
    if (c.fy >= 0) {
        const int64_t q = ((int64_t)k * (p.np[c.fy] + 1) + c.syl) * d.px + i;
        r.y0 = p.qe[c.fy][0][q]; r.y1 = p.qe[c.fy][1][q];
    }
    int fz = -1, szl = 0;
    if (k <= p.np[kFZ1]) { fz = kFZ1; szl = k; }
    else if (k >= d.nz - p.np[kFZ2]) { fz = kFZ2; szl = k - (d.nz - p.np[kFZ2]); }
    if (fz >= 0) {
        const int64_t q = ((int64_t)szl * (d.ny + 1) + j) * d.px + i;
        r.z0 = p.qe[fz][0][q]; r.z1 = p.qe[fz][1][q];
    }
}

// H-side psi of plane k for a column (slabs [0, np-1] and [n-np, n-1])
template <typename T>
__device__ __forceinline__ void psi_load_h(const PmlView<T> &p, const Dims &d, const ColPml<T> &c, int i, int j, int k,
                                           PsiRegs<T> &r)
{
    if (c.fx >= 0) {
        const int64_t q = ((int64_t)k * (d.ny + 1) + j) * psi_xw(p.np[c.fx]) + c.sxl;
        r.x0 = p.qh[c.fx][0][q]; r.x1 = p.qh[c.fx][1][q];
    }
    if (c.fy >= 0) {
        const int64_t q = ((int64_t)k * (p.np[c.fy] + 1) + c.syl) * d.px + i;
        r.y0 = p.qh[c.fy][0][q]; r.y1 = p.qh[c.fy][1][q];
    }
    int fz = -1, szl = 0;
    if (k < p.np[kFZ1]) { fz = kFZ1; szl = k; }
    else if (k >= d.nz - p.np[kFZ2]) { fz = kFZ2; szl = k - (d.nz - p.np[kFZ2]); }
    if (fz >= 0) {
        const int64_t q = ((int64_t)szl * (d.ny + 1) + j) * d.px + i;
        r.z0 = p.qh[fz][0][q]; r.z1 = p.qh[fz][1][q];
    }
}

// CPML E corrections with psi already in registers (same arithmetic as pml_e_cell)
template <typename T>
__device__ __forceinline__ void pml_e_cell_pre(const PmlView<T> &p, const Dims &d, const ColPml<T> &c, T ce, int i,
                                               int j, int k, const PsiRegs<T> &r, T dHz_i, T dHy_i, T dHx_j, T dHz_j,
                                               T dHy_k, T dHx_k, T &ex, T &ey, T &ez)
{
    if (c.fx >= 0) {
        const int64_t q = ((int64_t)k * (d.ny + 1) + j) * psi_xw(p.np[c.fx]) + c.sxl;
        const T a0 = psi_new(c.bx, r.x0, c.cx, dHz_i), a1 = psi_new(c.bx, r.x1, c.cx, dHy_i);
        p.qe[c.fx][0][q] = a0; p.qe[c.fx][1][q] = a1;
        ey = psi_sub(ey, a0, ce);
        ez = psi_add(ez, a1, ce);
    }
    if (c.fy >= 0) {
        const int64_t q = ((int64_t)k * (p.np[c.fy] + 1) + c.syl) * d.px + i;
        const T a0 = psi_new(c.by, r.y0, c.cy, dHx_j), a1 = psi_new(c.by, r.y1, c.cy, dHz_j);
        p.qe[c.fy][0][q] = a0; p.qe[c.fy][1][q] = a1;
        ez = psi_sub(ez, a0, ce);
        ex = psi_add(ex, a1, ce);
    }
    int fz = -1, szl = 0;
    if (k <= p.np[kFZ1]) { fz = kFZ1; szl = k; }
    else if (k >= d.nz - p.np[kFZ2]) { fz = kFZ2; szl = k - (d.nz - p.np[kFZ2]); }
    if (fz >= 0) {
        const int64_t q = ((int64_t)szl * (d.ny + 1) + j) * d.px + i;
        const T b = p.bE[fz][szl], cc = p.cE[fz][szl];
        const T a0 = psi_new(b, r.z0, cc, dHy_k), a1 = psi_new(b, r.z1, cc, dHx_k);
        p.qe[fz][0][q] = a0; p.qe[fz][1][q] = a1;
        ex = psi_sub(ex, a0, ce);
        ey = psi_add(ey, a1, ce);
    }
}

// CPML H corrections (CPML.cpp:617-682), x then y then z slabs, with psi already
// in registers; STORE = false computes the corrected H without writing psi
template <typename T, bool STORE = true>
__device__ __forceinline__ void pml_h_cell_pre(const PmlView<T> &p, const Dims &d, const ColPml<T> &c, T ch, int i,
                                               int j, int k, const PsiRegs<T> &r, T dEz_i, T dEy_i, T dEx_j, T dEz_j,
                                               T dEy_k, T dEx_k, T &hx, T &hy, T &hz, bool store = true)
{
    if (c.fx >= 0) {
        const int64_t q = ((int64_t)k * (d.ny + 1) + j) * psi_xw(p.np[c.fx]) + c.sxl;
        const T a0 = psi_new(c.bx, r.x0, c.cx, dEz_i), a1 = psi_new(c.bx, r.x1, c.cx, dEy_i);
        if (STORE && store) { p.qh[c.fx][0][q] = a0; p.qh[c.fx][1][q] = a1; }
        hy = psi_add(hy, a0, ch);
        hz = psi_sub(hz, a1, ch);
    }
    if (c.fy >= 0) {
        const int64_t q = ((int64_t)k * (p.np[c.fy] + 1) + c.syl) * d.px + i;
        const T a0 = psi_new(c.by, r.y0, c.cy, dEx_j), a1 = psi_new(c.by, r.y1, c.cy, dEz_j);
        if (STORE && store) { p.qh[c.fy][0][q] = a0; p.qh[c.fy][1][q] = a1; }
        hz = psi_sub(hz, a0, ch);
        hx = psi_add(hx, a1, ch);
    }
    int fz = -1, szl = 0;
    if (k < p.np[kFZ1]) { fz = kFZ1; szl = k; }
    else if (k >= d.nz - p.np[kFZ2]) { fz = kFZ2; szl = k - (d.nz - p.np[kFZ2]); }
    if (fz >= 0) {
        const int64_t q = ((int64_t)szl * (d.ny + 1) + j) * d.px + i;
        const T b = p.bH[fz][szl], cc = p.cH[fz][szl];
        const T a0 = psi_new(b, r.z0, cc, dEy_k), a1 = psi_new(b, r.z1, cc, dEx_k);
        if (STORE && store) { p.qh[fz][0][q] = a0; p.qh[fz][1][q] = a1; }
        hx = psi_sub(hx, a0, ch);
        hy = psi_add(hy, a1, ch);
    }
}

// dl_component for compile-time pole counts, from state words already in
// registers (w[0 .. ND+2NL], the component's words in order)
template <typename T, int ND, int NL>
__device__ __forceinline__ T dl_component_regs(const DlCoef<T> &D, T E, T curl, const T *w, T *st, int64_t sc)
{
    const T temp = E;
    T t1 = T(0), t2 = T(0);
#pragma unroll
    for (int p = 0; p < ND; ++p) t1 = rfma(D.C4[p], w[p], t1);
#pragma unroll
    for (int p = 0; p < NL; ++p) t2 = rfma(D.C6[p], w[ND + NL + p], rfma(D.C5[p], w[ND + p], t2));
    const T e1 = w[ND + 2 * NL];
    E = radd(radd(radd(rfma(D.C1, E, rmul(D.C2, e1)), curl), -t1), -t2);
#pragma unroll
    for (int p = 0; p < ND; ++p) st[p * sc] = rfma(D.kappa[p], w[p], rmul(D.beta[p], E + temp));
#pragma unroll
    for (int p = 0; p < NL; ++p) {
        const T t0 = w[ND + p];
        st[(ND + p) * sc] =
            radd(rfma(D.alpha[p], t0, rmul(D.xi[p], w[ND + NL + p])), rmul(D.gammaL[p], E - e1) / T(2.0) / D.dt);
        st[(ND + NL + p) * sc] = t0;
    }
    st[(ND + 2 * NL) * sc] = temp;
    return E;
}

// four-level gain P -> E -> N at the gain cells of a warp row; the whole warp
// must call it
template <typename T>
__device__ __forceinline__ void gain_warp(const GainView<T> &G, const Dims &d, int j, int k, int seg, bool act,
                                          int id, T &ex, T &ey, T &ez)
{
    const bool mine = act && id == G.gain_id;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (!m) return;
    const int nseg = d.px >> 5;
    const int64_t base = G.seg[((int64_t)k * (d.ny + 1) + j) * nseg + seg];
    if (!mine) return;
    const int64_t c = base + __popc(m & lanemask_lt()), sc = kGainGroup;
    T *st = G.state + (sizeof(T) == 4 ? gain_dense_index(d.idx(seg * 32 + (int)(threadIdx.x & 31u), j, k))
                                      : gain_base_index(c, kG64Words));
    T E[3] = {ex, ey, ez}, E1[3] = {ex, ey, ez};
    T Pa[3], Pa1[3], Pa2[3], Pb[3], Pb1[3], Pb2[3];
    Pops<T> N;
    if (sizeof(T) == 8) {
        using L = GainSite64;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            Pa[q] = st[(L::PA + q) * sc]; Pa1[q] = st[(L::PA1 + q) * sc];
            Pb[q] = st[(L::PB + q) * sc]; Pb1[q] = st[(L::PB1 + q) * sc];
        }
    } else {
        using L = GainSite32;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            Pa[q] = st[(L::PA + q) * sc]; Pa1[q] = st[(L::PA1 + q) * sc];
            Pb[q] = st[(L::PB + q) * sc]; Pb1[q] = st[(L::PB1 + q) * sc];
        }
    }
    gain_load_n<T>(st, sc, N);
    gain_p_update<T>(G.c, N, E, Pa, Pa1, Pa2, Pb, Pb1, Pb2);
#pragma unroll
    for (int q = 0; q < 3; ++q) E[q] = gain_e_corr<T>(G.c, E[q], Pa[q], Pa1[q], Pb[q], Pb1[q]);
    gain_n_update<T>(G.c, N, E, E1, Pa, Pa1, Pa2, Pb, Pb2);
    // the transient words (Pa2 Pb2 E1) are not stored: only the plain path's
    // separate routines read them, after its own polarisation routine wrote them
    if (sizeof(T) == 8) {
        using L = GainSite64;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            st[(L::PA + q) * sc] = Pa[q]; st[(L::PA1 + q) * sc] = Pa1[q];
            st[(L::PB + q) * sc] = Pb[q]; st[(L::PB1 + q) * sc] = Pb1[q];
        }
    } else {
        using L = GainSite32;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            st[(L::PA + q) * sc] = Pa[q]; st[(L::PA1 + q) * sc] = Pa1[q];
            st[(L::PB + q) * sc] = Pb[q]; st[(L::PB1 + q) * sc] = Pb1[q];
        }
    }
    gain_store_n<T>(st, sc, N);
    ex = E[0]; ey = E[1]; ez = E[2];
}

// ---- FP64 gain in the block-tile E sweep.  What bounded it was latency at 16
// warps per SM: the 16 words of a cell (Pa Pa1 Pb Pb1 x3, N0..N3) were asked
// for after the list look-up and right before their use, the CPML body spilled
// to a memory that L1, what the stages leave of it, does not hold, and fourteen
// divisions a cell ran one after the other.  Now a row segment's list offset
// and gain mask come a plane ahead, the words are asked for at the top of the
// plane and used at its end, the psi words of the next plane go to shared slots
// of their own lane (8-byte asynchronous copies: no registers, no barrier) and
// the eleven divisions by constants are three operations each.  176^3 laser:
// CPML tiles 309 -> 222 us, interior 236 -> 187 us, 76 % of the copy bandwidth.
// (The gain words through shared slots too: 249 and 215 us, the 8-byte copies
// then fill the load-store queue.)
constexpr int kFetchSlots = 6;  // psi words per lane

__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// psi_load_e into slots
__device__ __forceinline__ void psi_fetch_e(const PmlView<double> &p, const Dims &d, const ColPml<double> &c, int i,
                                            int j, int k, double *slot)
{
    if (c.fx >= 0) {
        const int64_t q = ((int64_t)k * (d.ny + 1) + j) * psi_xw(p.np[c.fx]) + c.sxl;
        cp_async8(slot, p.qe[c.fx][0] + q); cp_async8(slot + 32, p.qe[c.fx][1] + q);
    }
    if (c.fy >= 0) {
        const int64_t q = ((int64_t)k * (p.np[c.fy] + 1) + c.syl) * d.px + i;
        cp_async8(slot + 64, p.qe[c.fy][0] + q); cp_async8(slot + 96, p.qe[c.fy][1] + q);
    }
    int fz = -1, szl = 0;
    if (k <= p.np[kFZ1]) { fz = kFZ1; szl = k; }
    else if (k >= d.nz - p.np[kFZ2]) { fz = kFZ2; szl = k - (d.nz - p.np[kFZ2]); }
    if (fz >= 0) {
        const int64_t q = ((int64_t)szl * (d.ny + 1) + j) * d.px + i;
        cp_async8(slot + 128, p.qe[fz][0] + q); cp_async8(slot + 160, p.qe[fz][1] + q);
    }
}


struct GainRegs64 {
    double a[6], b[6];  // Pa Pa1, Pb Pb1
    Pops<double> N;
};
// m: list offset and gain mask of the lane's row segment; the returned state
// pointer is null on a lane without a gain cell
__device__ __forceinline__ double *gain_fetch64(const GainView<double> &G, uint2 m, GainRegs64 &r)
{
    if (!((m.y >> (threadIdx.x & 31u)) & 1u)) return nullptr;
    using L = GainSite64;
    double *st = G.state + gain_base_index((int64_t)m.x + __popc(m.y & lanemask_lt()), kG64Words);
#pragma unroll
    for (int w = 0; w < 6; ++w) { r.a[w] = st[(L::PA + w) * kGainGroup]; r.b[w] = st[(L::PB + w) * kGainGroup]; }
    gain_load_n<double>(st, kGainGroup, r.N);
    return st;
}

// a / b by b's reciprocal r = 1 / b (rounded): a quotient to an ulp or two and
// one Newton correction with its exact remainder (Markstein, IBM J. Res. Dev.
// 34, 1990), three operations against the dozen and the branch of a division
__device__ __forceinline__ double div_by(double a, double b, double r)
{
    const double q = a * r;
    return __fma_rn(__fma_rn(-q, b, a), r, q);
}

// gain_n_update<double> with the constant divisors' reciprocals from the host
__device__ __forceinline__ void gain_n64(const GainCoef &G, Pops<double> &P, const double E[3], const double E1[3],
                                         const double Pa[3], const double Pa1[3], const double Pa2[3],
                                         const double Pb[3], const double Pb2[3])
{
    double *N = P.N;
    const double sb = E1[0] * (Pb[0] - Pb2[0]) + E1[1] * (Pb[1] - Pb2[1]) + E1[2] * (Pb[2] - Pb2[2]);
    const double sa = E1[0] * (Pa[0] - Pa2[0]) + E1[1] * (Pa[1] - Pa2[1]) + E1[2] * (Pa[2] - Pa2[2]);
    const double s2 = (E[0] + E1[0]) * (Pa[0] - Pa2[0]) + (E[1] + E1[1]) * (Pa[1] - Pa1[1]) +
                      (E[2] + E1[2]) * (Pa[2] - Pa2[2]);
    const double N0old = N[0];
    N[3] = G.t30t32dt / (G.t30t32_2 + G.t30dt * (1 - N[2]) + G.t32dt * (1 - N[0])) *
           (N[3] * (div_by(N[0] - 1, G.t30, G.r_t30) + div_by(N[2] - 1, G.t32, G.r_t32) + G.dt_2) +
            div_by(sb, G.homega_bdt, G.r_hwb));
    N[3] = N[3] + G.pump_dt * N0old;
    N[1] = G.t10t21dt / (G.t10t21_2 + G.t10dt * N[2] + G.t21dt * (1 - N[0])) *
           (N[1] * (div_by(N[0] - 1, G.t10, G.r_t10) - div_by(N[2], G.t21, G.r_t21) + G.dt_2) +
            div_by(N[2], G.t21_2, G.r_t21_2) - div_by(sa, G.homega_adt, G.r_hwa));
    N[2] = G.t32t21dt / (G.t32t21_2 + G.t21dt * N[3] + G.t32dt * (1 - N[1])) *
           (N[2] * (div_by(N[1] - 1, G.t21, G.r_t21) - div_by(N[3], G.t32, G.r_t32) + G.dt_2) +
            div_by(N[3], G.t32_2, G.r_t32_2) + div_by(s2, G.homega_adt, G.r_hwa));
    N[0] = 2.0 - N[1] - N[2] - N[3];
}

// P -> E -> N at a gain cell from its words (gain_warp's arithmetic)
__device__ __forceinline__ void gain_apply64(const GainView<double> &G, double *st, GainRegs64 &r, double &ex,
                                             double &ey, double &ez)
{
    using L = GainSite64;
    constexpr int64_t sc = kGainGroup;
    double E[3] = {ex, ey, ez};
    const double E1[3] = {ex, ey, ez};
    double Pa2[3], Pb2[3];
    gain_p_update<double>(G.c, r.N, E, r.a, r.a + 3, Pa2, r.b, r.b + 3, Pb2);
#pragma unroll
    for (int q = 0; q < 3; ++q) E[q] = gain_e_corr<double>(G.c, E[q], r.a[q], r.a[3 + q], r.b[q], r.b[3 + q]);
    gain_n64(G.c, r.N, E, E1, r.a, r.a + 3, Pa2, r.b, Pb2);
#pragma unroll
    for (int q = 0; q < 6; ++q) { st[(L::PA + q) * sc] = r.a[q]; st[(L::PB + q) * sc] = r.b[q]; }
    gain_store_n<double>(st, sc, r.N);
    ex = E[0]; ey = E[1]; ez = E[2];
}

// ---- FP32 gain on the segment-dense layout: the 15 persistent words of the
// cell at device index g are at gain_dense_index(g) + 32 w, for every cell of
// the grid, so a plane's words can be requested (or staged by TMA) before its
// fields and IDs arrive.  The arithmetic is gain_warp's.
struct GainRegs32 {
    float pa[3], pa1[3], pb[3], pb1[3];
    float n[3];  // the population offsets N1 - 1, N2, N3
};

// the words of the cell at device index g from global memory
__device__ __forceinline__ void gain_fetch32(const GainView<float> &G, int64_t g, GainRegs32 &r)
{
    using L = GainSite32;
    const float *st = G.state + gain_dense_index(g);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        r.pa[q] = __ldg(st + (L::PA + q) * kGainGroup);
        r.pa1[q] = __ldg(st + (L::PA1 + q) * kGainGroup);
        r.pb[q] = __ldg(st + (L::PB + q) * kGainGroup);
        r.pb1[q] = __ldg(st + (L::PB1 + q) * kGainGroup);
    }
    r.n[0] = __ldg(st + L::DN1 * kGainGroup);
    r.n[1] = __ldg(st + L::N2 * kGainGroup);
    r.n[2] = __ldg(st + L::N3 * kGainGroup);
}

// the words of a cell from a staged tile: word w at ws[32 w]
__device__ __forceinline__ void gain_staged32(const float *ws, GainRegs32 &r)
{
    using L = GainSite32;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        r.pa[q] = ws[(L::PA + q) * 32];
        r.pa1[q] = ws[(L::PA1 + q) * 32];
        r.pb[q] = ws[(L::PB + q) * 32];
        r.pb1[q] = ws[(L::PB1 + q) * 32];
    }
    r.n[0] = ws[L::DN1 * 32];
    r.n[1] = ws[L::N2 * 32];
    r.n[2] = ws[L::N3 * 32];
}

// one component of the gain update at a cell: P (FourLevelLaser.cpp:274-295,
// words scaled by CEP), E -= dP (:302-305); E1 is the field before
__device__ __forceinline__ void gain_comp32(const GainCoef &G, float E1, float dNa, float dNb, float pa, float pa1,
                                            float pb, float pb1, float &a, float &b, float &E)
{
    a = rfma(rmul(E1, G.fa3), dNa, rfma(G.fa1, pa, rmul(G.fa2, pa1)));
    b = rfma(rmul(E1, G.fb3), dNb, rfma(G.fb1, pb, rmul(G.fb2, pb1)));
    E = E1 - radd(radd(radd(a, -pa), b), -pb);
}

// population offsets from the energy-exchange sums (gain_n_update<float>)
__device__ __forceinline__ void gain_pops32(const GainCoef &G, float sa, float sb, float s2, float m0, float &n1,
                                            float &n2, float &n3)
{
    const float q3 = rfma(G.k3a, 1.0f - n2, -rmul(G.k3b, m0));
    const float n3n = rfma(G.fpump, 1.0f + m0, __fdividef(rfma(n3, 1.0f - q3, rmul(G.hb, sb)), 1.0f + q3));
    const float q1 = rfma(G.k1a, n2, -rmul(G.k1b, m0));
    const float n1n = __fdividef(rfma(-G.ha, sa, rfma(n1, 1.0f - q1, rmul(2.0f * G.k1b, m0))), 1.0f + q1);
    const float q2 = rfma(G.k3a, n3n, -rmul(G.k1a, n1n));
    const float n2n = __fdividef(rfma(G.ha, s2, rfma(n2, 1.0f - q2, rmul(2.0f * G.k3a, n3n))), 1.0f + q2);
    n1 = n1n;
    n2 = n2n;
    n3 = n3n;
}

// P -> E -> N at a gain cell (device index g) from its words r; the new words
// go to the dense state.  The Ey term of the N2 sum uses P - P' as the
// reference does (FourLevelLaser.cpp:316).
__device__ __forceinline__ void gain_apply32(const GainView<float> &G, int64_t g, const GainRegs32 &r, float &ex,
                                             float &ey, float &ez)
{
    using L = GainSite32;
    float *st = G.state + gain_dense_index(g);
    const int64_t sc = kGainGroup;
    float n1 = r.n[0], n2 = r.n[1], n3 = r.n[2];
    const float m0 = conserve_m0(n1, n2, n3);  // FP64 conservation, FourLevelLaser.cpp:324
    const float dNa = (n2 - n1) - 1.0f, dNb = (n3 - m0) - 1.0f;
    float sa = 0.0f, sb = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
        const int q = o == 0 ? 1 : o == 1 ? 0 : 2;
        float &F = q == 0 ? ex : q == 1 ? ey : ez;
        const float E1 = F;
        float a, b, E;
        gain_comp32(G.c, E1, dNa, dNb, r.pa[q], r.pa1[q], r.pb[q], r.pb1[q], a, b, E);
        const float da = a - r.pa1[q], db = b - r.pb1[q], d2 = q == 1 ? a - r.pa[q] : da;
        sa = o == 0 ? rmul(E1, da) : rfma(E1, da, sa);
        sb = o == 0 ? rmul(E1, db) : rfma(E1, db, sb);
        s2 = o == 0 ? rmul(E + E1, d2) : rfma(E + E1, d2, s2);
        st[(L::PA + q) * sc] = a; st[(L::PA1 + q) * sc] = r.pa[q];
        st[(L::PB + q) * sc] = b; st[(L::PB1 + q) * sc] = r.pb[q];
        F = E;
    }
    gain_pops32(G.c, sa, sb, s2, m0, n1, n2, n3);
    st[L::DN1 * sc] = n1;
    st[L::N2 * sc] = n2;
    st[L::N3 * sc] = n3;
}

}  // namespace cps
