// kernels_plain.cu -- one kernel per reference routine ("plain" path).
//
// Compiled with --fmad=false: every multiply and add rounds on its own, in
// the reference's order, so the FP64 instantiation reproduces the reference
// arithmetic of BasicFDTD.cpp, CPML.cpp, TF_SF.cpp and the oracle's
// Drude-Lorentz/gain recursions operation by operation.
#include <string.h>

#include "batch.h"
#include "cells.cuh"
#include "pdl.cuh"

namespace cps {

namespace {

// rows of a block of the bulk and CPML kernels.  A block with slab cells takes
// several times as long as one without, so small blocks fill the SMs better:
// 96^3 FP64 43.1, 41.0 and 45.4 us a step with 8, 4 and 2 rows.  (Requesting a
// cell's psi words before its field words costs the registers of a third of the
// warps: 52 us.)
constexpr int kBY = 4;

// psi index of slab-local s at (i,j,k) for axis a (x: [k][j][s], y: [k][s][i], z: [s][j][i])
__device__ __forceinline__ int64_t psi_index(const Dims &d, int axis, int np, int s, int i, int j, int k)
{
    if (axis == 0) return ((int64_t)k * (d.ny + 1) + j) * psi_xw(np) + s;
    if (axis == 1) return ((int64_t)k * (np + 1) + s) * d.px + i;
    return ((int64_t)s * (d.ny + 1) + j) * d.px + i;
}

// slab of index `at` on an axis of n cells (f1 its first face): E slabs are
// [1, np] and [n-np, n-1] (CPML.cpp:534, 546), H slabs [0, np-1] and [n-np, n-1]
// (CPML.cpp:614, 626); -1 outside
__device__ __forceinline__ int slab_of(const int np[6], int f1, int n, int at, bool eside, int &s)
{
    s = at;
    if (at < np[f1] + (eside ? 1 : 0)) return f1;
    s = at - (n - np[f1 + 1]);
    return s >= 0 ? f1 + 1 : -1;
}

// one face's psi pair: q <- b q + c d
template <typename T>
__device__ __forceinline__ void psi_pair(T *const q[2], int64_t o, T b, T c, T d0, T d1, T &a0, T &a1)
{
    a0 = b * q[0][o] + c * d0;
    a1 = b * q[1][o] + c * d1;
    q[0][o] = a0;
    q[1][o] = a1;
}

// CPML::UpdateCPMLHFields at one cell (CPML.cpp:609-689): the faces in the
// reference's order x1 x2 y1 y2 z1 z2.  A cell lies in one end of an axis at
// most, so its corrections are those of the per-face loops in their order.
template <typename T>
__device__ __forceinline__ void h_pml_at(const FieldView<T> &f, const PmlView<T> &p, int i, int j, int k, int64_t g,
                                         int id, T &hx, T &hy, T &hz)
{
    const Dims &d = f.d;
    int sx, sy, sz;
    const int fx = slab_of(p.np, kFX1, d.nx, i, false, sx), fy = slab_of(p.np, kFY1, d.ny, j, false, sy);
    const int fz = slab_of(p.np, kFZ1, d.nz, k, false, sz);
    if (fx < 0 && fy < 0 && fz < 0) return;
    const T ch = pml_ch_cell(p, f.bH, id);
    T a0, a1;
    if (fx >= 0) {
        psi_pair(p.qh[fx], psi_index(d, 0, p.np[fx], sx, i, j, k), p.bH[fx][sx], p.cH[fx][sx], f.Ez[g + 1] - f.Ez[g],
                 f.Ey[g + 1] - f.Ey[g], a0, a1);
        hy = hy + a0 * ch;
        hz = hz - a1 * ch;
    }
    if (fy >= 0) {
        psi_pair(p.qh[fy], psi_index(d, 1, p.np[fy], sy, i, j, k), p.bH[fy][sy], p.cH[fy][sy],
                 f.Ex[g + d.px] - f.Ex[g], f.Ez[g + d.px] - f.Ez[g], a0, a1);
        hz = hz - a0 * ch;
        hx = hx + a1 * ch;
    }
    if (fz >= 0) {
        psi_pair(p.qh[fz], psi_index(d, 2, p.np[fz], sz, i, j, k), p.bH[fz][sz], p.cH[fz][sz],
                 f.Ey[g + d.pxy] - f.Ey[g], f.Ex[g + d.pxy] - f.Ex[g], a0, a1);
        hx = hx - a0 * ch;
        hy = hy + a1 * ch;
    }
}

// CPML::UpdateCPMLEFields at one cell (CPML.cpp:529-607), likewise
template <typename T>
__device__ __forceinline__ void e_pml_at(const FieldView<T> &f, const PmlView<T> &p, int i, int j, int k, int64_t g,
                                         int id, T &ex, T &ey, T &ez)
{
    const Dims &d = f.d;
    int sx, sy, sz;
    const int fx = slab_of(p.np, kFX1, d.nx, i, true, sx), fy = slab_of(p.np, kFY1, d.ny, j, true, sy);
    const int fz = slab_of(p.np, kFZ1, d.nz, k, true, sz);
    if (fx < 0 && fy < 0 && fz < 0) return;
    const T ce = pml_ce_cell(p, f.bE, id);
    T a0, a1;
    if (fx >= 0) {
        psi_pair(p.qe[fx], psi_index(d, 0, p.np[fx], sx, i, j, k), p.bE[fx][sx], p.cE[fx][sx], f.Hz[g] - f.Hz[g - 1],
                 f.Hy[g] - f.Hy[g - 1], a0, a1);
        ey = ey - a0 * ce;
        ez = ez + a1 * ce;
    }
    if (fy >= 0) {
        psi_pair(p.qe[fy], psi_index(d, 1, p.np[fy], sy, i, j, k), p.bE[fy][sy], p.cE[fy][sy],
                 f.Hx[g] - f.Hx[g - d.px], f.Hz[g] - f.Hz[g - d.px], a0, a1);
        ez = ez - a0 * ce;
        ex = ex + a1 * ce;
    }
    if (fz >= 0) {
        psi_pair(p.qe[fz], psi_index(d, 2, p.np[fz], sz, i, j, k), p.bE[fz][sz], p.cE[fz][sz],
                 f.Hy[g] - f.Hy[g - d.pxy], f.Hx[g] - f.Hx[g - d.pxy], a0, a1);
        ex = ex - a0 * ce;
        ey = ey + a1 * ce;
    }
}

// BasicHFieldUpdate, BasicFDTD.cpp:67-84: i,j,k in [0, N-1]; PML: the cell's
// CPML corrections too (steps whose TF/SF-H targets lie outside the slabs, so
// that nothing comes between the two routines at any cell).  One launch in the
// place of seven: at 96^3 in FP64 the six face launches took 37 us beside 14 us
// of bulk update and, with their issue, most of a 114 us step.
template <typename T, bool PML>
__global__ void __launch_bounds__(32 * kBY) k_h_bulk(FieldView<T> f, PmlView<T> p)
{
    pdl_go();
    pdl_wait();
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y, k = blockIdx.z;
    if (i >= f.d.nx || j >= f.d.ny) return;
    const int64_t g = f.d.idx(i, j, k), sy = f.d.px, sz = f.d.pxy;
    const int id = f.id[g];
    const T aH = f.aH[id], bH = f.bH[id];
    const StretchView<T> &s = f.s;
    T hx = aH * f.Hx[g] - bH * (f.Ez[g + sy] - f.Ez[g]) * s.cHxz[j] + bH * (f.Ey[g + sz] - f.Ey[g]) * s.cHxy[k];
    T hy = aH * f.Hy[g] - bH * (f.Ex[g + sz] - f.Ex[g]) * s.cHyx[k] + bH * (f.Ez[g + 1] - f.Ez[g]) * s.cHyz[i];
    T hz = aH * f.Hz[g] + bH * (f.Ex[g + sy] - f.Ex[g]) * s.cHzx[j] - bH * (f.Ey[g + 1] - f.Ey[g]) * s.cHzy[i];
    if (PML) h_pml_at(f, p, i, j, k, g, id, hx, hy, hz);
    f.Hx[g] = hx;
    f.Hy[g] = hy;
    f.Hz[g] = hz;
}

// BasicEFieldUpdate, BasicFDTD.cpp:25-47: i,j,k in [1, N-1]; ID 4 zeroes E,
// ID 2 is left to the Drude-Lorentz routine.  PML: the cell's CPML corrections
// too (steps without dispersive or gain terms whose TF/SF-E targets and sources
// lie outside the slabs).
template <typename T, bool PML>
__global__ void __launch_bounds__(32 * kBY) k_e_bulk(FieldView<T> f, PmlView<T> p)
{
    pdl_go();
    pdl_wait();
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y, k = blockIdx.z + 1;
    if (i < 1 || i >= f.d.nx || j < 1 || j >= f.d.ny) return;
    const int64_t g = f.d.idx(i, j, k), sy = f.d.px, sz = f.d.pxy;
    const int id = f.id[g];
    T ex, ey, ez;
    if (id == CPS_ID_PEC) {
        ex = T(0); ey = T(0); ez = T(0);
    } else if (id != CPS_ID_DISPERSIVE) {
        const T aE = f.aE[id], bE = f.bE[id];
        const StretchView<T> &s = f.s;
        ex = aE * f.Ex[g] + bE * (f.Hz[g] - f.Hz[g - sy]) * s.cExz[j] - bE * (f.Hy[g] - f.Hy[g - sz]) * s.cExy[k];
        ey = aE * f.Ey[g] + bE * (f.Hx[g] - f.Hx[g - sz]) * s.cEyx[k] - bE * (f.Hz[g] - f.Hz[g - 1]) * s.cEyz[i];
        ez = aE * f.Ez[g] + bE * (f.Hy[g] - f.Hy[g - 1]) * s.cEzy[i] - bE * (f.Hx[g] - f.Hx[g - sy]) * s.cEzx[j];
    } else {
        if (!PML) return;
        ex = f.Ex[g]; ey = f.Ey[g]; ez = f.Ez[g];
    }
    if (PML) e_pml_at(f, p, i, j, k, g, id, ex, ey, ez);
    f.Ex[g] = ex;
    f.Ey[g] = ey;
    f.Ez[g] = ez;
}

// The CPML routine of one side alone, every slab in one launch: the cells of
// the z slabs, then of the y slabs between them, then of the x slabs between
// those, a block row of 32 x kBY threads at a time.
struct SlabBoxes {
    int n;
    int start[7];              // first block of each box
    int i0[6], j0[6], k0[6];   // first cell
    int ni[6], nj[6], nk[6];   // cells
};

template <typename T, bool ESIDE>
__global__ void __launch_bounds__(32 * kBY) k_pml(FieldView<T> f, PmlView<T> p, const __grid_constant__ SlabBoxes B)
{
    int b = 0;
    while (b + 1 < B.n && (int)blockIdx.x >= B.start[b + 1]) ++b;
    int r = (int)blockIdx.x - B.start[b];
    const int bx = (B.ni[b] + 31) / 32, by = (B.nj[b] + kBY - 1) / kBY;
    const int z = r / (bx * by);
    r -= z * bx * by;
    const int y = r / bx, u = (r - y * bx) * 32 + (int)threadIdx.x, v = y * kBY + (int)threadIdx.y;
    if (u >= B.ni[b] || v >= B.nj[b]) return;
    const int i = B.i0[b] + u, j = B.j0[b] + v, k = B.k0[b] + z;
    const int64_t g = f.d.idx(i, j, k);
    if (ESIDE) {
        T ex = f.Ex[g], ey = f.Ey[g], ez = f.Ez[g];
        e_pml_at(f, p, i, j, k, g, (int)f.id[g], ex, ey, ez);
        f.Ex[g] = ex; f.Ey[g] = ey; f.Ez[g] = ez;
    } else {
        T hx = f.Hx[g], hy = f.Hy[g], hz = f.Hz[g];
        h_pml_at(f, p, i, j, k, g, (int)f.id[g], hx, hy, hz);
        f.Hx[g] = hx; f.Hy[g] = hy; f.Hz[g] = hz;
    }
}

__device__ __forceinline__ void decode(const Dims &d, int64_t g, int &i, int &j, int &k)
{
    k = (int)(g / d.pxy);
    const int64_t r = g - (int64_t)k * d.pxy;
    j = (int)(r / d.px);
    i = (int)(r - (int64_t)j * d.px);
}

// 3-D Drude-Lorentz ADE on the ID==2 cell list (Drude_Lorentz.cpp:153-227
// with the curl terms of BasicFDTD.cpp:39-41 and bE replaced by C3)
template <typename T>
__global__ void k_dl(FieldView<T> f, DlView<T> D)
{
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= D.ncell) return;
    const int64_t g = D.cell[c];
    int i, j, k;
    decode(f.d, g, i, j, k);
    const int64_t sy = f.d.px, sz = f.d.pxy;
    const StretchView<T> &s = f.s;
    const T C3 = D.c.C3;
    const T cx = C3 * (f.Hz[g] - f.Hz[g - sy]) * s.cExz[j] - C3 * (f.Hy[g] - f.Hy[g - sz]) * s.cExy[k];
    const T cy = C3 * (f.Hx[g] - f.Hx[g - sz]) * s.cEyx[k] - C3 * (f.Hz[g] - f.Hz[g - 1]) * s.cEyz[i];
    const T cz = C3 * (f.Hy[g] - f.Hy[g - 1]) * s.cEzy[i] - C3 * (f.Hx[g] - f.Hx[g - sy]) * s.cEzx[j];
    const int64_t sc = D.ncell;
    T *st = D.state + c;
    f.Ex[g] = dl_component(D.c, f.Ex[g], cx, st, sc);
    f.Ey[g] = dl_component(D.c, f.Ey[g], cy, st + (int64_t)D.c.stride * sc, sc);
    f.Ez[g] = dl_component(D.c, f.Ez[g], cz, st + (int64_t)2 * D.c.stride * sc, sc);
}

// FourLevelLaser routines on the gain cell list: which 0 = polarization
// (:270-298), 1 = E correction (:300-308), 2 = populations (:310-325)
template <typename T, typename L>
__global__ void k_gain(FieldView<T> f, GainView<T> G, int which)
{
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= G.ncell) return;
    const int64_t g = G.cell[c], sc = kGainGroup;
    // persistent words (stride 32 in both layouts) and the transient words
    // Pa2 Pb2 E1 (FP32: their own list-layout array)
    T *st, *tr;
    if (sizeof(T) == 4) {
        st = G.state + gain_dense_index(g);
        tr = G.trans + gain_base_index(c, kGainTrans);
    } else {
        st = G.state + gain_base_index(c, kG64Words);
        tr = st;
    }
    auto tw = [&](int w) -> T & { return sizeof(T) == 4 ? tr[(w - kGainPersist) * sc] : st[w * sc]; };
    T *F[3] = {f.Ex, f.Ey, f.Ez};
    T E[3] = {F[0][g], F[1][g], F[2][g]};
    T Pa[3], Pa1[3], Pa2[3], Pb[3], Pb1[3], Pb2[3];
    for (int q = 0; q < 3; ++q) {
        Pa[q] = st[(L::PA + q) * sc]; Pa1[q] = st[(L::PA1 + q) * sc];
        Pb[q] = st[(L::PB + q) * sc]; Pb1[q] = st[(L::PB1 + q) * sc];
    }
    if (which == 0) {
        Pops<T> N;
        gain_load_n<T>(st, sc, N);
        gain_p_update<T>(G.c, N, E, Pa, Pa1, Pa2, Pb, Pb1, Pb2);
        for (int q = 0; q < 3; ++q) {
            st[(L::PA + q) * sc] = Pa[q]; st[(L::PA1 + q) * sc] = Pa1[q]; tw(L::PA2 + q) = Pa2[q];
            st[(L::PB + q) * sc] = Pb[q]; st[(L::PB1 + q) * sc] = Pb1[q]; tw(L::PB2 + q) = Pb2[q];
            tw(L::E1 + q) = E[q];
        }
    } else if (which == 1) {
        for (int q = 0; q < 3; ++q) F[q][g] = gain_e_corr<T>(G.c, E[q], Pa[q], Pa1[q], Pb[q], Pb1[q]);
    } else {
        Pops<T> N;
        T E1[3];
        gain_load_n<T>(st, sc, N);
        for (int q = 0; q < 3; ++q) {
            Pa2[q] = tw(L::PA2 + q); Pb2[q] = tw(L::PB2 + q); E1[q] = tw(L::E1 + q);
        }
        gain_n_update<T>(G.c, N, E, E1, Pa, Pa1, Pa2, Pb, Pb2);
        gain_store_n<T>(st, sc, N);
    }
}

// FP32 population offsets of each list cell for the host read-out
__global__ void k_gain_pops32(const float *state, const int64_t *cell, int64_t ncell, float *out)
{
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    const float *st = state + gain_dense_index(cell[c]);
    for (int q = 0; q < 3; ++q) out[c * 3 + q] = st[(GainSite32::DN1 + q) * kGainGroup];
}

// FP64 initial populations N0 = N1 = 1 (words 21, 22 of each cell)
__global__ void k_gain_init64(double *state, int64_t ncell)
{
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    double *st = state + gain_base_index(c, kG64Words);
    st[GainSite64::N * kGainGroup] = 1.0;
    st[(GainSite64::N + 1) * kGainGroup] = 1.0;
}

// TF/SF (and any other table-driven) injection in CSR form: each thread owns
// one (cell, component) target and adds its contributions in order,
// F += coef * inc(n - delay) * profile (TF_SF.cpp:992-1087, 1206-1299)
// one TF/SF target: its contributions in the reference's face order
template <typename T>
__device__ __forceinline__ T inject_add(T v, const InjContrib &a, const T *table, int Nt, double n)
{
    const T inc = (T)inc_lookup<T>(table, Nt, n - a.delay);
    return v + (T)a.coef * inc * (T)a.profile;
}

template <typename T>
__device__ __forceinline__ void inject_target(const FieldView<T> &f, const InjTarget &q, const InjContrib *ct,
                                              const T *table, int Nt, double n, uint32_t face_mask)
{
    T *F = field_comp(f, q.comp) + q.idx;
    T v = *F;
    for (int c = q.start; c < q.start + q.count; ++c) {
        const InjContrib a = ct[c];
        if (!(face_mask & (1u << a.face))) continue;
        v = inject_add(v, a, table, Nt, n);
    }
    *F = v;
}

template <typename T>
__global__ void k_inject(FieldView<T> f, const InjTarget *tg, int ntarget, const InjContrib *ct,
                         const T *table, int Nt, double n, uint32_t face_mask)
{
    pdl_go();
    pdl_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntarget) return;
    inject_target<T>(f, tg[t], ct, table, Nt, n, face_mask);
}

template <typename T>
__global__ void k_inject_pack(uint64_t *word, double *delay, Pair<T> *cp, const InjTarget *tg, int ntarget,
                              const InjContrib *ct)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntarget) return;
    const InjTarget q = tg[t];
    const InjContrib a = ct[q.start];  // every target has at least one contribution
    word[t] = (uint64_t)q.idx | (uint64_t)q.comp << 48 | (q.count > 1 ? 1ull << 51 : 0ull);
    delay[t] = a.delay;
    cp[t] = Pair<T>{(T)a.coef, (T)a.profile};
}

// Every face of one side.  A few megabytes move, so what bounds this is the
// chain of dependent loads; each thread takes two targets kInjThreads apart and
// asks for both at every link.  With the first contribution beside the target
// and the grid's pointers as kernel parameters the chain is record, then table
// and field: 256^3 (580 k targets a side), 16.3 -> 12.4 us; through the CSR
// lists and a descriptor it was block, grid, target, contribution, table.
// Each target's contributions are added in its own order, as in inject_target;
// the two targets are distinct (cell, component) pairs.
template <typename T>
__device__ __forceinline__ void inject_two(const FieldView<T> &f, const InjView<T> &V, int t0, int end, double n)
{
    if (t0 >= end) return;
    const int t1 = t0 + kInjThreads;
    const bool two = t1 < end;
    const int u1 = two ? t1 : t0;
    const uint64_t w0 = V.word[t0], w1 = V.word[u1];
    const double d0 = V.delay[t0], d1 = V.delay[u1];
    const Pair<T> c0 = V.cp[t0], c1 = V.cp[u1];
    const uint64_t mask = (1ull << 48) - 1;
    T *F0 = field_comp(f, (int)(w0 >> 48 & 7)) + (w0 & mask);
    T *F1 = field_comp(f, (int)(w1 >> 48 & 7)) + (w1 & mask);
    T v0 = *F0, v1 = *F1;
    v0 = v0 + c0.a * (T)inc_lookup<T>(V.table, V.Nt, n - d0) * c0.b;
    v1 = v1 + c1.a * (T)inc_lookup<T>(V.table, V.Nt, n - d1) * c1.b;
    auto rest = [&](int t, T v) {
        const InjTarget q = V.tg[t];
        for (int c = q.start + 1; c < q.start + q.count; ++c) v = inject_add(v, V.ct[c], V.table, V.Nt, n);
        return v;
    };
    if (w0 >> 51) v0 = rest(t0, v0);
    *F0 = v0;
    if (!two) return;
    if (w1 >> 51) v1 = rest(t1, v1);
    *F1 = v1;
}

template <typename T>
__global__ void __launch_bounds__(kInjThreads) k_inject_all(FieldView<T> f, InjView<T> V, const int64_t *n0, int64_t n)
{
    pdl_go();
    pdl_wait();
    inject_two<T>(f, V, blockIdx.x * kInjPerBlock + (int)threadIdx.x, min((int)(blockIdx.x + 1) * kInjPerBlock, V.n),
                  (double)((n0 ? *n0 : 0) + n));
}

// batched form: the step number is the grid's chunk start plus step_off; a
// block entry covers up to kInjPerBlock targets
template <typename T>
__global__ void __launch_bounds__(kInjThreads) k_inject_batch(const BatchGrid<T> *__restrict__ grids,
                                                              const int4 *__restrict__ blocks, int side,
                                                              int step_off)
{
    pdl_go();
    pdl_wait();
    const int4 e = blocks[blockIdx.x];
    const BatchGrid<T> &B = grids[e.x];
    inject_two<T>(B.f, B.inj[side], e.y + (int)threadIdx.x, e.z, (double)(B.n0 + step_off));
}

template <typename T>
__global__ void k_sources_batch(const BatchGrid<T> *__restrict__ grids, const int2 *__restrict__ ents, int n,
                                int step_off)
{
    pdl_go();
    pdl_wait();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int2 e = ents[q];
    const BatchGrid<T> &B = grids[e.x];
    const int s = e.y;
    const int64_t nn = B.n0 + step_off;
    if (nn < 0 || nn >= B.src_len[s]) return;
    const FieldView<T> &f = B.f;
    T *F[6] = {f.Ex, f.Ey, f.Ez, f.Hx, f.Hy, f.Hz};
    const int64_t g = B.src_idx[s];
    T *dst = F[B.src_comp[s]];
    dst[g] = dst[g] + (T)B.src_wave[B.src_off[s] + nn];
}

template <typename T>
__global__ void k_sources(FieldView<T> f, int nsrc, const int64_t *idx, const int32_t *comp,
                          const double *waves, const int32_t *off, const int32_t *len, int n)
{
    pdl_go();
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsrc || n < 0 || n >= len[s]) return;
    T *F[6] = {f.Ex, f.Ey, f.Ez, f.Hx, f.Hy, f.Hz};
    F[comp[s]][idx[s]] = F[comp[s]][idx[s]] + (T)waves[off[s] + n];
}

inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

}  // namespace

// the slab cells of a side as disjoint boxes
template <typename T>
static SlabBoxes slab_boxes(const PmlView<T> &p, const Dims &d, bool eside)
{
    SlabBoxes B;
    memset(&B, 0, sizeof(B));
    const int lo = eside ? 1 : 0;  // first updated index
    const int n[3] = {d.nx, d.ny, d.nz};
    int a[3], e[3];  // the interior between the slabs, shrunk axis by axis
    for (int q = 0; q < 3; ++q) { a[q] = lo; e[q] = n[q]; }
    for (int ax = 2; ax >= 0; --ax)
        for (int end = 0; end < 2; ++end) {
            const int np = p.np[2 * ax + end];
            int b0[3] = {a[0], a[1], a[2]}, b1[3] = {e[0], e[1], e[2]};
            if (end == 0) {
                b1[ax] = lo + np;
                a[ax] = lo + np;
            } else {
                b0[ax] = n[ax] - np;
                e[ax] = n[ax] - np;
            }
            if (np <= 0 || b1[0] <= b0[0] || b1[1] <= b0[1] || b1[2] <= b0[2]) continue;
            const int q = B.n++;
            B.i0[q] = b0[0]; B.j0[q] = b0[1]; B.k0[q] = b0[2];
            B.ni[q] = b1[0] - b0[0]; B.nj[q] = b1[1] - b0[1]; B.nk[q] = b1[2] - b0[2];
            B.start[q + 1] = B.start[q] + (int)(cdiv(B.ni[q], 32) * cdiv(B.nj[q], kBY)) * B.nk[q];
        }
    return B;
}

template <typename T>
void launch_h_bulk(const FieldView<T> &f, const PmlView<T> &p, bool with_pml, cudaStream_t s)
{
    dim3 grid(cdiv(f.d.nx, 32), cdiv(f.d.ny, kBY), f.d.nz);
    if (with_pml) launch_pdl(true, k_h_bulk<T, true>, grid, dim3(32, kBY), 0, s, f, p);
    else launch_pdl(true, k_h_bulk<T, false>, grid, dim3(32, kBY), 0, s, f, p);
}

template <typename T>
void launch_e_bulk(const FieldView<T> &f, const PmlView<T> &p, bool with_pml, cudaStream_t s)
{
    if (f.d.nz < 2) return;
    dim3 grid(cdiv(f.d.nx, 32), cdiv(f.d.ny, kBY), f.d.nz - 1);
    if (with_pml) launch_pdl(true, k_e_bulk<T, true>, grid, dim3(32, kBY), 0, s, f, p);
    else launch_pdl(true, k_e_bulk<T, false>, grid, dim3(32, kBY), 0, s, f, p);
}

template <typename T>
void launch_e_pml(const FieldView<T> &f, const PmlView<T> &p, cudaStream_t s)
{
    const SlabBoxes B = slab_boxes(p, f.d, true);
    if (B.n > 0) k_pml<T, true><<<B.start[B.n], dim3(32, kBY), 0, s>>>(f, p, B);
}

template <typename T>
void launch_h_pml(const FieldView<T> &f, const PmlView<T> &p, cudaStream_t s)
{
    const SlabBoxes B = slab_boxes(p, f.d, false);
    if (B.n > 0) k_pml<T, false><<<B.start[B.n], dim3(32, kBY), 0, s>>>(f, p, B);
}

template <typename T>
void launch_dl(const FieldView<T> &f, const DlView<T> &d, cudaStream_t s)
{
    if (d.ncell <= 0) return;
    k_dl<T><<<cdiv(d.ncell, 128), 128, 0, s>>>(f, d);
}

template <typename T>
void launch_gain(const FieldView<T> &f, const GainView<T> &g, int which, cudaStream_t s)
{
    if (g.ncell <= 0) return;
    if (sizeof(T) == 8)
        k_gain<T, GainSite64><<<cdiv(g.ncell, 128), 128, 0, s>>>(f, g, which);
    else
        k_gain<T, GainSite32><<<cdiv(g.ncell, 128), 128, 0, s>>>(f, g, which);
}

void launch_gain_pops32(const float *state, const int64_t *cell, int64_t ncell, float *out, cudaStream_t s)
{
    if (ncell <= 0) return;
    k_gain_pops32<<<cdiv(ncell, 256), 256, 0, s>>>(state, cell, ncell, out);
}

void launch_gain_init64(double *state, int64_t ncell, cudaStream_t s)
{
    if (ncell <= 0) return;
    k_gain_init64<<<cdiv(ncell, 256), 256, 0, s>>>(state, ncell);
}

template <typename T>
void launch_inject(const FieldView<T> &f, const InjTarget *tg, int ntarget, const InjContrib *ct,
                   const T *table, int Nt, double n, uint32_t face_mask, cudaStream_t s)
{
    if (ntarget <= 0) return;
    launch_pdl(true, k_inject<T>, cdiv(ntarget, 128), 128, 0, s, f, tg, ntarget, ct, table, Nt, n, face_mask);
}

template <typename T>
void launch_inject_pack(void *pack, const InjTarget *tg, int ntarget, const InjContrib *ct, cudaStream_t s)
{
    if (ntarget <= 0) return;
    InjView<T> v;
    inj_pack_view(v, pack, ntarget);
    k_inject_pack<T><<<cdiv(ntarget, 256), 256, 0, s>>>((uint64_t *)v.word, (double *)v.delay, (Pair<T> *)v.cp, tg,
                                                        ntarget, ct);
}

template <typename T>
void launch_inject_all(const FieldView<T> &f, const InjView<T> &v, const int64_t *n0, int64_t n, bool early,
                       cudaStream_t s)
{
    if (v.n <= 0) return;
    launch_pdl(early, k_inject_all<T>, cdiv(v.n, kInjPerBlock), kInjThreads, 0, s, f, v, n0, n);
}

template <typename T>
void launch_sources(const FieldView<T> &f, int nsrc, const int64_t *idx, const int32_t *comp,
                    const double *waves, const int32_t *wave_off, const int32_t *wave_len, int n,
                    cudaStream_t s)
{
    if (nsrc <= 0) return;
    launch_pdl(true, k_sources<T>, cdiv(nsrc, 64), 64, 0, s, f, nsrc, idx, comp, waves, wave_off, wave_len, n);
}

template <typename T>
void launch_inject_batch(const BatchGrid<T> *grids, const int4 *blocks, int nblocks, int side, int step_off,
                         cudaStream_t s)
{
    if (nblocks <= 0) return;
    k_inject_batch<T><<<nblocks, kInjThreads, 0, s>>>(grids, blocks, side, step_off);
}

template <typename T>
void launch_sources_batch(const BatchGrid<T> *grids, const int2 *ents, int n, int step_off, cudaStream_t s)
{
    if (n <= 0) return;
    k_sources_batch<T><<<cdiv(n, 64), 64, 0, s>>>(grids, ents, n, step_off);
}

#define CPS_INSTANTIATE(T)                                                                              \
    template void launch_h_bulk<T>(const FieldView<T> &, const PmlView<T> &, bool, cudaStream_t);       \
    template void launch_e_bulk<T>(const FieldView<T> &, const PmlView<T> &, bool, cudaStream_t);       \
    template void launch_h_pml<T>(const FieldView<T> &, const PmlView<T> &, cudaStream_t);              \
    template void launch_e_pml<T>(const FieldView<T> &, const PmlView<T> &, cudaStream_t);              \
    template void launch_dl<T>(const FieldView<T> &, const DlView<T> &, cudaStream_t);                  \
    template void launch_gain<T>(const FieldView<T> &, const GainView<T> &, int, cudaStream_t);         \
    template void launch_inject_pack<T>(void *, const InjTarget *, int, const InjContrib *, cudaStream_t); \
    template void launch_inject_all<T>(const FieldView<T> &, const InjView<T> &, const int64_t *, int64_t, bool, \
                                       cudaStream_t);                                                    \
    template void launch_inject<T>(const FieldView<T> &, const InjTarget *, int, const InjContrib *,    \
                                   const T *, int, double, uint32_t, cudaStream_t);                     \
    template void launch_sources<T>(const FieldView<T> &, int, const int64_t *, const int32_t *,        \
                                    const double *, const int32_t *, const int32_t *, int, cudaStream_t); \
    template void launch_inject_batch<T>(const BatchGrid<T> *, const int4 *, int, int, int, cudaStream_t); \
    template void launch_sources_batch<T>(const BatchGrid<T> *, const int2 *, int, int, cudaStream_t);
CPS_INSTANTIATE(double)
CPS_INSTANTIATE(float)

}  // namespace cps
