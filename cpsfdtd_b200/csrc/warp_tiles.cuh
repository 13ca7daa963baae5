// warp_tiles.cuh -- per-tile bodies of the fused H and E sweeps: one warp per
// tile, one 16-byte vector of cells per lane.
//
// A tile is a 32 x BY block of (i, j) columns marching planes [k0, k1) in k.
// A warp covers 32 columns x RY rows (FP32: 8 lanes x 4 cells, 4 rows; FP64:
// 16 lanes x 2 cells, 2 rows) and takes G = BY / RY such groups per plane.
// Lane 0 keeps the planes ahead in flight with TMA loads into the warp's own
// ring of stages of P planes each: one box per side for the three components
// with their halo, one for the swept side's, one for the material IDs and one
// per CPML axis the tile meets for its two psi words.  One mbarrier per stage, no block barrier anywhere.
//
// What bounds these sweeps is DRAM as long as the warps get through a plane
// fast enough: 128 FP32 cells are 4.7 KB of traffic, 110 ns of an SM's share
// of the bandwidth.  So the plane loop is kept short of instructions (vectors,
// few boxes, P planes per wait, one look-up of the material coefficients when
// the warp holds one medium) and free of global loads: one that misses costs a
// microsecond or more while DRAM is saturated.  What varies along k (stretch
// factors, z-slab coefficients) is loaded 32 planes at a time, one plane per
// lane, and broadcast by shuffles.
//
// Measured against block tiles with one cell per thread (B200, FP32, CPML):
// 301x419x262, H sweep 262 -> 235 us and E sweep 287 -> 228 us (DRAM at 76 % of
// its peak, 1.41 GB a sweep); 256^3 dispersive, H 147 -> 127 us; 384^3 laser, H 424 ->
// 380 us.  E sweeps with gain stay on block tiles (a lane with four cells' gain
// words leaves six warps per SM: 1407 us either way at 384^3, 6 % slower at
// 150x117x98), and so does the FP64 H sweep (90 against 100 us at 165x150x181).
//
// The arithmetic of a cell is that of the bodies in tma_bodies.cuh, operation
// by operation (sweep_cells.cuh), so results do not depend on which kernel,
// tile or launch processed a cell.
#pragma once

#include "tma_bodies.cuh"

namespace cps {

template <typename T>
struct alignas(16) Vec {
    static constexpr int N = 16 / (int)sizeof(T);
    T v[N];
};

template <typename T>
__device__ __forceinline__ Vec<T> vld(const T *p)
{
    return *reinterpret_cast<const Vec<T> *>(p);
}
template <typename T>
__device__ __forceinline__ void vst(T *p, const Vec<T> &a)
{
    *reinterpret_cast<Vec<T> *>(p) = a;
}
// tile q of a grid of nbx x nby tiles per plane row of tiles, x fastest
__device__ __forceinline__ TileXYZ grid_tile(int q, int nbx, int nby)
{
    const int r = q / nbx, z = r / nby;
    return TileXYZ{q - r * nbx, r - z * nby, z};
}

constexpr int kMaxStages = 10;
// mbarriers of a warp's ring
__device__ __forceinline__ void init_ring(uint64_t *full)
{
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) mbar_init(&full[s], 1);
        fence_mbar_init();
    }
    __syncwarp();
}

// lanes of a warp over the tile's columns and rows
template <typename T>
struct WarpShape {
    static constexpr int V = Vec<T>::N;     // cells per lane
    static constexpr int LX = 32 / V;       // lanes across the 32 columns
    static constexpr int RY = 32 / LX;      // rows a warp covers at once
};

// The planes per stage of a tile: two where the stage holds fields alone, one
// with psi words (two such stages would not leave enough warps per SM)
constexpr int kPlanes = 2;

// Stage of P planes (offsets in bytes): halo components [3][P][BY+1][36], own
// components [3][P][BY][32], IDs [P][BY][32]; the psi boxes [2][P][BY][32] of
// each axis follow.
template <typename T, int BY, int P>
struct WarpStage {
    static constexpr int HROW = 36, HPL = HROW * (BY + 1), HC = P * HPL;  // elements: row, plane, component
    static constexpr int OPL = 32 * BY, OC = P * OPL;
    static constexpr int OWN = a128(3 * HC * (int)sizeof(T));
    static constexpr int ID = OWN + 3 * OC * (int)sizeof(T);
    static constexpr int BYTES = ID + a128(OC);
    static constexpr int PSI = 2 * OC * (int)sizeof(T);                   // one axis
    static constexpr uint32_t TX = 3 * HC * sizeof(T) + 3 * OC * sizeof(T) + OC;
    static constexpr uint32_t TAIL = 2 * HPL * sizeof(T);                 // Ex, Ey of one plane past the tile
};

template <typename T>
__device__ __forceinline__ Vec<T> splat(T a)
{
    Vec<T> r;
#pragma unroll
    for (int q = 0; q < Vec<T>::N; ++q) r.v[q] = a;
    return r;
}

// cells of a vector inside [lo, hi)
template <int V>
__device__ __forceinline__ unsigned cells_in(int i0, int lo, int hi)
{
    unsigned m = 0;
#pragma unroll
    for (int q = 0; q < V; ++q) m |= (i0 + q >= lo && i0 + q < hi) ? 1u << q : 0u;
    return m;
}

// ---- CPML.  E slabs are [1, np] and [n-np, n-1], H slabs [0, np-1] and
// [n-np, n-1] on each axis.

// face of index `at` on an axis (f1 its first face), -1 none, and the slab index
__device__ __forceinline__ int slab_face(const int np[6], int f1, int n, int at, bool eside, int &s)
{
    s = at;
    if (at < np[f1] + (eside ? 1 : 0)) return f1;
    s = at - (n - np[f1 + 1]);
    return s >= 0 ? f1 + 1 : -1;
}

// first face of an axis that [lo, hi] meets, -1 none
__device__ __forceinline__ int tile_face(const int np[6], int f1, int n, int lo, int hi, bool eside)
{
    if (lo < np[f1] + (eside ? 1 : 0)) return f1;
    return hi >= n - np[f1 + 1] ? f1 + 1 : -1;
}

// The x slab of a lane's vector: the face it meets (-1 none) and the
// coefficients of its cells, zero outside the slab.  A vector meets both ends
// only when fewer than a vector of cells lie between the slabs; its second end
// is then `also`, handled cell by cell.
template <typename T>
struct VecX {
    int fx, s0, also;
    unsigned in;  // cells of the vector inside the slab
    Vec<T> b, c;
};

template <typename T, bool ESIDE>
__device__ __forceinline__ VecX<T> vec_x(const PmlView<T> &p, const Dims &d, int i0)
{
    constexpr int V = Vec<T>::N, lo = ESIDE ? 1 : 0;
    VecX<T> x;
    x.fx = x.also = -1;
    x.s0 = 0;
    x.in = 0;
    x.b = splat(T(0));
    x.c = splat(T(0));
    const bool m1 = i0 + V - 1 >= lo && i0 < lo + p.np[kFX1];
    const bool m2 = i0 + V - 1 >= d.nx - p.np[kFX2] && i0 < d.nx;
    if (m1) {
        x.fx = kFX1;
        if (m2) x.also = kFX2;
    } else if (m2) {
        x.fx = kFX2;
    }
    if (x.fx < 0) return x;
    const int f = x.fx, np = p.np[f];
    x.s0 = f == kFX1 ? i0 : i0 - (d.nx - np);
    const T *b = ESIDE ? p.bE[f] : p.bH[f], *c = ESIDE ? p.cE[f] : p.cH[f];
    const int s_lo = f == kFX1 ? lo : 0, s_hi = f == kFX1 ? lo + np : np;
#pragma unroll
    for (int q = 0; q < V; ++q) {
        const int s = x.s0 + q;
        if (s >= s_lo && s < s_hi) {
            x.b.v[q] = b[s];
            x.c.v[q] = c[s];
            x.in |= 1u << q;
        }
    }
    return x;
}


// The psi boxes a tile stages with its planes: at most one face per axis (a
// tile that meets both ends of x or y reads the second end's psi from global
// memory; on z the face is the plane's).  ox, oy, oz: byte offsets in the
// stage; oz < 0: no plane of the tile lies in a z slab.
struct TilePsi {
    int fx, fy;
    int ox, oy, oz;
    int bytes;  // of the stage
};

template <typename T, int BY, bool ESIDE>
__device__ __forceinline__ TilePsi tile_psi(const PmlView<T> &p, const Dims &d, int x0, int y0, int k0, int k1,
                                            int base, int psi)
{
    TilePsi t;
    t.fx = tile_face(p.np, kFX1, d.nx, x0, x0 + 31, ESIDE);
    t.fy = tile_face(p.np, kFY1, d.ny, y0, y0 + BY - 1, ESIDE);
    t.ox = base;
    t.oy = t.ox + (t.fx >= 0 ? psi : 0);
    t.bytes = t.oy + (t.fy >= 0 ? psi : 0);
    t.oz = -1;
    if (tile_face(p.np, kFZ1, d.nz, k0, k1 - 1, ESIDE) >= 0) {
        t.oz = t.bytes;
        t.bytes += psi;
    }
    return t;
}

// z face that planes [k, k + P) meet (at most one: an interior lies between
// the slabs), -1 none, and the slab index of plane k (-1 possible)
__device__ __forceinline__ int pair_face(const int np[6], int n, int k, int P, bool eside, int &s)
{
    s = k;
    if (k < np[kFZ1] + (eside ? 1 : 0)) return kFZ1;
    s = k - (n - np[kFZ2]);
    return s + P > 0 && k < n ? kFZ2 : -1;
}

// one pair of psi vectors of a slab, a = b psi + c d: written back whole when
// `wr` allows every cell, else the cells of `wr`.  Cells with zero coefficients
// or outside the update range hold words nobody reads.
template <typename T>
__device__ __forceinline__ void psi_pair(const T *p0, const T *p1, const Vec<T> &b, const Vec<T> &c, const Vec<T> &d0,
                                         const Vec<T> &d1, unsigned wr, T *q0, T *q1, Vec<T> &a0, Vec<T> &a1)
{
    constexpr int V = Vec<T>::N;
    const Vec<T> o0 = vld(p0), o1 = vld(p1);
#pragma unroll
    for (int q = 0; q < V; ++q) {
        a0.v[q] = psi_new(b.v[q], o0.v[q], c.v[q], d0.v[q]);
        a1.v[q] = psi_new(b.v[q], o1.v[q], c.v[q], d1.v[q]);
    }
    if (wr == (1u << V) - 1) {
        vst(q0, a0);
        vst(q1, a1);
    } else if (wr) {
#pragma unroll
        for (int q = 0; q < V; ++q)
            if ((wr >> q) & 1u) { q0[q] = a0.v[q]; q1[q] = a1.v[q]; }
    }
}

// row coefficients of the y slab
template <typename T>
struct RowY {
    int f, s;
    T b, c;
};

// CPML corrections of a vector, x then y then z slabs.  The differences are
// named by the component pairs of the slabs: (dx0, dx1) along i, (dy0, dy1)
// along j, (dz0, dz1) along k, and F1..F3 the components x, y, z.
//   E: dx = (dHz_i, dHy_i), dy = (dHx_j, dHz_j), dz = (dHy_k, dHx_k),
//      Ey -= x0, Ez += x1; Ez -= y0, Ex += y1; Ex -= z0, Ey += z1 (times ce)
//   H: dx = (dEz_i, dEy_i), dy = (dEx_j, dEz_j), dz = (dEy_k, dEx_k),
//      Hy += x0, Hz -= x1; Hz -= y0, Hx += y1; Hx -= z0, Hy += z1 (times ch)
// st: the plane's stage at this vector's place in its boxes, oc: elements
// between the two words; fz, sz, bz, cz: the plane's z slab; wr: the cells
// whose psi may be written.
template <typename T, bool ESIDE>
__device__ __forceinline__ void pml_vec(const PmlView<T> &p, const Dims &d, const TilePsi &tp, const unsigned char *st,
                                        int oc, const VecX<T> &x, const RowY<T> &y, int fz, int sz, T bz, T cz,
                                        const Vec<T> &cc, int i0, int j, int k, unsigned wr, const Vec<T> &dx0,
                                        const Vec<T> &dx1, const Vec<T> &dy0, const Vec<T> &dy1, const Vec<T> &dz0,
                                        const Vec<T> &dz1, Vec<T> &F1, Vec<T> &F2, Vec<T> &F3)
{
    constexpr int V = Vec<T>::N;
    Vec<T> a0, a1;
    if (x.fx >= 0) {
        T *const *q = ESIDE ? p.qe[x.fx] : p.qh[x.fx];
        const int64_t g = ((int64_t)k * (d.ny + 1) + j) * psi_xw(p.np[x.fx]) + x.s0;
        const bool staged = x.fx == tp.fx;
        const T *p0 = staged ? (const T *)(st + tp.ox) : q[0] + g;
        const T *p1 = staged ? (const T *)(st + tp.ox) + oc : q[1] + g;
        psi_pair(p0, p1, x.b, x.c, dx0, dx1, wr, q[0] + g, q[1] + g, a0, a1);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const bool in = (x.in >> e) & 1u;
            const T u0 = in ? a0.v[e] : T(0), u1 = in ? a1.v[e] : T(0);
            F2.v[e] = ESIDE ? psi_sub(F2.v[e], u0, cc.v[e]) : psi_add(F2.v[e], u0, cc.v[e]);
            F3.v[e] = ESIDE ? psi_add(F3.v[e], u1, cc.v[e]) : psi_sub(F3.v[e], u1, cc.v[e]);
        }
        if (x.also >= 0) {  // the vector meets the second end too: its cells one by one
            const int f = x.also, np = p.np[f], s0 = i0 - (d.nx - np);
            const T *bt = ESIDE ? p.bE[f] : p.bH[f], *ct = ESIDE ? p.cE[f] : p.cH[f];
            T *const *q2 = ESIDE ? p.qe[f] : p.qh[f];
            const int64_t g2 = ((int64_t)k * (d.ny + 1) + j) * psi_xw(np) + s0;
#pragma unroll
            for (int e = 0; e < V; ++e) {
                if (s0 + e < 0 || s0 + e >= np) continue;
                const T b0 = psi_new(bt[s0 + e], q2[0][g2 + e], ct[s0 + e], dx0.v[e]);
                const T b1 = psi_new(bt[s0 + e], q2[1][g2 + e], ct[s0 + e], dx1.v[e]);
                if ((wr >> e) & 1u) { q2[0][g2 + e] = b0; q2[1][g2 + e] = b1; }
                F2.v[e] = ESIDE ? psi_sub(F2.v[e], b0, cc.v[e]) : psi_add(F2.v[e], b0, cc.v[e]);
                F3.v[e] = ESIDE ? psi_add(F3.v[e], b1, cc.v[e]) : psi_sub(F3.v[e], b1, cc.v[e]);
            }
        }
    }
    if (y.f >= 0) {
        T *const *q = ESIDE ? p.qe[y.f] : p.qh[y.f];
        const int64_t g = ((int64_t)k * (p.np[y.f] + 1) + y.s) * d.px + i0;
        const bool staged = y.f == tp.fy;
        const T *p0 = staged ? (const T *)(st + tp.oy) : q[0] + g;
        const T *p1 = staged ? (const T *)(st + tp.oy) + oc : q[1] + g;
        psi_pair(p0, p1, splat(y.b), splat(y.c), dy0, dy1, wr, q[0] + g, q[1] + g, a0, a1);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            F3.v[e] = psi_sub(F3.v[e], a0.v[e], cc.v[e]);
            F1.v[e] = psi_add(F1.v[e], a1.v[e], cc.v[e]);
        }
    }
    if (fz >= 0) {
        T *const *q = ESIDE ? p.qe[fz] : p.qh[fz];
        const int64_t g = ((int64_t)sz * (d.ny + 1) + j) * d.px + i0;
        psi_pair((const T *)(st + tp.oz), (const T *)(st + tp.oz) + oc, splat(bz), splat(cz), dz0, dz1, wr, q[0] + g,
                 q[1] + g, a0, a1);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            F1.v[e] = psi_sub(F1.v[e], a0.v[e], cc.v[e]);
            F2.v[e] = psi_add(F2.v[e], a1.v[e], cc.v[e]);
        }
    }
}

// packed material IDs of a vector
template <typename T>
__device__ __forceinline__ unsigned vec_ids(const uint8_t *p)
{
    if (Vec<T>::N == 4) return *reinterpret_cast<const uint32_t *>(p);
    return *reinterpret_cast<const uint16_t *>(p);
}

// (a, b) of the media of a vector's cells; one look-up when the whole warp
// holds one medium, which the return value says (its ID, -1 mixed)
template <typename T>
__device__ __forceinline__ int vec_coefs(unsigned ids, const Coef2<T> *tab, const T *ga, const T *gb, Vec<T> &a,
                                         Vec<T> &b)
{
    constexpr int V = Vec<T>::N;
    const unsigned first = __shfl_sync(0xffffffffu, ids, 0), id0 = first & 255u;
    const bool one = __all_sync(0xffffffffu, ids == id0 * (V == 4 ? 0x01010101u : 0x0101u));
    if (one && id0 < (unsigned)kTab) {
        const Coef2<T> c = tab[id0];
        a = splat(c.a);
        b = splat(c.b);
        return (int)id0;
    }
#pragma unroll
    for (int q = 0; q < V; ++q) {
        const unsigned id = (ids >> (8 * q)) & 255u;
        Coef2<T> c = tab[id & (kTab - 1)];
        if (id >= (unsigned)kTab) {
            c.a = __ldg(&ga[id]);
            c.b = __ldg(&gb[id]);
        }
        a.v[q] = c.a;
        b.v[q] = c.b;
    }
    return -1;
}

// store a field vector: whole when `wr` allows every cell (cells that are not
// updated then carry their old value), else the cells of `wr`
template <typename T>
__device__ __forceinline__ void field_vst(T *p, const Vec<T> &a, unsigned wr)
{
    constexpr int V = Vec<T>::N;
    if (wr == (1u << V) - 1) {
        vst(p, a);
    } else if (wr) {
#pragma unroll
        for (int q = 0; q < V; ++q)
            if ((wr >> q) & 1u) p[q] = a.v[q];
    }
}

// Shared memory of a warp's ring (with 128 spare bytes to align it): two stages
// of two planes, or of one plane of a tile that meets a CPML slab on every axis.
template <typename T, int BY>
__host__ __device__ constexpr int warp_ring()
{
    constexpr int a = 2 * WarpStage<T, BY, kPlanes>::BYTES;
    constexpr int b = 2 * (WarpStage<T, BY, 1>::BYTES + 3 * WarpStage<T, BY, 1>::PSI);
    return (a > b ? a : b) + 128;
}

// A warp's ring of stages: shared memory, one mbarrier per stage and, per
// barrier, the parity of its next phase (bit s of ph; every load that was
// issued is waited for before a tile ends, so the bits carry over to the
// warp's next tile).
struct Ring {
    unsigned char *sm;
    uint64_t *full;
    int bytes;      // of shared memory
    uint32_t ph;
    uint32_t skew;  // test setting: extra bytes the first plane of a tile expects
    int *err;
};

// the whole warp waits for stage s; false when the wait gave up
__device__ __forceinline__ bool ring_wait(Ring &r, int s)
{
    const bool ok = wait_stage(&r.full[s], (r.ph >> s) & 1u);
    if (__any_sync(0xffffffffu, !ok)) return false;
    r.ph ^= 1u << s;
    return true;
}

// after a wait gave up: lane 0 records the code and waits (bounded) for the n
// stages from s whose loads may still be in flight, so that no copy outlives
// the block
__device__ __forceinline__ void ring_fail(const Ring &r, int code, int s, int n, int ns)
{
    if (threadIdx.x != 0) return;
    atomicExch(r.err, code);
    for (int q = 0; q < n; ++q, s = s + 1 == ns ? 0 : s + 1) wait_stage(&r.full[s], (r.ph >> s) & 1u);
}

// stages of stage_b bytes in a ring (two at least fit every layout)
__device__ __forceinline__ int ring_stages(const Ring &r, int stage_b) { return min(kMaxStages, r.bytes / stage_b); }

// what varies along k for a warp: lane l holds the values of plane k0 + 32 m + l
template <typename T>
struct Along {
    T c0, c1;  // stretch factors
    T b, c;    // z-slab coefficients (0 outside)
};

template <typename T, bool ESIDE, bool PML>
__device__ __forceinline__ Along<T> along_k(const FieldView<T> &f, const PmlView<T> &p, int k)
{
    Along<T> r{T(0), T(0), T(0), T(0)};
    if (k >= f.d.nz) return r;
    r.c0 = ESIDE ? f.s.cExy[k] : f.s.cHxy[k];
    r.c1 = ESIDE ? f.s.cEyx[k] : f.s.cHyx[k];
    if (PML) {
        int s;
        const int fz = slab_face(p.np, kFZ1, f.d.nz, k, ESIDE, s);
        if (fz >= 0) {
            r.b = ESIDE ? p.bE[fz][s] : p.bH[fz][s];
            r.c = ESIDE ? p.cE[fz][s] : p.cH[fz][s];
        }
    }
    return r;
}

// stretch factors of a lane's columns (the arrays are padded to vectors)
template <typename T>
__device__ __forceinline__ Vec<T> along_i(const T *c, int i0, int nx)
{
    return vld(c + min(i0, (nx - 1) / Vec<T>::N * Vec<T>::N));
}

// the psi boxes of a stage's planes from k; returns their bytes
template <typename T, int BY, int P, bool ESIDE>
__device__ __forceinline__ uint32_t psi_bytes(const PmlView<T> &p, const Dims &d, const TilePsi &tp, int k, int &fz,
                                              int &sz)
{
    using L = WarpStage<T, BY, P>;
    fz = -1;
    if (tp.oz >= 0) fz = pair_face(p.np, d.nz, k, P, ESIDE, sz);
    return (tp.fx >= 0 ? L::PSI : 0) + (tp.fy >= 0 ? L::PSI : 0) + (fz >= 0 ? L::PSI : 0);
}

template <typename T>
__device__ __forceinline__ void psi_issue(const SweepMaps &M, const PmlView<T> &p, const Dims &d, const TilePsi &tp,
                                          unsigned char *b, uint64_t *bar, int x0, int y0, int k, int fz, int sz)
{
    if (tp.fx >= 0)
        tma_load_4d(b + tp.ox, &M.psi[tp.fx], bar, tp.fx == kFX1 ? x0 : x0 - ((d.nx - p.np[kFX2]) & ~3), y0, k, 0);
    if (tp.fy >= 0)
        tma_load_4d(b + tp.oy, &M.psi[tp.fy], bar, x0, tp.fy == kFY1 ? y0 : y0 - (d.ny - p.np[kFY2]), k, 0);
    if (fz >= 0) tma_load_4d(b + tp.oz, &M.psi[fz], bar, x0, y0, sz, 0);
}

// H sweep of one tile by one warp: planes bz*kc .. min(bz*kc+kc, nz)-1 (kc a
// multiple of P); Ex and Ey of the plane past the last come with its stage or
// in a short stage of their own.
template <typename T, int BY, int P, bool PML>
__device__ __forceinline__ bool h_warp_tile(const SweepMaps &M, const FieldView<T> &f, const PmlView<T> &p, int kc,
                                            TileXYZ t, Ring &R, const Coef2<T> *tab)
{
    static_assert(!PML || P == 1, "psi boxes hold one plane");
    using L = WarpStage<T, BY, P>;
    using W = WarpShape<T>;
    constexpr int V = W::V, G = BY / W::RY;
    const Dims d = f.d;
    const int lane = threadIdx.x, lx = lane % W::LX, ly = lane / W::LX;
    const int x0 = t.bx * 32, y0 = t.by * BY, i0 = x0 + lx * V;
    const int k0 = t.bz * kc, k1 = min(k0 + kc, d.nz);
    const int nst = (k1 - k0 + P - 1) / P, nload = nst + ((k1 - k0) % P == 0 ? 1 : 0);
    TilePsi tp{-1, -1, 0, 0, -1, L::BYTES};
    if (PML) tp = tile_psi<T, BY, false>(p, d, x0, y0, k0, k1, L::BYTES, L::PSI);
    const int stage_b = PML ? tp.bytes : L::BYTES, ns = ring_stages(R, stage_b);
    unsigned char *const sm = R.sm;
    int is = 0;  // stage of the next load
    auto issue = [&](int m) {
        const int k = k0 + m * P;
        unsigned char *b = sm + is * stage_b;
        uint64_t *bar = &R.full[is];
        is = is + 1 == ns ? 0 : is + 1;
        fence_proxy_async_smem();  // the stage's previous contents were read through the generic proxy
        if (m == nst) {
            mbar_expect_tx(bar, L::TAIL);
            tma_load_4d(b, &M.tail, bar, x0, y0, k, 0);
            return;
        }
        int fz = -1, sz = 0;
        uint32_t tx = L::TX;
        if (PML) tx += psi_bytes<T, BY, P, false>(p, d, tp, k, fz, sz);
        mbar_expect_tx(bar, tx + (m == 0 ? R.skew : 0u));
        tma_load_4d(b, &M.halo[P - 1], bar, x0, y0, k, 0);
        tma_load_4d(b + L::OWN, &M.own[P - 1], bar, x0, y0, k, 0);
        tma_load_3d(b + L::ID, &M.id[P - 1], bar, x0, y0, k);
        if (PML) psi_issue(M, p, d, tp, b, bar, x0, y0, k, fz, sz);
    };
    if (lane == 0)
        for (int m = 0; m < ns && m < nload; ++m) issue(m);
    const StretchView<T> &sv = f.s;
    const Vec<T> cHyz = along_i(sv.cHyz, i0, d.nx), cHzy = along_i(sv.cHzy, i0, d.nx);
    const bool edge = x0 + 32 > d.nx;  // some cells lie past the update range: they keep their value
    const unsigned act = cells_in<V>(i0, 0, d.nx);
    T cHxz[G], cHzx[G];
    RowY<T> ry[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const int j = min(y0 + g * W::RY + ly, d.ny - 1);
        cHxz[g] = sv.cHxz[j];
        cHzx[g] = sv.cHzx[j];
        if (PML) {
            ry[g].f = slab_face(p.np, kFY1, d.ny, j, false, ry[g].s);
            if (ry[g].f >= 0) {
                ry[g].b = p.bH[ry[g].f][ry[g].s];
                ry[g].c = p.cH[ry[g].f][ry[g].s];
            }
        }
    }
    VecX<T> px;
    if (PML) px = vec_x<T, false>(p, d, i0);
    Along<T> ak = along_k<T, false, PML>(f, p, k0 + lane);
    const int er = ly * L::HROW + lx * V, orow = ly * 32 + lx * V;
    if (!ring_wait(R, 0)) {
        ring_fail(R, 2, 1 % ns, min(ns - 1, nload - 1), ns);
        return false;
    }
    Vec<T> ex[G], ey[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        ex[g] = vld((const T *)sm + er + g * W::RY * L::HROW);
        ey[g] = vld((const T *)sm + L::HC + er + g * W::RY * L::HROW);
    }
    int s = 0;
    int64_t w0 = d.idx(i0, y0 + ly, k0);
    for (int m = 0; m < nst; ++m) {
        const int kb = k0 + m * P;
        if (m > 0 && (m * P & 31) == 0) ak = along_k<T, false, PML>(f, p, kb + lane);
        const unsigned char *b = sm + s * stage_b;
        const int sn = s + 1 == ns ? 0 : s + 1;
        int fzp = -1, szp = 0;
        if (PML && tp.oz >= 0) fzp = pair_face(p.np, d.nz, kb, P, false, szp);
#pragma unroll
        for (int u = 0; u < P; ++u) {
            const int k = kb + u;
            if (k >= k1) break;
            // Ex and Ey of the next plane: this stage's, or the next one's
            const T *nxp = (const T *)b + (u + 1) * L::HPL;
            int nc = L::HC;
            if (u + 1 == P) {
                if (!ring_wait(R, sn)) {
                    ring_fail(R, 2, sn + 1 == ns ? 0 : sn + 1, min(ns - 2, nload - m - 2), ns);
                    return false;
                }
                nxp = (const T *)(sm + sn * stage_b);
                nc = m + 1 == nst ? L::HPL : L::HC;
            }
            const int kl = (m * P + u) & 31;
            const T cHxy = __shfl_sync(0xffffffffu, ak.c0, kl), cHyx = __shfl_sync(0xffffffffu, ak.c1, kl);
            T bz = T(0), cz = T(0);
            int fz = -1;
            if (PML && fzp >= 0) {
                bz = __shfl_sync(0xffffffffu, ak.b, kl);
                cz = __shfl_sync(0xffffffffu, ak.c, kl);
                if (szp + u >= 0 && szp + u < p.np[fzp]) fz = fzp;
            }
            const T *ext = (const T *)b + u * L::HPL, *hxt = (const T *)(b + L::OWN) + u * L::OPL;
            const uint8_t *idt = b + L::ID + u * L::OPL;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int e = er + g * W::RY * L::HROW, o = orow + g * W::RY * 32;
                const Vec<T> exk = vld(nxp + e), eyk = vld(nxp + nc + e);
                const T *ezt = ext + 2 * L::HC, *eyt = ext + L::HC;
                const Vec<T> ez = vld(ezt + e), exj = vld(ext + e + L::HROW), ezj = vld(ezt + e + L::HROW);
                const T eyi = eyt[e + V], ezi = ezt[e + V];
                const Vec<T> ox = vld(hxt + o), oy = vld(hxt + L::OC + o), oz = vld(hxt + 2 * L::OC + o);
                Vec<T> hx, hy, hz, dEz_i, dEz_j, dEx_j, dEy_i, dEx_k, dEy_k, aH, bH;
                vec_coefs(vec_ids<T>(idt + o), tab, f.aH, f.bH, aH, bH);
#pragma unroll
                for (int q = 0; q < V; ++q) {
                    const T ey_n = q + 1 < V ? ey[g].v[q + 1 < V ? q + 1 : 0] : eyi;
                    const T ez_n = q + 1 < V ? ez.v[q + 1 < V ? q + 1 : 0] : ezi;
                    dEz_i.v[q] = ez_n - ez.v[q];
                    dEz_j.v[q] = ezj.v[q] - ez.v[q];
                    dEx_j.v[q] = exj.v[q] - ex[g].v[q];
                    dEy_i.v[q] = ey_n - ey[g].v[q];
                    dEx_k.v[q] = exk.v[q] - ex[g].v[q];
                    dEy_k.v[q] = eyk.v[q] - ey[g].v[q];
                    hx.v[q] = yee_n(aH.v[q], ox.v[q], bH.v[q], dEz_j.v[q], cHxz[g], dEy_k.v[q], cHxy);
                    hy.v[q] = yee_n(aH.v[q], oy.v[q], bH.v[q], dEx_k.v[q], cHyx, dEz_i.v[q], cHyz.v[q]);
                    hz.v[q] = yee_z(aH.v[q], oz.v[q], bH.v[q], dEx_j.v[q], cHzx[g], dEy_i.v[q], cHzy.v[q]);
                }
                const int j = y0 + g * W::RY + ly;
                const bool row = j < d.ny;
                if (PML) {
                    if (p.literal) bH = splat(p.cpmlH);
                    pml_vec<T, false>(p, d, tp, b + (u * L::OPL + o) * (int)sizeof(T), L::OC, px, ry[g], fz, szp + u,
                                      bz, cz, bH, i0, row ? j : 0, k, row ? act : 0u, dEz_i, dEy_i, dEx_j, dEz_j, dEy_k, dEx_k,
                                      hx, hy, hz);
                }
                if (edge) {
#pragma unroll
                    for (int q = 0; q < V; ++q)
                        if (!((act >> q) & 1u)) { hx.v[q] = ox.v[q]; hy.v[q] = oy.v[q]; hz.v[q] = oz.v[q]; }
                }
                if (row) {
                    const int64_t w = w0 + (int64_t)(g * W::RY) * d.px;
                    vst(f.Hx + w, hx);
                    vst(f.Hy + w, hy);
                    vst(f.Hz + w, hz);
                }
                ex[g] = exk;
                ey[g] = eyk;
            }
            w0 += d.pxy;
        }
        s = sn;
        __syncwarp();
        if (lane == 0 && m + ns < nload) issue(m + ns);
    }
    return true;
}

// E sweep of one tile by one warp: planes max(1, bz*kc) .. min(bz*kc+kc, nz)-1
// (plane 0 is staged for its H alone).
template <typename T, int BY, int P, bool PML, bool DL>
__device__ __forceinline__ bool e_warp_tile(const SweepMaps &M, const FieldView<T> &f, const PmlView<T> &p, int kc,
                                            TileXYZ t, Ring &R, const Coef2<T> *tab)
{
    static_assert(!PML || P == 1, "psi boxes hold one plane");
    using L = WarpStage<T, BY, P>;
    using W = WarpShape<T>;
    constexpr int V = W::V, G = BY / W::RY;
    constexpr unsigned ALL = (1u << V) - 1;
    const Dims d = f.d;
    const int lane = threadIdx.x, lx = lane % W::LX, ly = lane / W::LX;
    const int x0 = t.bx * 32, y0 = t.by * BY, i0 = x0 + lx * V;
    const int k0 = t.bz * kc, k1 = min(k0 + kc, d.nz);
    const int nst = (k1 - k0 + P - 1) / P;
    TilePsi tp{-1, -1, 0, 0, -1, L::BYTES};
    if (PML) tp = tile_psi<T, BY, true>(p, d, x0, y0, max(k0, 1), k1, L::BYTES, L::PSI);
    const int stage_b = PML ? tp.bytes : L::BYTES, ns = ring_stages(R, stage_b);
    unsigned char *const sm = R.sm;
    int is = 0;  // stage of the next load
    auto issue = [&](int m) {
        const int k = k0 + m * P;
        unsigned char *b = sm + is * stage_b;
        uint64_t *bar = &R.full[is];
        is = is + 1 == ns ? 0 : is + 1;
        int fz = -1, sz = 0;
        uint32_t tx = L::TX;
        if (PML) tx += psi_bytes<T, BY, P, true>(p, d, tp, k, fz, sz);
        fence_proxy_async_smem();  // the stage's previous contents were read through the generic proxy
        mbar_expect_tx(bar, tx + (m == 0 ? R.skew : 0u));
        tma_load_4d(b, &M.halo[P - 1], bar, x0 - 4, y0 - 1, k, 0);
        tma_load_4d(b + L::OWN, &M.own[P - 1], bar, x0, y0, k, 0);
        tma_load_3d(b + L::ID, &M.id[P - 1], bar, x0, y0, k);
        if (PML) psi_issue(M, p, d, tp, b, bar, x0, y0, k, fz, sz);
    };
    if (lane == 0)
        for (int m = 0; m < ns && m < nst; ++m) issue(m);
    const StretchView<T> &sv = f.s;
    const Vec<T> cEyz = along_i(sv.cEyz, i0, d.nx), cEzy = along_i(sv.cEzy, i0, d.nx);
    const bool edge = x0 == 0 || x0 + 32 > d.nx;
    const unsigned act = cells_in<V>(i0, 1, d.nx);
    T cExz[G], cEzx[G];
    Vec<T> hxm[G], hym[G];
    RowY<T> ry[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const int j = min(max(y0 + g * W::RY + ly, 1), d.ny - 1);
        cExz[g] = sv.cExz[j];
        cEzx[g] = sv.cEzx[j];
        const int64_t w = d.idx(i0, j, max(k0 - 1, 0));
        hxm[g] = vld(f.Hx + w);
        hym[g] = vld(f.Hy + w);
        if (PML) {
            ry[g].f = slab_face(p.np, kFY1, d.ny, j, true, ry[g].s);
            if (ry[g].f >= 0) {
                ry[g].b = p.bE[ry[g].f][ry[g].s];
                ry[g].c = p.cE[ry[g].f][ry[g].s];
            }
        }
    }
    VecX<T> px;
    if (PML) px = vec_x<T, true>(p, d, i0);
    Along<T> ak = along_k<T, true, PML>(f, p, k0 + lane);
    const int hr = (ly + 1) * L::HROW + lx * V + 4, orow = ly * 32 + lx * V;
    int s = 0;
    int64_t w0 = d.idx(i0, y0 + ly, k0);
    for (int m = 0; m < nst; ++m) {
        const int kb = k0 + m * P;
        if (m > 0 && (m * P & 31) == 0) ak = along_k<T, true, PML>(f, p, kb + lane);
        int fzp = -1, szp = 0;
        if (PML && tp.oz >= 0) fzp = pair_face(p.np, d.nz, kb, P, true, szp);
        if (!ring_wait(R, s)) {
            ring_fail(R, 1, s + 1 == ns ? 0 : s + 1, min(ns - 1, nst - m - 1), ns);
            return false;
        }
        const unsigned char *b = sm + s * stage_b;
#pragma unroll
        for (int u = 0; u < P; ++u) {
            const int k = kb + u;
            if (k >= k1) break;
            const T *hxt = (const T *)b + u * L::HPL, *hyt = hxt + L::HC, *hzt = hxt + 2 * L::HC;
            const T *ext = (const T *)(b + L::OWN) + u * L::OPL;
            const uint8_t *idt = b + L::ID + u * L::OPL;
            const int kl = (m * P + u) & 31;
            const T cExy = __shfl_sync(0xffffffffu, ak.c0, kl), cEyx = __shfl_sync(0xffffffffu, ak.c1, kl);
            T bz = T(0), cz = T(0);
            int fz = -1;
            if (PML && fzp >= 0) {
                bz = __shfl_sync(0xffffffffu, ak.b, kl);
                cz = __shfl_sync(0xffffffffu, ak.c, kl);
                if (fzp == kFZ1 ? szp + u <= p.np[kFZ1] : szp + u >= 0) fz = fzp;
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int h = hr + g * W::RY * L::HROW, o = orow + g * W::RY * 32;
                const Vec<T> hx = vld(hxt + h), hy = vld(hyt + h);
                if (k > 0) {
                    const Vec<T> hz = vld(hzt + h), hzj = vld(hzt + h - L::HROW), hxj = vld(hxt + h - L::HROW);
                    const T hzi = hzt[h - 1], hyi = hyt[h - 1];
                    const Vec<T> ox = vld(ext + o), oy = vld(ext + L::OC + o), oz = vld(ext + 2 * L::OC + o);
                    const unsigned ids = vec_ids<T>(idt + o);
                    Vec<T> ex, ey, ez, dHz_j, dHx_j, dHz_i, dHy_i, dHy_k, dHx_k, aE, bE;
                    const int one = vec_coefs(ids, tab, f.aE, f.bE, aE, bE);
#pragma unroll
                    for (int q = 0; q < V; ++q) {
                        const T hz_p = q > 0 ? hz.v[q > 0 ? q - 1 : 0] : hzi, hy_p = q > 0 ? hy.v[q > 0 ? q - 1 : 0] : hyi;
                        dHz_j.v[q] = hz.v[q] - hzj.v[q];
                        dHx_j.v[q] = hx.v[q] - hxj.v[q];
                        dHz_i.v[q] = hz.v[q] - hz_p;
                        dHy_i.v[q] = hy.v[q] - hy_p;
                        dHy_k.v[q] = hy.v[q] - hym[g].v[q];
                        dHx_k.v[q] = hx.v[q] - hxm[g].v[q];
                        ex.v[q] = yee(aE.v[q], ox.v[q], bE.v[q], dHz_j.v[q], cExz[g], dHy_k.v[q], cExy);
                        ey.v[q] = yee(aE.v[q], oy.v[q], bE.v[q], dHx_k.v[q], cEyx, dHz_i.v[q], cEyz.v[q]);
                        ez.v[q] = yee(aE.v[q], oz.v[q], bE.v[q], dHy_i.v[q], cEzy.v[q], dHx_j.v[q], cEzx[g]);
                    }
                    const int j = y0 + g * W::RY + ly;
                    const bool row = j >= 1 && j < d.ny;
                    unsigned wr = act;
                    if (one < 0 || one == CPS_ID_PEC || one == CPS_ID_DISPERSIVE) {
#pragma unroll
                        for (int q = 0; q < V; ++q) {
                            const unsigned id = (ids >> (8 * q)) & 255u;
                            if (id == CPS_ID_PEC) {
                                ex.v[q] = ey.v[q] = ez.v[q] = T(0);
                            } else if (id == CPS_ID_DISPERSIVE) {
                                // left untouched here: the Drude-Lorentz cell pass updates
                                // these cells (ADE, then CPML, the reference order)
                                ex.v[q] = ox.v[q]; ey.v[q] = oy.v[q]; ez.v[q] = oz.v[q];
                                if (PML) bE.v[q] = p.ce_disp;
                                if (DL) wr &= ~(1u << q);
                            }
                        }
                    }
                    const int64_t w = w0 + (int64_t)(g * W::RY) * d.px;
                    if (PML) {
                        if (p.literal) bE = splat(p.cpmlE);
                        pml_vec<T, true>(p, d, tp, b + (u * L::OPL + o) * (int)sizeof(T), L::OC, px, ry[g], fz,
                                         szp + u, bz, cz, bE, i0, row ? j : 0, k, row ? wr : 0u, dHz_i, dHy_i, dHx_j, dHz_j,
                                         dHy_k, dHx_k, ex, ey, ez);
                    }
                    if (edge) {
#pragma unroll
                        for (int q = 0; q < V; ++q)
                            if (!((act >> q) & 1u)) { ex.v[q] = ox.v[q]; ey.v[q] = oy.v[q]; ez.v[q] = oz.v[q]; }
                    }
                    if (row) {
                        // with Drude-Lorentz cells only updated cells are written (theirs
                        // are written beside this tile)
                        const unsigned st = DL ? wr : ALL;
                        field_vst(f.Ex + w, ex, st);
                        field_vst(f.Ey + w, ey, st);
                        field_vst(f.Ez + w, ez, st);
                    }
                }
                hxm[g] = hx;
                hym[g] = hy;
            }
            w0 += d.pxy;
        }
        s = s + 1 == ns ? 0 : s + 1;
        __syncwarp();
        if (lane == 0 && m + ns < nst) issue(m + ns);
    }
    return true;
}

}  // namespace cps
