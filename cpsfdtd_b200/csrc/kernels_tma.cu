// kernels_tma.cu -- one-grid launches of the TMA-fed fused H and E sweeps
// (sm_100a), one 32 x BY x kc tile per block: one-warp tiles (warp_tiles.cuh) for
// FP32 H sweeps and E sweeps without gain, block tiles (tma_bodies.cuh) for FP64
// H sweeps and E sweeps with gain.
#include <cuda.h>
#include <string.h>

#include <algorithm>

#include "pdl.cuh"
#include "warp_tiles.cuh"

namespace cps {

namespace {

// E sweep with gain (block tiles): one block per tile of the launch's boxes,
// every tile on the CPML body (PML) or on the CPML-free one.  In FP32 (gain
// words staged with the fields) one launch runs every tile of a grid with CPML
// on the CPML body (it leaves cells outside the slabs as the CPML-free body
// would, bit for bit): measured faster than CPML and interior tiles as two
// launches at every grid size tried, 128^3 to 384^3, since a second launch's
// partial last wave costs more than the interior blocks gain from the CPML-free
// body's lower register count.  In FP64 (gain words read on the cell list) the
// two launches stay, so its interior blocks are not held to the CPML body's
// registers.
template <typename T, int BY, bool PML, bool DL>
__global__ void __launch_bounds__(32 * BY, 512 / (32 * BY))
    k_e_tma(const __grid_constant__ TmaMaps M, FieldView<T> f, PmlView<T> p, DlView<T> D, GainView<T> G, int kc,
            const __grid_constant__ TileBoxes tb, int *err)
{
    extern __shared__ __align__(128) unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[kStages];
    pdl_go();
    unsigned char *sm = align_smem(sm_raw);
    const TileXYZ t = box_tile(tb, (int)blockIdx.x);
    const int k0 = max(1, t.bz * kc), k1 = min(t.bz * kc + kc, f.d.nz);
    if (k0 >= k1) {
        pdl_wait();
        return;
    }
    init_stages(full);
    pdl_wait();
    uint32_t ctr = 0;
    e_tma_body<T, BY, PML, DL, true>(M, f, p, D, G, kc, t, ctr, err, sm, full);
}

// FP64 H sweep (block tiles): one launch; on a grid with CPML (PML) the body each
// tile needs
template <typename T, int BY, bool PML>
__global__ void __launch_bounds__(32 * BY) k_h_tma(const __grid_constant__ TmaMaps M, FieldView<T> f, PmlView<T> p,
                                                    int kc, const __grid_constant__ TileBoxes tb, int *err)
{
    extern __shared__ __align__(128) unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[kStages];
    pdl_go();
    unsigned char *sm = align_smem(sm_raw);
    const TileXYZ t = box_tile(tb, (int)blockIdx.x);
    const int k0 = t.bz * kc, k1 = min(k0 + kc, f.d.nz);
    if (k0 >= k1) {
        pdl_wait();
        return;
    }
    init_stages(full);
    pdl_wait();
    uint32_t ctr = 0;
    if (PML && tile_in_pml(p.np, f.d, t.bx * 32, t.by * BY, BY, k0, k1, false))
        h_tma_body<T, BY, PML>(M, f, p, kc, t, ctr, err, sm, full);
    else
        h_tma_body<T, BY, false>(M, f, p, kc, t, ctr, err, sm, full);
}

// blocks of one warp that fit an SM's shared memory
template <typename T, int BY>
constexpr int warp_blocks()
{
    return (227 * 1024) / (warp_ring<T, BY>() + 1024 + 640);
}

// One warp per tile; on a grid with CPML (PML) the body each tile needs.
template <typename T, int BY, bool PML>
__global__ void __launch_bounds__(32, warp_blocks<T, BY>())
    k_h_warp(const __grid_constant__ SweepMaps M, FieldView<T> f, PmlView<T> p, int kc, int nbx, int nby, int *err)
{
    extern __shared__ __align__(128) unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[kMaxStages];
    pdl_go();
    const TileXYZ t = grid_tile((int)blockIdx.x, nbx, nby);
    const int k0 = t.bz * kc, k1 = min(k0 + kc, f.d.nz);
    if (k0 >= k1) {
        pdl_wait();
        return;
    }
    __shared__ Coef2<T> tab[kTab];
    if (threadIdx.x < kTab) tab[threadIdx.x] = Coef2<T>{f.aH[threadIdx.x], f.bH[threadIdx.x]};
    init_ring(full);
    pdl_wait();
    Ring R{align_smem(sm_raw), full, warp_ring<T, BY>() - 128, 0u, wait_skew(err), err};
    if (PML && tile_in_pml(p.np, f.d, t.bx * 32, t.by * BY, BY, k0, k1, false))
        h_warp_tile<T, BY, 1, PML>(M, f, p, kc, t, R, tab);
    else
        h_warp_tile<T, BY, kPlanes, false>(M, f, p, kc, t, R, tab);
}

template <typename T, int BY, bool PML, bool DL>
__global__ void __launch_bounds__(32, warp_blocks<T, BY>())
    k_e_warp(const __grid_constant__ SweepMaps M, FieldView<T> f, PmlView<T> p, int kc, int nbx, int nby, int *err)
{
    extern __shared__ __align__(128) unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[kMaxStages];
    pdl_go();
    const TileXYZ t = grid_tile((int)blockIdx.x, nbx, nby);
    const int k0 = max(1, t.bz * kc), k1 = min(t.bz * kc + kc, f.d.nz);
    if (k0 >= k1) {
        pdl_wait();
        return;
    }
    __shared__ Coef2<T> tab[kTab];
    if (threadIdx.x < kTab) tab[threadIdx.x] = Coef2<T>{f.aE[threadIdx.x], f.bE[threadIdx.x]};
    init_ring(full);
    pdl_wait();
    Ring R{align_smem(sm_raw), full, warp_ring<T, BY>() - 128, 0u, wait_skew(err), err};
    if (PML && tile_in_pml(p.np, f.d, t.bx * 32, t.by * BY, BY, k0, k1, true))
        e_warp_tile<T, BY, 1, PML, DL>(M, f, p, kc, t, R, tab);
    else
        e_warp_tile<T, BY, kPlanes, false, DL>(M, f, p, kc, t, R, tab);
}

// The ID-2 cells the TMA E sweep leaves alone, one thread per cell of the
// compacted list.
template <typename T, bool PML>
__global__ void __launch_bounds__(128) k_dl_cells(FieldView<T> f, PmlView<T> p, DlView<T> D)
{
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= D.ncell) return;
    dl_cell_any<T, PML>(f, f, p, D, c);
}

inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

// the shared-memory attribute of each kernel, set once per device (outside
// any capture when tma_attributes runs first)
template <auto K>
bool set_smem(int bytes)
{
    return kernel_smem<K>(bytes);
}

// Interior and CPML tiles of a sweep as tile boxes.  A tile meets a CPML slab
// when its x, y or z range does (tile_in_pml in tma_bodies.cuh, per axis), so
// the interior tiles form one box [a0, a1) per axis and the CPML tiles the
// rest: below and above the interior in z (whole planes of tiles), then in y,
// then in x.
struct SweepTiles {
    TileBoxes interior, pml;
};

inline void add_box(TileBoxes &b, int x0, int x1, int y0, int y1, int z0, int z1)
{
    if (x1 <= x0 || y1 <= y0 || z1 <= z0) return;
    const int k = b.n++;
    b.bx0[k] = x0; b.by0[k] = y0; b.bz0[k] = z0;
    b.nbx[k] = x1 - x0; b.nby[k] = y1 - y0;
    b.start[k + 1] = b.start[k] + (x1 - x0) * (y1 - y0) * (z1 - z0);
}

// every tile of the grid as one box
inline TileBoxes whole_grid(const Dims &d, int by, int kc)
{
    TileBoxes b;
    memset(&b, 0, sizeof(b));
    add_box(b, 0, (int)cdiv(d.nx, 32), 0, (int)cdiv(d.ny, by), 0, (int)cdiv(d.nz, kc));
    return b;
}

inline SweepTiles sweep_tiles(const int np[6], bool pml_on, const Dims &d, int by, int kc, bool eside)
{
    const int tx = (int)cdiv(d.nx, 32), ty = (int)cdiv(d.ny, by), tz = (int)cdiv(d.nz, kc);
    SweepTiles t;
    memset(&t, 0, sizeof(t));
    if (!pml_on) {
        add_box(t.interior, 0, tx, 0, ty, 0, tz);
        return t;
    }
    const int lo = eside ? 0 : 1;
    // per axis: the first and one-past-last tile index that meets no slab
    auto interval = [](int n, auto in_slab, int &a0, int &a1) {
        a0 = 0;
        while (a0 < n && in_slab(a0)) ++a0;
        a1 = a0;
        while (a1 < n && !in_slab(a1)) ++a1;
        for (int q = a1; q < n; ++q)
            if (!in_slab(q)) { a0 = a1 = 0; return; }  // not one interval: every tile takes the CPML body
    };
    int ax0, ax1, ay0, ay1, az0, az1;
    interval(tx, [&](int b) { const int x0 = 32 * b; return x0 <= np[kFX1] - lo || x0 + 31 >= d.nx - np[kFX2]; },
             ax0, ax1);
    interval(ty, [&](int b) { const int y0 = by * b; return y0 <= np[kFY1] - lo || y0 + by - 1 >= d.ny - np[kFY2]; },
             ay0, ay1);
    interval(tz, [&](int b) {
        const int k0 = eside ? std::max(1, b * kc) : b * kc, k1 = std::min(b * kc + kc, d.nz);
        return k0 <= np[kFZ1] - lo || k1 - 1 >= d.nz - np[kFZ2];
    }, az0, az1);
    if (ax1 <= ax0 || ay1 <= ay0 || az1 <= az0) {
        add_box(t.pml, 0, tx, 0, ty, 0, tz);
        return t;
    }
    add_box(t.interior, ax0, ax1, ay0, ay1, az0, az1);
    add_box(t.pml, 0, tx, 0, ty, 0, az0);
    add_box(t.pml, 0, tx, 0, ty, az1, tz);
    add_box(t.pml, 0, tx, 0, ay0, az0, az1);
    add_box(t.pml, 0, tx, ay1, ty, az0, az1);
    add_box(t.pml, 0, ax0, ay0, ay1, az0, az1);
    add_box(t.pml, ax1, tx, ay0, ay1, az0, az1);
    return t;
}

template <typename T, int BY, bool PML, bool DL>
int e_tma_launch(const TmaMaps &M, const FieldView<T> &f, const PmlView<T> &p, const DlView<T> &D,
                 const GainView<T> &G, int kc, const TileBoxes &tb, int *err, cudaStream_t s)
{
    using L = ELayout<T, BY, true>;
    const int blocks = tb.start[tb.n];
    if (blocks <= 0) return 0;
    if (!set_smem<k_e_tma<T, BY, PML, DL>>(L::SMEM)) return 0;
    launch_pdl(!DL, k_e_tma<T, BY, PML, DL>, blocks, dim3(32, BY), L::SMEM, s, M, f, p, D, G, kc, tb, err);
    return 1;
}

template <typename T, int BY, bool PML>
int h_tma_launch(const TmaMaps &M, const FieldView<T> &f, const PmlView<T> &p, int kc, const TileBoxes &tb,
                 int *err, cudaStream_t s)
{
    using L = StageLayout<T, BY>;
    const int blocks = tb.start[tb.n];
    if (blocks <= 0) return 0;
    if (!set_smem<k_h_tma<T, BY, PML>>(L::SMEM)) return 0;
    launch_pdl(true, k_h_tma<T, BY, PML>, blocks, dim3(32, BY), L::SMEM, s, M, f, p, kc, tb, err);
    return 1;
}

template <typename T, int BY, bool PML>
int h_warp_launch(const SweepMaps &M, const FieldView<T> &f, const PmlView<T> &p, int kc, int *err, cudaStream_t s)
{
    kc = (kc + kPlanes - 1) / kPlanes * kPlanes;
    constexpr int smem = warp_ring<T, BY>();
    const int nbx = (int)cdiv(f.d.nx, 32), nby = (int)cdiv(f.d.ny, BY), nbz = (int)cdiv(f.d.nz, kc);
    if (!set_smem<k_h_warp<T, BY, PML>>(smem)) return 0;
    launch_pdl(true, k_h_warp<T, BY, PML>, nbx * nby * nbz, 32, smem, s, M, f, p, kc, nbx, nby, err);
    return 1;
}

template <typename T, int BY, bool PML, bool DL>
int e_warp_launch(const SweepMaps &M, const FieldView<T> &f, const PmlView<T> &p, int kc, int *err, cudaStream_t s)
{
    kc = (kc + kPlanes - 1) / kPlanes * kPlanes;
    constexpr int smem = warp_ring<T, BY>();
    const int nbx = (int)cdiv(f.d.nx, 32), nby = (int)cdiv(f.d.ny, BY), nbz = (int)cdiv(f.d.nz, kc);
    if (!set_smem<k_e_warp<T, BY, PML, DL>>(smem)) return 0;
    launch_pdl(!DL, k_e_warp<T, BY, PML, DL>, nbx * nby * nbz, 32, smem, s, M, f, p, kc, nbx, nby, err);
    return 1;
}

// the kernels the launchers below use
template <typename T, int BY>
void attrs_by()
{
    constexpr int S = warp_ring<T, BY>(), SB = StageLayout<T, BY>::SMEM;
    constexpr int SG = ELayout<T, BY, true>::SMEM;
    if constexpr (sizeof(T) == 4) {
        set_smem<k_h_warp<T, BY, false>>(S);
        set_smem<k_h_warp<T, BY, true>>(S);
    } else {
        set_smem<k_h_tma<T, BY, false>>(SB);
        set_smem<k_h_tma<T, BY, true>>(SB);
    }
    set_smem<k_e_warp<T, BY, false, false>>(S);
    set_smem<k_e_warp<T, BY, false, true>>(S);
    set_smem<k_e_warp<T, BY, true, false>>(S);
    set_smem<k_e_warp<T, BY, true, true>>(S);
    set_smem<k_e_tma<T, BY, false, false>>(SG);
    set_smem<k_e_tma<T, BY, false, true>>(SG);
    set_smem<k_e_tma<T, BY, true, false>>(SG);
    set_smem<k_e_tma<T, BY, true, true>>(SG);
}

template <typename T, int BY>
int e_tma_by(const GridMaps &M, const FieldView<T> &f, const PmlView<T> &p, const DlView<T> &D,
             const GainView<T> &G, int kc, int *err, cudaStream_t s)
{
    const bool dl = D.on && D.ncell > 0, gn = G.on && G.ncell > 0;
    if (gn && sizeof(T) == 4 && p.on) {  // every tile on the CPML body, one launch
        const TileBoxes all = whole_grid(f.d, BY, kc);
        return dl ? e_tma_launch<T, BY, true, true>(M.t, f, p, D, G, kc, all, err, s)
                  : e_tma_launch<T, BY, true, false>(M.t, f, p, D, G, kc, all, err, s);
    }
    if (gn) {  // CPML tiles (if any) and interior tiles as two launches
        const SweepTiles t = sweep_tiles(p.np, p.on, f.d, BY, kc, true);
        return (dl ? e_tma_launch<T, BY, true, true>(M.t, f, p, D, G, kc, t.pml, err, s)
                   : e_tma_launch<T, BY, true, false>(M.t, f, p, D, G, kc, t.pml, err, s)) +
               (dl ? e_tma_launch<T, BY, false, true>(M.t, f, p, D, G, kc, t.interior, err, s)
                   : e_tma_launch<T, BY, false, false>(M.t, f, p, D, G, kc, t.interior, err, s));
    }
    if (p.on)
        return dl ? e_warp_launch<T, BY, true, true>(M.e, f, p, kc, err, s)
                  : e_warp_launch<T, BY, true, false>(M.e, f, p, kc, err, s);
    return dl ? e_warp_launch<T, BY, false, true>(M.e, f, p, kc, err, s)
              : e_warp_launch<T, BY, false, false>(M.e, f, p, kc, err, s);
}

template <typename T, int BY>
int h_tma_by(const GridMaps &M, const FieldView<T> &f, const PmlView<T> &p, int kc, int *err, cudaStream_t s)
{
    if constexpr (sizeof(T) == 8) {
        const TileBoxes all = whole_grid(f.d, BY, kc);
        return p.on ? h_tma_launch<T, BY, true>(M.t, f, p, kc, all, err, s) : h_tma_launch<T, BY, false>(M.t, f, p, kc, all, err, s);
    } else {
        return p.on ? h_warp_launch<T, BY, true>(M.h, f, p, kc, err, s) : h_warp_launch<T, BY, false>(M.h, f, p, kc, err, s);
    }
}

// Planes per tile: as set, or the sweep's default, halved (to two at least)
// while the grid has fewer tiles than 14 per SM (one-warp tiles) or five (block
// tiles of either height).  A tile marches its planes one after the other, so on
// a small grid the sweep takes the time of one tile: at 48^3, H and E sweeps of
// 22 and 14 us with 16 and 8 planes.  The line is measured.  It lies at about
// one wave in FP32 (13 one-warp tiles fit an SM) and at two in FP64 (7 fit); with
// the resident numbers in its place, us a step with CPML: 128^3 FP32 38.9 and
// 45.2, 96^3 FP64 42.0 and 41.4, 112^3 FP64 69.6 and 73.5, 128^3 FP64 89.1 and
// 86.3, other sizes from 36^3 to 176^3 within 1 %.
int planes(int kc, const FusedShape &sh, const Dims &d, bool warp)
{
    const int64_t cols = (int64_t)cdiv(d.nx, 32) * cdiv(d.ny, sh.by), want = (int64_t)sm_count() * (warp ? 14 : 5);
    while (!sh.fixed && kc > 2 && cols * cdiv(d.nz, kc) < want) kc /= 2;
    return kc;
}

}  // namespace

template <typename T>
int launch_h_tma(const GridMaps &M, const FieldView<T> &f, const PmlView<T> &p, FusedShape sh, int *err,
                 cudaStream_t s)
{
    const int kc = planes(sh.kch > 0 ? sh.kch : sh.kc, sh, f.d, sizeof(T) == 4);
    return sh.by == 4 ? h_tma_by<T, 4>(M, f, p, kc, err, s) : h_tma_by<T, 8>(M, f, p, kc, err, s);
}

template <typename T>
int launch_e_tma(const GridMaps &M, const FieldView<T> &f, const PmlView<T> &p, const DlView<T> &D,
                 const GainView<T> &G, FusedShape sh, int *err, cudaStream_t s, const SideLane *lane)
{
    const bool dl = D.on && D.ncell > 0;
    const bool beside = dl && lane && lane->s;
    cudaStream_t ds = s;
    if (beside) {
        cudaEventRecord(lane->fork, s);
        cudaStreamWaitEvent(lane->s, lane->fork, 0);
        ds = lane->s;
    }
    if (dl) {  // launched first, so its blocks start beside the sweep's first wave
        if (p.on) k_dl_cells<T, true><<<cdiv(D.ncell, 128), 128, 0, ds>>>(f, p, D);
        else k_dl_cells<T, false><<<cdiv(D.ncell, 128), 128, 0, ds>>>(f, p, D);
    }
    // an FP32 sweep with gain takes its own plane count
    const bool gn = G.on && G.ncell > 0;
    const int kc = planes(gn && sizeof(T) == 4 && sh.kcg > 0 ? sh.kcg : sh.kc, sh, f.d, !gn);
    const int n = sh.by == 4 ? e_tma_by<T, 4>(M, f, p, D, G, kc, err, s) : e_tma_by<T, 8>(M, f, p, D, G, kc, err, s);
    if (beside) {
        cudaEventRecord(lane->join, lane->s);
        cudaStreamWaitEvent(s, lane->join, 0);
    }
    return n + (dl ? 1 : 0);
}

template <typename T>
void tma_attributes()
{
    attrs_by<T, 4>();
    attrs_by<T, 8>();
}

template void tma_attributes<float>();
template void tma_attributes<double>();
template int launch_h_tma<float>(const GridMaps &, const FieldView<float> &, const PmlView<float> &, FusedShape, int *,
                                  cudaStream_t);
template int launch_h_tma<double>(const GridMaps &, const FieldView<double> &, const PmlView<double> &, FusedShape,
                                   int *, cudaStream_t);
template int launch_e_tma<float>(const GridMaps &, const FieldView<float> &, const PmlView<float> &,
                                  const DlView<float> &, const GainView<float> &, FusedShape, int *, cudaStream_t,
                                  const SideLane *);
template int launch_e_tma<double>(const GridMaps &, const FieldView<double> &, const PmlView<double> &,
                                   const DlView<double> &, const GainView<double> &, FusedShape, int *, cudaStream_t,
                                   const SideLane *);

}  // namespace cps
