// hb_step.cuh -- device side of the handle path: the device mesh, the step
// kernels of both layouts, and the staging and setup kernels.  Shared by
// hb_solver.cu (the forward step) and hb_adjoint.cu (the reverse step).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "hb_common.cuh"
#include "hb_physics.cuh"
#include "hydrob200.h"

namespace hb {

// ---------------------------------------------------------------------------
// device mesh
// ---------------------------------------------------------------------------
enum : uint8_t { META_CODE = 0x0F, META_OWN_FIRST = 0x10, META_HAS_NB = 0x20 };

// Launch shapes.  Edge layout: the flux kernel's threads per CTA and CTAs per
// SM asked of the compiler through __launch_bounds__ (which caps registers
// per thread), and the cell kernel's CTAs per SM (it has UPDATE_THREADS
// threads).  Tile layout: the tile kernel's threads per CTA and CTAs per SM.
enum Layout : int { LAYOUT_EDGE = HB_LAYOUT_EDGE, LAYOUT_TILE = HB_LAYOUT_TILE };
struct LaunchConfig { int layout, threads, min_blocks, update_min_blocks; };
constexpr LaunchConfig LAUNCH_CONFIGS[] = {
    {LAYOUT_EDGE, 128, 7, 8}, {LAYOUT_EDGE, 128, 6, 8}, {LAYOUT_EDGE, 128, 8, 8}, {LAYOUT_EDGE, 256, 3, 6},
    {LAYOUT_EDGE, 256, 4, 8}, {LAYOUT_EDGE, 128, 7, 6}, {LAYOUT_EDGE, 256, 2, 6}, {LAYOUT_EDGE, 64, 12, 8},
    {LAYOUT_TILE, 256, 3, 0}, {LAYOUT_TILE, 256, 2, 0}, {LAYOUT_TILE, 128, 6, 0}, {LAYOUT_TILE, 128, 4, 0},
    {LAYOUT_TILE, 512, 1, 0}, {LAYOUT_TILE, 256, 4, 0},
    {LAYOUT_EDGE, 128, 6, 6}, {LAYOUT_EDGE, 128, 6, 9}, {LAYOUT_EDGE, 128, 7, 9}, {LAYOUT_TILE, 128, 8, 0},
    {LAYOUT_TILE, 256, 5, 0}};
constexpr int N_LAUNCH_CONFIGS = sizeof(LAUNCH_CONFIGS) / sizeof(LAUNCH_CONFIGS[0]);
// Entries keep their places: tile_config numbers name them, and callers keep
// those.  A persistent handle has a kernel of its own and reports entry 0.
constexpr int DEFAULT_EDGE_CONFIG = 2, PERSISTENT_CONFIG = 0;
// Tile layout, fp32 and split: 256 threads, 4 CTAs per SM (64 registers, no
// spills).  us per step against 3 per SM, each with its own balanced tiles:
// split 207,234 cells 9.3 / 9.8, 500,001-cell dam break 21.4 / 23.5, 1,000,000
// cells 43.0 / 49.2, 64 scenarios of 3.8 M cells 147 / 174; fp32 120,000 cells
// 6.9 / 7.3; it loses on about 60,000 cells (5.75 / 5.60).  fp64, whose tile
// kernel spills below 80 registers: 20.2 at 3 per SM, 22.6 at 4 (207,234).
constexpr int DEFAULT_TILE_CONFIG = 13, DEFAULT_TILE_CONFIG_FP64 = 8;
constexpr int UPDATE_THREADS = 128;

// One tile of the tile layout: a compact group of cells, contiguous in the
// device order, with its records (mirror pairs inside the tile, then every
// other real slot of its cells).
struct TileDesc { int scn, cell0, cells, rec0, npairs, nsingles; };

// Constants of one scenario of a batch (the only entry for a single mesh).
struct ScnParams {
    double hm1, hm2, jl, dt;
    int per_day, ndays;        // steps per table interval; intervals in the tables
    int cell0, cells;          // the scenario's cells in the device order
};

// Device mesh.  Cells are in reverse Cuthill-McKee order.  The flux work is a
// list of records: first the interior edges whose two slots both have code 0
// and mirror each other exactly (reciprocal neighbours, negated normal, same
// length), then every other real slot on its own.  The zero-length fourth slot
// of a triangle is no record; the cell update evaluates it.
template <class A>
struct DevMesh {
    using Policy = A;
    using R = typename A::real;
    using L = typename A::level;
    int C;                     // cells
    int per_day;               // steps per table interval (steps_per_day - 1)
    int ndays, nb, nhq;
    int npairs, nrecords;
    double hm1, hm2, jl, dt;
    R *S[2];                   // [C][4] state {H, U, V, Z}, split precision {H, U, V, H_lo};
                               // a step reads S[step & 1], writes the other
    R *W;
    const L *zbc;
    const R *fnc, *dta;        // dta: DT/AREA (variant H) or AREA (variant F)
    const R *sidex;            // variant F CFL length
    const int32_t *bcell;      // [C] row of the boundary tables, -1 = none
    const uint8_t *cmask;      // [C] bit j: slot j is a real slot
    R *slotw;                  // [4C][4] per-slot terms of the cell sums {F0, dWU, dWV, SIDE}
    double *ucoef;             // [C][UPDATE_COEF] update coefficients (update kernels with COEF only)
    // Adjoint forward rollout (fp64; set only on a copy of the mesh whose
    // step launches are captured for it, null otherwise): the cell update of
    // step t also writes the new state into checkpoint (t + 1) / ckpt_every
    // of `ckpt` ([][C][4]) when t + 1 is a multiple of ckpt_every, and, when
    // t + 1 ends on an observation, a gauge cell's new depth into row
    // (t + 1) / obs_every - 1, column gauge_of[cell], of `gauge_out`.
    double *ckpt;
    const int32_t *gauge_of;   // [C] gauge index of the cell, -1 for none
    double *gauge_out;         // [observations][ngauge]
    int ckpt_every, obs_every, ngauge;
    // records [nrecords]
    const int4 *rix;           // {a, b, sa, sb}: cell of the slot, its neighbour (-1 = none),
                               // slot 4*a+j, and for a pair the slot of b (-1 otherwise)
    uint8_t *rmeta;            // code | own_first | has_nb of slot a (code changes on breach)
    const R *rgeo;             // [nrecords][4] {COSF, SINF, SIDE, x} of slot a; x: fp64 pack_slots, else 0
    const R *sgeo;             // [real slots][4] {COSF, SINF, SIDE, SlotRef::pack} (cell_kernel; else null)
    const int4 *cseg;          // cell_kernel CTAs {first cell, cells, first slot record, slot records}
    R *flux;                   // [4C][4] FLUX0..3 of the last step, index 4*cell + j
    const R *bqt, *bdqt;       // [ndays*nb]
    const L *bzt, *bdzt;       // [ndays*nb]
    const L *btop;             // [nb]
    const int32_t *bnhq1;      // [nb]
    const L *bzw;              // [nb*nhq]; one extra zero row at index nb
    const R *bqw;              // [nb*nhq]; one extra zero row at index nb
    uint32_t *err;
    long long *step_ctr;
    unsigned *tick;            // cell_kernel: CTAs of a sequence's last step that are done (0 between sequences)
    // batches: per-CTA segment tables, one scenario per CTA
    int nscen;
    const ScnParams *scn;      // [nscen]
    const int4 *fseg;          // flux CTAs {scenario, first record, records, 1 = mirror pairs}
    const int4 *useg;          // update CTAs {scenario, first cell, cells, 0}
    // edge layout, single mesh: the flux kernel takes its CTAs' record ranges
    // in reverse order (rev_flux), so the single records at the end of the
    // list (boundary slots, whose fixed-point iterations make them the slowest)
    // start first instead of forming the launch's tail.  The cell kernel takes
    // its ranges in the opposite order of the flux kernel (batches: reversed
    // when rev_update), so it starts on the slot terms the flux kernel wrote
    // last, which are still in L2 when the mesh's terms exceed it
    int rev_flux, rev_update;
    // tile layout
    const TileDesc *tiles;     // [ntiles]
    int ntiles, max_tile_cells, max_tile_queue;   // the largest tile's cells and queue entries (2 per pair)
};

// One step: the state buffer it reads, its number, and its scenario's table
// intervals.
struct StepIndex { int par, per_day, ndays; long long step; };

// EARLY: read ahead of the dependency wait, so from L2 (a line that an earlier
// launch left in L1 may be old).
template <bool EARLY = false, class A>
__device__ __forceinline__ StepIndex step_index(const DevMesh<A> &m, int k, int per_day, int ndays) {
    const long long step = (EARLY ? __ldcg(m.step_ctr) : *m.step_ctr) + k;
    if (threadIdx.x == 0 && step >= (long long)per_day * ndays) atomicOr(m.err, ERRBIT_TABLE_RANGE);
    return {(int)(step & 1), per_day, ndays, step};
}

// The step's day and step within it, for the slots that read boundary tables:
// the division (by a value known at run time) is left to them, since it costs
// about as much as a fifth of a cell's whole update.  Beyond the tables (which
// step_index reports) the last interval, so that they are never read past.
__device__ __forceinline__ StepParams with_time(StepParams p, const StepIndex &si) {
    int day, in_day;
    if (si.step <= 0xFFFFFFFFll) {
        const unsigned s = (unsigned)si.step, q = s / (unsigned)si.per_day;
        day = (int)q;
        in_day = (int)(s - q * (unsigned)si.per_day);
    } else {
        day = (int)(si.step / si.per_day);
        in_day = (int)(si.step % si.per_day);
    }
    p.jt = day >= si.ndays ? si.ndays - 1 : day;
    p.kt = 1 + in_day;
    return p;
}

template <class R> struct Vec4 { R x, y, z, w; };
__device__ __forceinline__ Vec4<double> ld4(const double *p) {
    const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
    return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ Vec4<float> ld4(const float *p) {
    const float4 a = *reinterpret_cast<const float4 *>(p);
    return {a.x, a.y, a.z, a.w};
}
__device__ __forceinline__ void st4(double *p, double x, double y, double z, double w) {
    *reinterpret_cast<double2 *>(p) = make_double2(x, y);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(z, w);
}
__device__ __forceinline__ void st4(float *p, float x, float y, float z, float w) {
    *reinterpret_cast<float4 *>(p) = make_float4(x, y, z, w);
}

// The same for memory known to be global, 32-byte aligned: one 256-bit access
// for fp64 records on sm_100 (half the instructions of two 16-byte ones).
// Ordered like any other access (volatile, memory clobber), so they stay
// after a dependency wait.
__device__ __forceinline__ Vec4<double> ldg4(const double *p) {
    Vec4<double> v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ Vec4<float> ldg4(const float *p) { return ld4(p); }
__device__ __forceinline__ void stg4(double *p, double x, double y, double z, double w) {
    st_global_f64x4(p, x, y, z, w);
}
__device__ __forceinline__ void stg4(float *p, float x, float y, float z, float w) { st4(p, x, y, z, w); }

template <class A>
__device__ __forceinline__ CellStateA<A> load_cell(const DevMesh<A> &m, int par, int c) {
    const Vec4<typename A::real> v = ldg4(m.S[par] + 4 * (size_t)c);
    const typename A::level zbc = m.zbc[c];
    if constexpr (is_split<A>::value) return {v.x, v.y, v.z, split_level<A>(v.x, v.w, zbc), zbc};
    else return {v.x, v.y, v.z, v.w, zbc};
}

// Where a step keeps the slots' terms of the cell sums between the flux and
// the update: slot s at p + 4 * (s - slot0).  Global memory (m.slotw, slot0 =
// 0) between the two kernels of the edge layout; shared memory (slot0 = the
// tile's first slot) inside the tile kernel (SMEM).
template <class R, bool SMEM = false>
struct Terms {
    R *p;
    int slot0;
    static constexpr bool smem = SMEM;
};

// the slot's terms of the cell sums (functors.cu:733-741): F0 and SIDE for
// WH = fma(SIDE, F0, WH), and the complete WU / WV increments
template <class A, class T>
__device__ __forceinline__ void store_terms(const T &t, int s, const typename A::real f[4],
                                            typename A::real side, typename A::real cs, typename A::real sn) {
    using R = typename A::real;
    const R fr1 = A::add(f[1], f[3]);
    const R slcos = A::mul(side, cs), slsin = A::mul(side, sn);
    const R dwu = A::dot(slcos, fr1, -slsin, f[2], M_WU);
    const R dwv = A::dot(slsin, fr1, slcos, f[2], M_WV);
    if constexpr (T::smem) st4(t.p + 4 * (size_t)(s - t.slot0), f[0], dwu, dwv, side);
    else stg4(t.p + 4 * (size_t)(s - t.slot0), f[0], dwu, dwv, side);
}

// One record per slot: in four arrays, as the reference has them, a pair's two
// slots were eight scattered stores of eight bytes.  A single step, which
// leaves its fluxes: 207,234 cells 29.7 -> 24.7 us, 2,000,000 335 -> 195 us.
template <class A>
__device__ __forceinline__ void store_flux(const DevMesh<A> &m, int s, const typename A::real f[4]) {
    stg4(m.flux + 4 * (size_t)s, f[0], f[1], f[2], f[3]);
}

// One slot on its own: flux_slot with its boundary tables (functors.cu:47-202).
// single_core takes the slot's cell a (device order, for its table row), its
// slot sa, both cells' states and the record's code byte and geometry; for a
// boundary code p has the step's time (with_time).
template <class A, int VARIANT, class T>
__device__ __forceinline__ void single_core(const DevMesh<A> &m, int r, int a, int sa, const CellStateA<A> &own,
                                            const CellStateA<A> &nb, uint8_t meta, const Vec4<typename A::real> &g,
                                            const StepParams &p, int write_flux, const T &tout) {
    using R = typename A::real;
    using L = typename A::level;
    SlotInA<A> in;
    in.own = own;
    in.code = (int8_t)(meta & META_CODE);
    in.own_first = meta & META_OWN_FIRST;
    in.has_nb = meta & META_HAS_NB;
    in.nb = nb;
    in.cosj = g.x; in.sinj = g.y; in.side = g.z;
    auto fetch = [&]() {
        BoundaryInA<A> bi;
        const int row = m.bcell[a];
        if (row >= 0) {
            const size_t q = (size_t)p.jt * m.nb + row;
            bi.qt = m.bqt[q]; bi.dqt = m.bdqt[q]; bi.zt = m.bzt[q]; bi.dzt = m.bdzt[q];
            bi.top = m.btop[row]; bi.nhq1 = m.bnhq1[row];
            bi.zw = m.bzw + (size_t)row * m.nhq; bi.qw = m.bqw + (size_t)row * m.nhq;
        } else {
            bi.qt = bi.dqt = R(0); bi.zt = bi.dzt = bi.top = L(0); bi.nhq1 = 0;
            bi.zw = m.bzw + (size_t)m.nb * m.nhq; bi.qw = m.bqw + (size_t)m.nb * m.nhq;
        }
        bi.nhq = m.nhq;
        return bi;
    };
    SlotOut<R> o;
    flux_slot<A, VARIANT>(in, p, fetch, o);
    // A code that leaves fluxes unwritten keeps the old values (functors.cu:525-565),
    // so it stores all four at every step, also where a supercritical one wrote them.
    if (o.mask != 0xF) {
        const Vec4<R> old = ldg4(m.flux + 4 * (size_t)sa);
        if (!(o.mask & 1)) o.f[0] = old.x;
        if (!(o.mask & 2)) o.f[1] = old.y;
        if (!(o.mask & 4)) o.f[2] = old.z;
        if (!(o.mask & 8)) o.f[3] = old.w;
    }
    if (write_flux || in.code == CODE_BOUNDA_OTHER) store_flux(m, sa, o.f);
    store_terms<A>(tout, sa, o.f, in.side, in.cosj, in.sinj);
    if (o.klas_to_zero) m.rmeta[r] = (uint8_t)((meta & ~META_CODE) | CODE_ZERO);
    if (o.undefined) atomicOr(m.err, ERRBIT_UNDEFINED);
}

// A record's geometry, cells and slots.  fp64 records are one 256-bit load:
// the fourth value of rgeo holds both slots (pack_slots: 4a + j in the low
// word, 4b + j in the high one; a single's neighbour without a slot of its own
// as 4b, none as all ones), and rix is not read by the step.
__host__ __device__ inline unsigned long long pack_slots(int sa, int b, int sb) {
    return (unsigned long long)(unsigned)(sb >= 0 ? sb : b < 0 ? -1 : 4 * b) << 32 | (unsigned)sa;
}
template <class A>
struct Record {
    Vec4<typename A::real> g;
    int a, b, sa, sb;
};
template <class A>
__device__ __forceinline__ Record<A> load_record(const DevMesh<A> &m, int r) {
    Record<A> q;
    q.g = ldg4(m.rgeo + 4 * (size_t)r);
    if constexpr (std::is_same<typename A::real, double>::value) {
        const unsigned long long w = (unsigned long long)__double_as_longlong(q.g.w);
        q.sa = (int)(unsigned)w;
        q.sb = (int)(unsigned)(w >> 32);
        q.a = q.sa >> 2;
        q.b = q.sb >> 2;
    } else {
        const int4 ix = m.rix[r];
        q.a = ix.x; q.b = ix.y; q.sa = ix.z; q.sb = ix.w;
    }
    return q;
}

// One side of record r on its own: a single record's slot, or slot a
// (item = 2r) or b (item = 2r + 1) of a pair, computed as the reference
// computes every slot.  of_pair: the record is known to be a pair.
template <class A, int VARIANT, class T>
__device__ __forceinline__ void side_record(const DevMesh<A> &m, int item, bool of_pair, const StepIndex &si,
                                            const StepParams &p, int write_flux, const T &tout) {
    using R = typename A::real;
    using L = typename A::level;
    const int r = item >> 1;
    const bool other = item & 1;
    const Record<A> q = load_record(m, r);
    Vec4<R> g = q.g;
    uint8_t meta = of_pair ? (uint8_t)(CODE_ZERO | META_OWN_FIRST | META_HAS_NB) : m.rmeta[r];
    int c = q.a, n = q.b, s = q.sa;
    if (other) {   // negated normal, not the lower-numbered side
        c = q.b; n = q.a; s = q.sb;
        g.x = -g.x; g.y = -g.y;
        meta &= (uint8_t)~META_OWN_FIRST;
    }
    const CellStateA<A> own = load_cell(m, si.par, c);
    const CellStateA<A> nb =
        (meta & META_HAS_NB) ? load_cell(m, si.par, n) : CellStateA<A>{R(0), R(0), R(0), L(0), L(0)};
    const bool timed = code_is_bounda((int8_t)(meta & META_CODE));
    single_core<A, VARIANT>(m, r, c, s, own, nb, meta, g, timed ? with_time(p, si) : p, write_flux, tout);
}

// One side of a pair on its own (item as above), without the boundary codes.
template <class A, int VARIANT, class T>
__device__ __forceinline__ void pair_side(const DevMesh<A> &m, int item, const StepIndex &si,
                                          const StepParams &p, int write_flux, const T &tout) {
    const bool other = item & 1;
    const Record<A> q = load_record(m, item >> 1);
    SlotInA<A> in;
    in.own = load_cell(m, si.par, other ? q.b : q.a);
    in.nb = load_cell(m, si.par, other ? q.a : q.b);
    in.has_nb = true; in.own_first = !other; in.code = CODE_ZERO;
    in.cosj = other ? -q.g.x : q.g.x; in.sinj = other ? -q.g.y : q.g.y; in.side = q.g.z;
    const int s = other ? q.sb : q.sa;
    SlotOut<typename A::real> o;
    flux_slot<A, VARIANT>(in, p, []() { return BoundaryInA<A>{}; }, o);
    if (write_flux) store_flux(m, s, o.f);
    store_terms<A>(tout, s, o.f, in.side, in.cosj, in.sinj);
}

// The sides that a CTA computes after its main pass (side_record's items): entry i
// of the front has its partner, or -1, in entry i of the back.  The two sides of
// an edge take different branches of the chain (the lower one the inflow, the
// higher one the weir's power) or different Osher routes, so they are kept apart
// and a warp runs one of them: the thin sheet's flux kernel 16.2 -> 11.2 M warp
// instructions.
struct SideQueue {
    int *e;
    int cap;    // entries; a pair takes two, and so does a single
    int *n;     // entries in the front, shared by the CTA
    __device__ __forceinline__ void push(int front, int back) const {
        const int i = atomicAdd(n, 1);
        e[i] = front;
        e[cap - 1 - i] = back;
    }
    __device__ __forceinline__ int item(int j, int count) const { return j < count ? e[j] : e[cap - 1 - (j - count)]; }
};

// One mirror-pair record: both sides' fluxes where both cells are deep and
// Osher takes one piece (osher_one_piece: subcritical flow across the edge, or
// supercritical either way), or both are dry: the bulk of any mesh.  The two
// routes (functors.cu:151-200) have the same cells, normal and inputs except two
// rotations that the reference build rounds differently (policies with
// route_modes), so they share the square roots, the depth ratio and their
// quotients, and each runs osher_one_piece from its own FIR.  Every other pair
// puts its two sides into the CTA's queue, which runs after the main pass.  So
// the main pass holds neither the powers of the one-sided branches nor Osher's
// other pieces.
//
// Bound by the gathers' latency and by issue.  207,234 cells, flux kernel, warp
// instructions per launch: both branch chains, Osher in full and a queue of
// mirrored evaluations 7.5 M; this form 3.6 M, of which the supercritical pieces
// are 0.2 M.  Step, still / supercritical / patchy wet and dry / thin sheet
// (all cells between HM1 and HM2) flow, us: that whole form 25.4 / 27.0 / 33.3 /
// 28.5; subcritical alone in the main pass, the two sides of an edge next to
// each other in one queue of general slots 15.6 / 28.5 / 26.3 / 33.6; this form
// 15.6 / 20.0 / 25.6 / 28.0.  Taken back: pairs instead of sides in the queue
// (15.4 / 28.4 / 28.6 / 29.9: half of the threads idle where half of the pairs
// are queued) and the chain of thin pairs in the main pass (16.5 / 21.1 / 29.9 /
// 27.5).
template <class A, class T>
__device__ __forceinline__ void pair_record(const DevMesh<A> &m, int r, const Record<A> &q, const StepIndex &si,
                                            const StepParams &p, int write_flux, const T &tout,
                                            const SideQueue &queue) {
    using R = typename A::real;
    using L = typename A::level;
    const CellStateA<A> a = load_cell(m, si.par, q.a), b = load_cell(m, si.par, q.b);
    const R cs = q.g.x, sn = q.g.y, side = q.g.z;
    const R qr0 = A::depth(b.z, a.zbc);
    bool low = true;   // a's side goes to the queue's front
    if (edge_deep<A>(a, b, qr0, p)) {
        const R cl = A::sqrt(A::mul(A::c(9.81), a.h)), cr = A::sqrt(A::mul(A::c(9.81), qr0));
        const R ratio = A::fmin(A::div(b.h, qr0), A::c(1.5));
        const R ql1 = A::dot(a.u, cs, a.v, sn, M_QL1), ql2 = A::dot(a.v, cs, -a.u, sn, M_QL2);
        const R qr2 = A::dot(b.v, cs, -b.u, sn, M_QR2);
        const R fil = A::add(ql1, A::mul(A::c(2.0), cl));
        const R ur = A::dot(b.u, cs, b.v, sn, M_UR);
        R fa[4], fb[4];
        R ql[3] = {a.h, ql1, ql2}, qr[3] = {qr0, A::mul(ur, ratio), qr2};
        bool ok = osher_one_piece<A>(cl, cr, ql, qr, fil, fa);
        R urm = ur;
        if constexpr (A::route_modes) {
            urm = A::dot(b.u, cs, b.v, sn, M_UR1);
            ql[2] = A::dot(a.v, cs, -a.u, sn, M_QL2M);
            qr[1] = A::mul(urm, ratio);
            ok &= osher_one_piece<A>(cl, cr, ql, qr, fil, fb);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) fb[i] = fa[i];
        }
        if (ok) {
            fa[1] = osher_f1<A>(fa[1], ratio, b.h, ur);
            if (write_flux) store_flux(m, q.sa, fa);
            store_terms<A>(tout, q.sa, fa, side, cs, sn);
            fb[0] = -fb[0];
            fb[1] = osher_f1<A>(fb[1], ratio, b.h, urm);
            // mirror_f3
            const L za = A::ladd(A::lvl(A::sqrt(A::divk_raw(fb[3], 4.905))), a.zbc);
            const R hc3 = za > b.zbc ? A::depth(za, b.zbc) : R(0);
            fb[3] = A::mul(A::mul(A::c(4.905), hc3), hc3);
            if (write_flux) store_flux(m, q.sb, fb);
            store_terms<A>(tout, q.sb, fb, side, -cs, -sn);
            return;
        }
    } else if (a.h <= A::c(p.hm1) && b.h <= A::c(p.hm1)) {   // both dry (functors.cu:98-105)
        const R f[4] = {R(0), R(0), R(0), R(0)};
        if (write_flux) { store_flux(m, q.sa, f); store_flux(m, q.sb, f); }
        store_terms<A>(tout, q.sa, f, side, cs, sn);
        store_terms<A>(tout, q.sb, f, side, -cs, -sn);
        return;
    } else {
        low = a.z < b.z;
    }
    queue.push(low ? 2 * r : 2 * r + 1, low ? 2 * r + 1 : 2 * r);
}

// Flux of every record of one step.  Single mesh (SEG = false): records
// [0, npairs) are mirror pairs and the rest single slots, one per thread.
// Batch (SEG = true): CTA b takes the scenario and record range of fseg[b].
// Singles go through the queue as well, so that the main pass holds the common
// case alone.
template <class A, int VARIANT, int THREADS, int MINB, bool SEG>
__global__ void __launch_bounds__(THREADS, MINB) flux_kernel(DevMesh<A> m, int k, int write_flux) {
    __shared__ int entries[2 * THREADS];
    __shared__ int qn;
    const SideQueue queue{entries, 2 * THREADS, &qn};
    if (threadIdx.x == 0) qn = 0;
    int r;
    bool valid, pair;
    StepIndex si;
    StepParams p;
    Record<A> q{};
    // constant tables: read before the dependency wait
    if constexpr (SEG) {
        const int4 d = m.fseg[blockIdx.x];
        const ScnParams sp = m.scn[d.x];
        r = d.y + (int)threadIdx.x;
        valid = (int)threadIdx.x < d.z;
        pair = d.w != 0;
        if (valid && pair) q = load_record(m, r);
        cudaGridDependencySynchronize();
        cudaTriggerProgrammaticLaunchCompletion();
        si = step_index(m, k, sp.per_day, sp.ndays);
        p = StepParams{sp.hm1, sp.hm2, sp.jl, sp.dt, 1, 0};
    } else {
        r = (m.rev_flux ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x) * THREADS + threadIdx.x;
        valid = r < m.nrecords;
        pair = r < m.npairs;
        if (pair) q = load_record(m, r);
        cudaGridDependencySynchronize();
        cudaTriggerProgrammaticLaunchCompletion();
        si = step_index(m, k, m.per_day, m.ndays);
        p = StepParams{m.hm1, m.hm2, m.jl, m.dt, 1, 0};
    }
    __syncthreads();
    const Terms<typename A::real> tout{m.slotw, 0};
    if (valid) {
        if (pair) pair_record<A>(m, r, q, si, p, write_flux, tout, queue);
        else queue.push(2 * r, -1);
    }
    __syncthreads();
    const int nq = qn;
    for (int j = threadIdx.x; j < 2 * nq; j += THREADS) {
        const int e = queue.item(j, nq);
        if (SEG ? pair : e >= 0 && (e >> 1) < m.npairs) pair_side<A, VARIANT>(m, e, si, p, write_flux, tout);
        else if (e >= 0) side_record<A, VARIANT>(m, e, false, si, p, write_flux, tout);
    }
}

// The fluxes of a cell's zero-length slot: the cell's state, no neighbour, zero
// geometry, code 0.  The two-kernel step calls it out of line: it is rarely
// needed, and its powers would take the cell kernel's registers.
template <class R> struct ZeroSlot { R f[4]; };
template <class A, int VARIANT>
__device__ __forceinline__ ZeroSlot<typename A::real> zero_slot(const CellStateA<A> &st, const StepParams &p,
                                                                int write_flux) {
    using R = typename A::real;
    using L = typename A::level;
    ZeroSlot<R> z;
    if (write_flux && closed_common<A>(st, R(0), R(0), p, z.f)) return z;
    SlotInA<A> in;
    in.own = st;
    in.nb = {R(0), R(0), R(0), L(0), L(0)};
    in.has_nb = false; in.own_first = false; in.code = CODE_ZERO;
    in.cosj = R(0); in.sinj = R(0); in.side = R(0);
    auto nofetch = []() { return BoundaryInA<A>{}; };
    SlotOut<R> o;
    if (write_flux) flux_slot<A, VARIANT, decltype(nofetch), false>(in, p, nofetch, o);
    else flux_chain<A, VARIANT, decltype(nofetch), true>(in, p, nofetch, o);
    return {{o.f[0], o.f[1], o.f[2], o.f[3]}};
}
// the fluxes of cell c's slots that are no real ones
template <class A>
__device__ __forceinline__ void store_zero(const DevMesh<A> &m, int c, unsigned mask,
                                           const ZeroSlot<typename A::real> &o) {
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(mask & (1u << j))) store_flux(m, 4 * c + j, o.f);
}
template <class A, int VARIANT>
__device__ __noinline__ ZeroSlot<typename A::real> zero_slot_call(const CellStateA<A> st, const StepParams p,
                                                                  int write_flux) {
    return zero_slot<A, VARIANT>(st, p, write_flux);
}

// Sums and update of one cell (UpdateCellKernel, functors.cu:717-784).  The
// zero-length fourth slot of a triangle is evaluated here, without pow
// (flux_slot's ZERO_LEN) unless fluxes are written out, and only where its
// zero addends can change the sums.
// TERMS: where `terms` is and when it is read.
// update_core takes the cell's state and constants `in`, and two functions
// that give its DT/AREA and its friction: a caller that formed them while it
// waited for the terms returns them, others compute them where they are used.
enum : int {
    TERMS_GLOBAL = 0,      // edge layout: global memory, all read up front
    TERMS_SMEM = 1,        // tile layout: shared memory, all read up front
    TERMS_SMEM_LATE = 2    // cell_kernel: shared memory, each read where it is added (24 registers fewer);
                           // the zero-length slots' fluxes are written by the caller
};
template <class A>
struct CellIn {
    Vec4<typename A::real> raw;         // the stored state record
    typename A::level zbc;
    unsigned mask;
    typename A::real fnc, dta, sidex;   // dta: DT/AREA (variant H) or AREA (variant F)
};
// EARLY: ahead of the dependency wait; ZBC and FNC, which the adjoint's
// parameters change between sequences, then come from L2.
template <class A, int VARIANT, bool EARLY = false>
__device__ __forceinline__ CellIn<A> load_cell_constants(const DevMesh<A> &m, int c) {
    using R = typename A::real;
    CellIn<A> in;
    in.zbc = EARLY ? __ldcg(m.zbc + c) : m.zbc[c];
    in.mask = m.cmask[c];
    in.fnc = EARLY ? __ldcg(m.fnc + c) : m.fnc[c];
    in.dta = m.dta[c];
    in.sidex = VARIANT == 1 ? m.sidex[c] : R(0);
    return in;
}

template <class A, int VARIANT, bool COEF, int TERMS, class DtaOf, class FrictionOf>
__device__ __forceinline__ void update_core(const DevMesh<A> &m, int c, const CellIn<A> &cin, const StepIndex &si,
                                            const StepParams &p, int write_flux, const typename A::real *terms,
                                            const DtaOf &dta_of, const FrictionOf &friction_of) {
    using R = typename A::real;
    using L = typename A::level;
    constexpr bool SMEM_TERMS = TERMS != TERMS_GLOBAL;
    const Vec4<R> raw = cin.raw;
    const unsigned mask = cin.mask;
    CellStateA<A> st;
    st.h = raw.x; st.u = raw.y; st.v = raw.z; st.zbc = cin.zbc;
    if constexpr (is_split<A>::value) st.z = split_level<A>(raw.x, raw.w, st.zbc);
    else st.z = raw.w;
    // A triangle's zero-length fourth slot is evaluated below and has no terms,
    // so they are not read.  Any other slot's place is read without asking
    // whether it is a real one (only a real slot's terms are used).
    auto terms_of = [&](int j) { return SMEM_TERMS ? ld4(terms + 4 * j) : ldg4(terms + 4 * j); };
    Vec4<R> t[4];
    if constexpr (TERMS != TERMS_SMEM_LATE) {
#pragma unroll
        for (int j = 0; j < 3; j++) t[j] = terms_of(j);
        if (mask & 8u) t[3] = terms_of(3);
    }
    // The slot sums in slot order j = 0..3.  A zero-length slot (a
    // triangle's fourth) adds SIDE*F0 = 0*F0 to WH and 0*(...) to WU and WV.
    // For a finite state (h > 0) its fluxes are finite, so each addend is a
    // zero and leaves a non-zero partial sum unchanged bit for bit: the first
    // pass skips such slots.  Only a zero partial sum at a zero-length slot
    // (whose sign the addend may change) or a non-finite state needs the slot's
    // flux: the second pass then evaluates it once (every zero-length slot of
    // a cell has the same inputs: the cell's state, no neighbour, zero
    // geometry and code 0) and redoes the sums with every slot in order.
    // Keeping that evaluation off the common path keeps the kernel's
    // register count that of the sums and the update.
    R wh = R(0), wu = R(0), wv = R(0);
    const bool finite_state = st.h > R(0) && isfinite((double)st.h) && isfinite((double)st.u) &&
                              isfinite((double)st.v) && isfinite((double)st.z) && isfinite((double)st.zbc);
    bool need_zero = false;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (mask & (1u << j)) {
            if constexpr (TERMS == TERMS_SMEM_LATE) t[j] = terms_of(j);
            // F0 and SIDE for WH; the WU/WV increments were formed by the flux kernel
            wh = A::madd(t[j].w, t[j].x, wh, M_WH);
            wu = A::add(wu, t[j].y);
            wv = A::add(wv, t[j].z);
        } else if (!finite_state || wh == R(0) || wu == R(0) || wv == R(0)) {
            need_zero = true;
        }
    }
    // The last step of a sequence leaves such slots' fluxes too.  One evaluation
    // serves both needs, and the sums are redone only where they need it: single
    // steps at 207,234 cells 24.7 -> 22.1 us, at 60,000 14.0 -> 12.5 us.
    const bool leave = TERMS != TERMS_SMEM_LATE && write_flux && (mask & 15u) != 15u;
    if (need_zero || leave) {
        const ZeroSlot<R> o =
            SMEM_TERMS ? zero_slot<A, VARIANT>(st, p, leave) : zero_slot_call<A, VARIANT>(st, p, leave);
        if (leave) store_zero(m, c, mask, o);
        if (need_zero) {
            wh = R(0); wu = R(0); wv = R(0);
#pragma unroll 1
            for (int j = 0; j < 4; j++) {
                if (mask & (1u << j)) {
                    const Vec4<R> tj = terms_of(j);
                    wh = A::madd(tj.w, tj.x, wh, M_WH);
                    wu = A::add(wu, tj.y);
                    wv = A::add(wv, tj.z);
                } else {
                    // zero-length slot: SIDE = SLCOS = SLSIN = 0 (mesh.cpp:293-306, :347-370)
                    wsum_add<A>(wh, wu, wv, o.f[0], o.f[1], o.f[2], o.f[3], R(0), R(0), R(0));
                }
            }
        }
    }
    CellUpdateIn<R, L> ci;
    ci.h = st.h; ci.u = st.u; ci.v = st.v; ci.zbc = st.zbc;
    ci.hlo = is_split<A>::value ? raw.w : R(0);
    ci.fnc = cin.fnc;
    CellUpdateOut<R, L> o = update_cell<A, VARIANT, COEF>(ci, dta_of(), wh, wu, wv, p, friction_of,
                                                          COEF ? m.ucoef + UPDATE_COEF * (size_t)c : nullptr);
    const int np = si.par ^ 1;
    if constexpr (is_split<A>::value) stg4(m.S[np] + 4 * (size_t)c, o.h, o.u, o.v, o.hlo);
    else stg4(m.S[np] + 4 * (size_t)c, o.h, o.u, o.v, o.z);
    // W enters no step: only the last one of a sequence leaves it
    if (write_flux) m.W[c] = speed<A>(o.u, o.v);
    // (U and V are always finite: each is the smaller of its size and a bound)
    if (!isfinite((double)o.h)) atomicOr(m.err, ERRBIT_NONFINITE);
    if constexpr (std::is_same<A, F64Exact>::value) {
        if (m.ckpt != nullptr) {
            const long long t1 = si.step + 1;
            if (t1 % m.ckpt_every == 0)
                stg4(m.ckpt + 4 * ((size_t)(t1 / m.ckpt_every) * (size_t)m.C + (size_t)c), o.h, o.u, o.v, o.z);
        }
        if (m.gauge_of != nullptr) {
            const long long t1 = si.step + 1;
            const int g = m.gauge_of[c];
            if (g >= 0 && t1 % m.obs_every == 0) m.gauge_out[(size_t)(t1 / m.obs_every - 1) * m.ngauge + g] = o.h;
        }
    }
}

// The update of cell c from its constants `in` (load_cell_constants).
template <class A, int VARIANT, bool COEF = false, int TERMS = TERMS_GLOBAL>
__device__ __forceinline__ void update_one(const DevMesh<A> &m, int c, CellIn<A> in, const StepIndex &si,
                                           const StepParams &p, int write_flux, const typename A::real *terms) {
    in.raw = ldg4(m.S[si.par] + 4 * (size_t)c);
    update_core<A, VARIANT, COEF, TERMS>(
        m, c, in, si, p, write_flux, terms,
        [&]() { return cell_dta<A, VARIANT>(in.raw.x, in.raw.y, in.dta, in.sidex, p); },
        [&]() { return cell_friction<A>(in.raw.x, in.raw.y, in.raw.z, in.fnc, p); });
}

// Every cell of one step, one per thread.  Batch: CTA b takes the scenario and
// cell range of useg[b].  COEF: also the update coefficients of the wet cells
// into m.ucoef.
//
// Bound by issue (3.1 M warp instructions at 207,234 cells, half of them fp64
// chains: a power, a square root and three quotients per cell) and by the tail:
// 1,620 CTAs are 1.37 waves of 8 per SM.  The constants' early loads: 14.5 ->
// 14.1 us per step.  Shapes (flux, cell CTAs per SM), 207,234-cell channel /
// mixed mesh / dam break / 2,000,000-cell dam break: (8, 8) 13.6 / 15.9 / 17.1 /
// 141.8 us, (7, 6) 13.9 / 15.9 / 17.5 / 141.9, (7, 8) 13.7 / 15.9 / 16.6 / 143.4.
template <class A, int VARIANT, int UMINB, bool SEG, bool COEF = false>
__global__ void __launch_bounds__(UPDATE_THREADS, UMINB) update_kernel(DevMesh<A> m, int k, int write_flux) {
    // batches: the flux segments run forward, so the cells run reversed
    const bool rev = SEG ? m.rev_update != 0 : m.rev_flux == 0;
    const int blk = rev ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
    int c, per_day, ndays;
    bool on;
    StepParams p;
    if constexpr (SEG) {
        const int4 d = m.useg[blk];
        const ScnParams sp = m.scn[d.x];
        c = d.y + (int)threadIdx.x;
        on = (int)threadIdx.x < d.z;
        per_day = sp.per_day; ndays = sp.ndays;
        p = StepParams{sp.hm1, sp.hm2, sp.jl, sp.dt, 1, 0};
    } else {
        c = blk * UPDATE_THREADS + (int)threadIdx.x;
        on = c < m.C;
        per_day = m.per_day; ndays = m.ndays;
        p = StepParams{m.hm1, m.hm2, m.jl, m.dt, 1, 0};
    }
    CellIn<A> in{};
    if (on) in = load_cell_constants<A, VARIANT, true>(m, c);
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const StepIndex si = step_index(m, k, per_day, ndays);
    if (on) update_one<A, VARIANT, COEF>(m, c, in, si, p, write_flux, m.slotw + 16 * (size_t)c);
}

// What a slot of cell_kernel needs besides its geometry, packed into the
// fourth value of its sgeo record: the neighbour (device order), the slot's
// place in its CTA, its code byte at creation, and its record, whose rmeta
// holds the current code of a slot that may breach.
struct SlotRef {
    static constexpr int NO_NB = 0xFFFFFF, MAX_RECORD = 1 << 24;
    int nb;                    // -1 = none
    int place;                 // 4 * (cell - the CTA's first cell) + j
    uint8_t meta;
    int record;
    static __device__ __forceinline__ unsigned long long pack(int nb, int place, uint8_t meta, int record) {
        return (unsigned long long)((unsigned)record << 8 | meta) << 32 |
               ((unsigned)place << 24 | (unsigned)(nb < 0 ? NO_NB : nb));
    }
    static __device__ __forceinline__ SlotRef unpack(unsigned long long w) {
        const unsigned lo = (unsigned)w, hi = (unsigned)(w >> 32);
        const int nb = (int)(lo & 0xFFFFFFu);
        return {nb == NO_NB ? -1 : nb, (int)(lo >> 24), (uint8_t)(hi & 0xFFu), (int)(hi >> 8)};
    }
};

// One whole step in one launch for small fp64 meshes: a CTA takes a run of at
// most 32 consecutive cells with at most CELL_SLOTS real slots.  One thread
// per real slot computes that slot's flux from its own side (as the reference
// does) into shared memory; meanwhile the last warp, one lane per cell, loads
// its cells and forms what does not depend on the fluxes (friction, variant
// F's time step); after a block barrier it sums the terms and updates the
// cells.  Every edge is computed twice and nothing passes through device
// memory between flux and update, so a step is one chain of latencies instead
// of two; that pays while the chip is not full (hb_cells.cu has the line).
// Same operations per slot and per cell, so the same bits as the two-kernel
// step.  COEF as in update_kernel.
//
// Bound by that chain: of a 3.9 us step at 6,675 cells about 1.3 us is the
// launch and the state's way through L2, the rest dependent fp64 operations.
// What shortened it there: one launch 8.4 -> 5.1 us; the update warp's early
// work and the step index read ahead of the wait 5.1 -> 4.3 us; the common
// case ahead of the general one (slot_common) 4.4 -> 3.9 us (it costs where
// many warps hold both: a developed dam break at 24,021 cells 5.7 -> 6.7 us).
// 96 slots per CTA are 32 triangles, one update warp; 7 CTAs per SM hold
// 33,000 cells at once.
constexpr int CELL_SLOTS = 96, CELL_MAX = 32, CELL_THREADS = CELL_SLOTS + CELL_MAX;
constexpr int CELL_TERMS = 18;   // values per cell in shared memory: 4 slots x 4, padded off the bank period
constexpr int CELL_CTAS = 7;     // CTAs per SM asked of the compiler
// tick > 0 (the last step of a sequence of that many): the CTA that is done
// last advances the step counter by it, and no launch of its own is needed for
// that.  That, and the last step's zero-length slots evaluated by the update
// warp while it waits, took 20 single steps and a read of the state at 1,500
// mixed cells from 160 to 147 and 129 us.
template <class A, int VARIANT, bool COEF>
__global__ void __launch_bounds__(CELL_THREADS, CELL_CTAS) cell_kernel(DevMesh<A> m, int k, int write_flux, int tick) {
    using R = typename A::real;
    using L = typename A::level;
    __shared__ __align__(16) R terms[CELL_TERMS * CELL_MAX];
    const int t = threadIdx.x;
    const int4 d = m.cseg[blockIdx.x];   // {first cell, cells, first slot record, slot records}
    // The step counter was last written before this sequence.  From the
    // second step on it is read before the dependency wait: this kernel can
    // only have been launched once every CTA of the step before had passed
    // its own wait, so everything before that step is complete.
    StepIndex si;
    if (k > 0) si = step_index<true>(m, k, m.per_day, m.ndays);
    if (t < CELL_SLOTS) {
        // constant tables: read before the dependency wait (ZBC and FNC, which
        // the adjoint's parameters change between sequences, from L2)
        Vec4<R> g{R(0), R(0), R(0), R(0)};
        SlotRef ref{-1, 0, 0, 0};
        L zba = L(0), zbb = L(0);
        int ca = 0, cb = -1;   // the lower-numbered cell of the edge and the other (slot_common); the slot's own if alone
        bool direct = true;
        if (t < d.w) {
            g = ldg4(m.sgeo + 4 * (size_t)(d.z + t));
            ref = SlotRef::unpack((unsigned long long)__double_as_longlong((double)g.w));
            direct = ref.nb < 0 || (ref.meta & META_OWN_FIRST);
            ca = d.x + (ref.place >> 2);
            cb = ref.nb;
            if (!direct) { cb = ca; ca = ref.nb; }
            zba = __ldcg(m.zbc + ca);
            if (cb >= 0) zbb = __ldcg(m.zbc + cb);
        }
        StepParams p{m.hm1, m.hm2, m.jl, m.dt, 1, 0};
        const bool timed = code_is_bounda((int8_t)(ref.meta & META_CODE));
        if (k > 0 && timed) p = with_time(p, si);
        cudaGridDependencySynchronize();
        cudaTriggerProgrammaticLaunchCompletion();
        if (k == 0) {
            si = step_index(m, k, m.per_day, m.ndays);
            if (timed) p = with_time(p, si);
        }
        if (t < d.w) {
            const R *S = m.S[si.par];
            const int sa = 4 * d.x + ref.place;
            const Vec4<R> va = ldg4(S + 4 * (size_t)ca);
            const CellStateA<A> a{va.x, va.y, va.z, va.w, zba};
            CellStateA<A> b{R(0), R(0), R(0), L(0), L(0)};
            if (cb >= 0) {
                const Vec4<R> vb = ldg4(S + 4 * (size_t)cb);
                b = {vb.x, vb.y, vb.z, vb.w, zbb};
            }
            uint8_t meta = ref.meta;
            if ((meta & META_CODE) == CODE_K7) meta = m.rmeta[ref.record];   // breached since?
            const Terms<R, true> tout{terms + CELL_TERMS * (ref.place >> 2) + 4 * (ref.place & 3), sa};
            R f[4];
            if ((meta & META_CODE) == CODE_ZERO && cb >= 0 && slot_common<A>(a, b, direct, g.x, g.y, p, f)) {
                if (write_flux) store_flux(m, sa, f);
                store_terms<A>(tout, sa, f, g.z, g.x, g.y);
            } else {
                single_core<A, VARIANT>(m, ref.record, sa >> 2, sa, direct ? a : b, direct ? b : a, meta, g, p,
                                        write_flux, tout);
            }
        }
        __syncthreads();
    } else {
        const int i = t - CELL_SLOTS, c = d.x + i;
        const bool on = i < d.y;
        CellIn<A> in{};
        if (on) in = load_cell_constants<A, VARIANT, true>(m, c);
        cudaGridDependencySynchronize();
        cudaTriggerProgrammaticLaunchCompletion();
        if (k == 0) si = step_index(m, k, m.per_day, m.ndays);
        const StepParams p{m.hm1, m.hm2, m.jl, m.dt, 1, 0};
        // a cell that is shallow now rarely needs its friction: it is formed late if it does
        Friction<R> f{R(0), R(0), R(0)};
        R dta = R(0);
        auto friction = [&]() { return cell_friction<A>(in.raw.x, in.raw.y, in.raw.z, in.fnc, p); };
        bool ready = false;
        if (on) {
            in.raw = ldg4(m.S[si.par] + 4 * (size_t)c);
            dta = cell_dta<A, VARIANT>(in.raw.x, in.raw.y, in.dta, in.sidex, p);
            ready = in.raw.x > A::c(p.hm2);
            if (ready) f = friction();
            // the last step's zero-length slots, while the others' fluxes are formed
            if (write_flux && (in.mask & 15u) != 15u)
                store_zero(m, c, in.mask,
                           zero_slot<A, VARIANT>(CellStateA<A>{in.raw.x, in.raw.y, in.raw.z, in.raw.w, in.zbc}, p, 1));
        }
        __syncthreads();
        if (on)
            update_core<A, VARIANT, COEF, TERMS_SMEM_LATE>(m, c, in, si, p, write_flux, terms + CELL_TERMS * i,
                                                [&]() { return dta; },
                                                [&]() { return ready ? f : friction(); });
        // every thread of the CTA has used the counter by the barrier above
        if (tick > 0 && i == 0 && atomicAdd(m.tick, 1u) == gridDim.x - 1) {
            *m.tick = 0u;
            *m.step_ctr += tick;
        }
    }
}

// The whole step of one tile (tile layout): every record of the tile writes
// its slots' terms into shared memory, then each cell of the tile sums its
// four slots in order and is updated.  Slots of edges that leave the tile are
// single records, computed by each tile for its own slot as the reference
// computes every slot; the state of the neighbour across is read from global
// memory, where the previous step (the previous launch) left it.
//
// The next pair's record is loaded while one is computed; the first one, the
// step index and the first cell's constants are loaded ahead of what they
// would wait behind.
//
// A 207,234-cell mesh is one wave of 590 CTAs, four to an SM (fp32 and split),
// bound by issue (half of the cycles) and the latencies of its phases.  us per
// step, split precision, 207,234-cell channel / 500,001-cell dam break, and fp32,
// 61,003 mixed cells, three CTAs to an SM: 13.0 / 29.3 / 7.0 before pair_record's
// common case, 10.4 / 24.8 / 5.8 with it, 10.0 / 23.5 / 5.8 with the next
// record's load, 9.8 / 23.5 / 5.6 with the early loads (four: DEFAULT_TILE_CONFIG).
// Chunks of 32 pairs drawn from a counter: 10.6 / 25.4 / 5.8.
template <class A, int VARIANT, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) tile_kernel(DevMesh<A> m, int k, int write_flux) {
    using R = typename A::real;
    extern __shared__ __align__(16) unsigned char tile_smem[];
    R *terms = reinterpret_cast<R *>(tile_smem);                                       // [max cells][4 slots][4]
    __shared__ int qn;
    const TileDesc td = m.tiles[blockIdx.x];   // constant tables: read before the dependency wait
    const SideQueue queue{reinterpret_cast<int *>(tile_smem + 16 * sizeof(R) * (size_t)m.max_tile_cells), 2 * td.npairs, &qn};
    const ScnParams sp = m.scn[td.scn];
    if (threadIdx.x == 0) qn = 0;
    Record<A> next{};
    if ((int)threadIdx.x < td.npairs) next = load_record(m, td.rec0 + threadIdx.x);
    StepIndex si;
    if (k > 0) si = step_index<true>(m, k, sp.per_day, sp.ndays);   // as cell_kernel
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    if (k == 0) si = step_index(m, k, sp.per_day, sp.ndays);
    const StepParams p{sp.hm1, sp.hm2, sp.jl, sp.dt, 1, 0};
    const Terms<R, true> tout{terms, 4 * td.cell0};
    __syncthreads();
    for (int i = threadIdx.x; i < td.npairs; i += THREADS) {
        const Record<A> q = next;
        if (i + THREADS < td.npairs) next = load_record(m, td.rec0 + i + THREADS);
        pair_record<A>(m, td.rec0 + i, q, si, p, write_flux, tout, queue);
    }
    __syncthreads();
    // the singles and the queued sides
    const int nq = qn, sides = td.nsingles + 2 * nq;
    for (int j = threadIdx.x; j < sides; j += THREADS) {
        const bool single = j < td.nsingles;
        side_record<A, VARIANT>(m, single ? 2 * (td.rec0 + td.npairs + j) : queue.item(j - td.nsingles, nq), !single, si,
                                p, write_flux, tout);
    }
    CellIn<A> in{};
    if ((int)threadIdx.x < td.cells) in = load_cell_constants<A, VARIANT>(m, td.cell0 + threadIdx.x);
    __syncthreads();
    for (int c = threadIdx.x; c < td.cells; c += THREADS) {
        if (c != (int)threadIdx.x) in = load_cell_constants<A, VARIANT>(m, td.cell0 + c);
        update_one<A, VARIANT, false, TERMS_SMEM>(m, td.cell0 + c, in, si, p, write_flux, terms + 16 * c);
    }
}

// ---------------------------------------------------------------------------
// persistent step sequence (edge layout, hb_options.persistent)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Backstop of a barrier wait when the global timer does not advance: each
// poll is an L2 round trip (>= 0.3 us), so this many polls last >= 10 s.
constexpr unsigned BARRIER_MAX_POLLS = 1u << 25;

// Grid-wide barrier of a cooperative launch.  bar[0] counts CTA arrivals
// since the launch began and bar[1] is the launch's give-up flag (the host
// zeroes both before each launch); a barrier returns once `target` arrivals
// are counted.  The wait is bounded: after limit_ns of the global timer (or
// BARRIER_MAX_POLLS polls), or as soon as another CTA of this launch has given
// up, it raises the flag and the sticky ERRBIT_BARRIER (which hb_sync reports)
// and returns false, and the caller's CTA leaves the kernel, so a barrier that
// cannot complete ends the launch with a status instead of a hang.  The flag
// is per launch, so an error bit left by an earlier launch (or restored from
// a checkpoint) does not end later launches.  Ordering is the grid-sync
// pattern: the CTA's writes are ordered before thread 0's arrival by
// __syncthreads and a device fence, and thread 0's fence after it saw the
// count orders the CTA's later reads after every arrived CTA's writes.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned target, uint32_t *err,
                                             unsigned long long limit_ns) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        __threadfence();
        unsigned seen = atomicAdd(bar, 1u) + 1u;
        if (seen < target) {
            const unsigned long long t0 = global_ns();
            for (unsigned polls = 1;; polls++) {
                __nanosleep(32);
                seen = *(volatile unsigned *)bar;
                if (seen >= target) break;
                if ((polls & 15u) == 0) {
                    const bool other_gave_up = *(volatile unsigned *)(bar + 1) != 0u;
                    if (other_gave_up || global_ns() - t0 > limit_ns || polls >= BARRIER_MAX_POLLS) {
                        atomicExch(bar + 1, 1u);
                        atomicOr(err, ERRBIT_BARRIER);
                        good = 0;
                        break;
                    }
                }
            }
        }
        __threadfence();
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// All n steps of a sequence in one cooperative launch whose CTAs are all
// resident: per step, the flux records in chunks of THREADS (batch: the flux
// segment table's entries) over the CTAs, a grid barrier, the cells in chunks
// of UPDATE_THREADS (batch: the cell segment table's entries), and a grid
// barrier before the next step.  Each chunk runs exactly as one CTA of
// flux_kernel / update_kernel does, so the results are those of the two-kernel
// sequence bit for bit.  `phantom` adds arrivals that never come to every
// barrier (0 in use; > 0 only to exercise the bounded wait).
template <class A, int VARIANT, int THREADS, int MINB, bool SEG>
__global__ void __launch_bounds__(THREADS, MINB)
    persistent_kernel(DevMesh<A> m, int n, int nflux, int ncell, unsigned *bar, unsigned phantom,
                      unsigned long long limit_ns) {
    // The queue of sides collects those of several chunks and is run when the
    // chunks since could have filled it but for one, and at the end of the flux
    // phase: one block barrier per chunk instead of three.  The bound is counted
    // from the chunks' records, the same in every thread: the queue's own count
    // may already hold the next chunk's sides when a slow thread reads it.
    // Every queued side is run before the grid barrier, as flux_kernel runs it
    // before it ends.
    constexpr int QCAP = 16 * THREADS;
    __shared__ int entries[QCAP];
    __shared__ int qn;
    const SideQueue queue{entries, QCAP, &qn};
    const Terms<typename A::real> tout{m.slotw, 0};
    unsigned arrivals = 0;
    if (threadIdx.x == 0) qn = 0;
    __syncthreads();
    // all threads; empties the queue (pairs: whether a batch's chunk holds pairs)
    auto run_queue = [&](const StepIndex &si, const StepParams &p, int wf, bool pairs) {
        const int nq = qn;
        for (int j = threadIdx.x; j < 2 * nq; j += THREADS) {
            const int e = queue.item(j, nq);
            if (SEG ? pairs : e >= 0 && (e >> 1) < m.npairs) pair_side<A, VARIANT>(m, e, si, p, wf, tout);
            else if (e >= 0) side_record<A, VARIANT>(m, e, false, si, p, wf, tout);
        }
        __syncthreads();
        if (threadIdx.x == 0) qn = 0;
        __syncthreads();
    };
    for (int k = 0; k < n; k++) {
        const int wf = k == n - 1;
        StepIndex si0{};
        StepParams p0{};
        if constexpr (!SEG) {
            si0 = step_index(m, k, m.per_day, m.ndays);
            p0 = StepParams{m.hm1, m.hm2, m.jl, m.dt, 1, 0};
        }
        int bound = 0;   // sides that the chunks since the queue was last run may have queued
        for (int b = blockIdx.x; b < nflux; b += gridDim.x) {
            int r0, cnt;
            bool seg_pairs = false;
            StepIndex si = si0;
            StepParams p = p0;
            if constexpr (SEG) {
                const int4 d = m.fseg[b];
                const ScnParams sp = m.scn[d.x];
                si = step_index(m, k, sp.per_day, sp.ndays);
                p = StepParams{sp.hm1, sp.hm2, sp.jl, sp.dt, 1, 0};
                r0 = d.y;
                cnt = d.z;
                seg_pairs = d.w != 0;
            } else {
                r0 = (m.rev_flux ? nflux - 1 - b : b) * THREADS;   // boundary singles first, as flux_kernel
                cnt = min(THREADS, m.nrecords - r0);
            }
            if ((int)threadIdx.x < cnt) {
                const int r = r0 + (int)threadIdx.x;
                const bool pair = SEG ? seg_pairs : r < m.npairs;
                if (pair) pair_record<A>(m, r, load_record(m, r), si, p, wf, tout, queue);
                else queue.push(2 * r, -1);
            }
            __syncthreads();   // the queue's count is complete
            // a batch chunk's sides have their scenario's parameters: its queue
            // runs at once; a single mesh's when another chunk might not fit
            bound += 2 * cnt;
            if (SEG || bound > QCAP - 2 * THREADS) {
                run_queue(si, p, wf, seg_pairs);
                bound = 0;
            }
        }
        if constexpr (!SEG) run_queue(si0, p0, wf, false);
        arrivals += gridDim.x;
        if (!grid_barrier(bar, arrivals + phantom, m.err, limit_ns)) return;
        for (int b = blockIdx.x; b < ncell; b += gridDim.x) {
            int c0, cnt;
            StepIndex si;
            StepParams p;
            if constexpr (SEG) {
                const int4 d = m.useg[b];
                const ScnParams sp = m.scn[d.x];
                si = step_index(m, k, sp.per_day, sp.ndays);
                p = StepParams{sp.hm1, sp.hm2, sp.jl, sp.dt, 1, 0};
                c0 = d.y;
                cnt = d.z;
            } else {
                si = step_index(m, k, m.per_day, m.ndays);
                p = StepParams{m.hm1, m.hm2, m.jl, m.dt, 1, 0};
                c0 = b * UPDATE_THREADS;
                cnt = min(UPDATE_THREADS, m.C - c0);
            }
            for (int i = threadIdx.x; i < cnt; i += THREADS)
                update_one<A, VARIANT>(m, c0 + i, load_cell_constants<A, VARIANT>(m, c0 + i), si, p, wf,
                                       m.slotw + 16 * (size_t)(c0 + i));
        }
        if (k + 1 < n) {
            arrivals += gridDim.x;
            if (!grid_barrier(bar, arrivals + phantom, m.err, limit_ns)) return;
        }
    }
}

// Advances the step counter after a step sequence.  Launched with
// programmatic dependent launch like the step kernels: it waits for the last
// step's results and lets the next kernel launch at once.
static __global__ void tick_kernel(long long *ctr, int n) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    *ctr += n;
}

// Split precision state <-> the reference's (H, Z) of one cell.  The depth is
// kept as the fp32 pair (h, hlo) with h + hlo = H; a cell at or below the dry
// threshold keeps in hlo the offset of its level instead (split_level).
struct SplitCodec {
    static __host__ __device__ inline void encode(double H, double Z, double zbc, float hm1f, float &h, float &hlo) {
        h = (float)H;
        hlo = h > hm1f ? (float)(H - (double)h) : (float)((Z - zbc) - (double)h);
    }
    static __host__ __device__ inline double depth(float h, float hlo, float hm1f, double hm1) {
        return h > hm1f ? (double)h + (double)hlo : (h == hm1f ? hm1 : (double)h);
    }
    static __host__ __device__ inline double level(float h, float hlo, double zbc) {
        return (double)h + ((double)hlo + zbc);
    }
};

// Flux array k of one scenario's cells ([slot][4] records, device order) into
// reference order.
template <class R>
__global__ void flux_out_kernel(const R *__restrict__ flux, int cells, int k, const int32_t *__restrict__ perm,
                                double *__restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < 4 * cells) out[4 * (size_t)perm[s >> 2] + (s & 3)] = (double)flux[4 * (size_t)s + k];
}
// Flux array k of n records to an array of its own, or (SET) back.
template <class R, bool SET>
__global__ void flux_array_kernel(R *flux, size_t n, int k, R *array) {
    const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    if (SET) flux[4 * s + k] = array[s];
    else array[s] = flux[4 * s + k];
}

// Reference-order staging <-> device-order state of one scenario: cells
// [cell0, cell0 + C) of the device state, perm[new] = old within the scenario.
template <class A>
__global__ void stage_in_kernel(DevMesh<A> m, int cell0, int C, double hm1, const int32_t *__restrict__ perm,
                                const double *__restrict__ stage) {
    using R = typename A::real;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C) return;
    const int o = perm[i];
    R *d = m.S[(*m.step_ctr) & 1] + 4 * ((size_t)cell0 + i);
    d[1] = (R)stage[(size_t)C + o];
    d[2] = (R)stage[2 * (size_t)C + o];
    if constexpr (is_split<A>::value) {
        float h, hlo;
        SplitCodec::encode(stage[o], stage[3 * (size_t)C + o], m.zbc[cell0 + i], (float)hm1, h, hlo);
        d[0] = h; d[3] = hlo;
    } else {
        d[0] = (R)stage[o];
        d[3] = (R)stage[3 * (size_t)C + o];
    }
}
template <class A>
__global__ void stage_out_kernel(DevMesh<A> m, int cell0, int C, double hm1, const int32_t *__restrict__ perm,
                                 double *__restrict__ stage) {
    using R = typename A::real;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C) return;
    const int o = perm[i];
    const R *d = m.S[(*m.step_ctr) & 1] + 4 * ((size_t)cell0 + i);
    stage[(size_t)C + o] = (double)d[1];
    stage[2 * (size_t)C + o] = (double)d[2];
    if constexpr (is_split<A>::value) {
        stage[o] = SplitCodec::depth(d[0], d[3], (float)hm1, hm1);
        stage[3 * (size_t)C + o] = SplitCodec::level(d[0], d[3], m.zbc[cell0 + i]);
    } else {
        stage[o] = (double)d[0];
        stage[3 * (size_t)C + o] = (double)d[3];
    }
    stage[4 * (size_t)C + o] = (double)m.W[cell0 + i];
}

// per-cell constants that the update needs, computed on the device with the
// reference's arithmetic (functors.cu:750, v0 functors.cu:752-763)
template <class A, int VARIANT>
__global__ void setup_cells_kernel(int C, double dt, const typename A::real *area, const typename A::real *side4,
                                   typename A::real *dta, typename A::real *sidex) {
    using R = typename A::real;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C) return;
    if (VARIANT == 1) {
        const R s0 = side4[4 * i], s1 = side4[4 * i + 1], s2 = side4[4 * i + 2], s3 = side4[4 * i + 3];
        if (s3 > R(0)) sidex[i] = A::fmin(A::mul(A::c(0.5), A::add(s0, s2)), A::mul(A::c(0.5), A::add(s1, s3)));
        else {
            R ss = A::mul(A::c(0.5), A::add(A::add(s0, s1), s2));
            sidex[i] = A::sqrt(A::div(A::mul(A::mul(A::sub(ss, s0), A::sub(ss, s1)), A::sub(ss, s2)), ss));
        }
        dta[i] = area[i];
    } else {
        dta[i] = A::div(A::c(dt), area[i]);
    }
}

}  // namespace hb
