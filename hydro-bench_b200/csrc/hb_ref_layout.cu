// hb_ref_layout.cu -- CalculateFlux / UpdateCell over the caller's own arrays
// in the reference layout (functors.cu:787-818).  One thread per slot for the
// flux (sorted within the block by what a slot needs), one per cell for the
// update; the arithmetic is the shared physics of hb_physics.cuh.
#include "hb_common.cuh"
#include "hb_physics.cuh"
#include "hydrob200_refview.h"

namespace hb {

__device__ uint32_t g_ref_errors;

template <class R>
struct RefView;
template <>
struct RefView<double> { using type = hb_ref_mesh_view; };
template <>
struct RefView<float> { using type = hb_ref_mesh_view_f32; };

// One slot in general, CalculateFluxKernel's body (functors.cu:47-202).
template <class A, int VARIANT>
__device__ __forceinline__ void ref_slot(const typename RefView<typename A::real>::type &m, int idx, int kt, int jt) {
    using R = typename A::real;
    const int pos = idx >> 2;
    const auto &c = m.cells;
    const auto &sd = m.sides;
    SlotIn<R> in;
    in.own = {c.H[pos], c.U[pos], c.V[pos], c.Z[pos], c.ZBC[pos]};
    const int nc = (int)(sd.NAC[idx] - R(1));
    in.has_nb = nc != -1;
    in.own_first = pos < nc;
    if (in.has_nb) in.nb = {c.H[nc], c.U[nc], c.V[nc], c.Z[nc], c.ZBC[nc]};
    else in.nb = {R(0), R(0), R(0), R(0), R(0)};
    in.code = klas_code((double)sd.KLAS[idx]);
    in.cosj = sd.COSF[idx];
    in.sinj = sd.SINF[idx];
    in.side = sd.SIDE[idx];
    StepParams p{(double)m.HM1, (double)m.HM2, (double)m.JL, (double)m.DT, kt, jt};
    auto fetch = [&]() {
        BoundaryIn<R> b;
        const size_t t = (size_t)jt * (size_t)m.CELL + (size_t)pos;
        b.qt = c.QT[t]; b.dqt = c.DQT[t]; b.zt = c.ZT[t]; b.dzt = c.DZT[t];
        b.top = c.BoundaryFeature[pos];
        b.zw = c.ZW + (size_t)pos * (size_t)m.NHQ;
        b.qw = c.QW + (size_t)pos * (size_t)m.NHQ;
        b.nhq1 = c.NHQ1[pos];
        b.nhq = m.NHQ;
        return b;
    };
    SlotOut<R> o;
    flux_slot<A, VARIANT>(in, p, fetch, o);
    if (o.undefined) atomicOr(&g_ref_errors, ERRBIT_UNDEFINED);
    if (o.klas_to_zero) sd.KLAS[idx] = R(0);
    if (o.mask & 1) sd.FLUX0[idx] = o.f[0];
    if (o.mask & 2) sd.FLUX1[idx] = o.f[1];
    if (o.mask & 4) sd.FLUX2[idx] = o.f[2];
    if (o.mask & 8) sd.FLUX3[idx] = o.f[3];
}

// One slot per thread, sorted within the block: the interior slots with code 0
// to the front threads, those without neighbour (a quarter of a triangle mesh's
// slots, one in every group of four lanes, whose flux takes a power) to the
// last ones, so that a warp runs one of the two common cases (slot_common,
// closed_common).  The others, and the slots that are in no common case, go to
// the block's queue and run the general path together at the end.
//
// Bound by the gathers' latency and by issue.  207,234 triangles, flux kernel
// alone: every slot through the whole chain in place 36 us and more, the common
// case in place and the rest in the queue 35.5 us (11.4 M warp instructions),
// sorted 26.4 us (9.6 M); the pair of calls 42.6 -> 29.5 us.  8 CTAs per SM (64
// registers) instead of 7, with the general slots' square root only where it is
// used: the pair of calls 30.0 -> 28.9 us, thin sheet flow 45.6 -> 41.2 us (41.5
// with the chain in place), supercritical 41.2 -> 30.6 us.
constexpr int REF_THREADS = 128;
template <class A, int VARIANT>
__global__ void __launch_bounds__(REF_THREADS, 8) ref_flux_kernel(const __grid_constant__
                                                               typename RefView<typename A::real>::type m,
                                                               int kt, int jt) {
    using R = typename A::real;
    __shared__ int2 list[REF_THREADS];   // {slot - the block's first, neighbour}
    __shared__ int queue[REF_THREADS];
    __shared__ int qn, nopen, nclosed;
    const int t = threadIdx.x;
    if (t == 0) qn = nopen = nclosed = 0;
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    __syncthreads();
    const int base = blockIdx.x * REF_THREADS;
    const auto &c = m.cells;
    const auto &sd = m.sides;
    if ((long long)base + t < 4LL * m.CELL) {
        const int nc = (int)(sd.NAC[base + t] - R(1));
        if (sd.KLAS[base + t] != R(0)) queue[atomicAdd(&qn, 1)] = base + t;
        else if (nc != -1) list[atomicAdd(&nopen, 1)] = make_int2(t, nc);
        else list[REF_THREADS - 1 - atomicAdd(&nclosed, 1)] = make_int2(t, -1);
    }
    __syncthreads();
    const bool open = t < nopen;
    if (open || t >= REF_THREADS - nclosed) {
        const int2 e = list[t];
        const int idx = base + e.x, pos = idx >> 2;
        const StepParams p{(double)m.HM1, (double)m.HM2, (double)m.JL, (double)m.DT, kt, jt};
        auto cell = [&](int i) { return CellState<R>{c.H[i], c.U[i], c.V[i], c.Z[i], c.ZBC[i]}; };
        R f[4];
        bool done;
        if (open) {
            const bool direct = pos < e.y;
            const int ca = direct ? pos : e.y, cb = direct ? e.y : pos;
            done = slot_common<A>(cell(ca), cell(cb), direct, sd.COSF[idx], sd.SINF[idx], p, f);
        } else {
            done = closed_common<A>(cell(pos), sd.COSF[idx], sd.SINF[idx], p, f);
        }
        if (done) {
            sd.FLUX0[idx] = f[0]; sd.FLUX1[idx] = f[1]; sd.FLUX2[idx] = f[2]; sd.FLUX3[idx] = f[3];
        } else {
            queue[atomicAdd(&qn, 1)] = idx;
        }
    }
    __syncthreads();
    if (t < qn) ref_slot<A, VARIANT>(m, queue[t], kt, jt);
}

// The four values of a cell in a slot array: one vector load where every slot
// array is aligned to it (VEC, the launch's check), four loads otherwise.
template <bool VEC>
__device__ __forceinline__ void ld_slots(const double *p, double v[4]) {
    if constexpr (VEC) {
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p) : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = p[j];
    }
}
template <bool VEC>
__device__ __forceinline__ void ld_slots(const float *p, float v[4]) {
    if constexpr (VEC) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = p[j];
    }
}

template <class A, int VARIANT, bool VEC>
__global__ void __launch_bounds__(REF_THREADS, 6) ref_update_kernel(typename RefView<typename A::real>::type m) {
    using R = typename A::real;
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int pos = blockIdx.x * REF_THREADS + threadIdx.x;
    if (pos >= m.CELL) return;
    const auto &c = m.cells;
    const auto &sd = m.sides;
    const size_t s = 4 * (size_t)pos;
    CellUpdateIn<R> ci;
    ci.h = c.H[pos]; ci.u = c.U[pos]; ci.v = c.V[pos]; ci.zbc = c.ZBC[pos]; ci.fnc = c.FNC[pos];
    ci.hlo = R(0);
    const R area = c.AREA[pos];
    R f0[4], f1[4], f2[4], f3[4], side[4], slcos[4], slsin[4];
    ld_slots<VEC>(sd.FLUX0 + s, f0);
    ld_slots<VEC>(sd.SIDE + s, side);
    ld_slots<VEC>(sd.FLUX1 + s, f1);
    ld_slots<VEC>(sd.FLUX3 + s, f3);
    ld_slots<VEC>(sd.FLUX2 + s, f2);
    ld_slots<VEC>(sd.SLCOS + s, slcos);
    ld_slots<VEC>(sd.SLSIN + s, slsin);
    R wh = R(0), wu = R(0), wv = R(0);
#pragma unroll
    for (int j = 0; j < 4; j++) wsum_add<A>(wh, wu, wv, f0[j], f1[j], f2[j], f3[j], side[j], slcos[j], slsin[j]);
    R dta, sidex = R(0);
    if (VARIANT == 1) {
        // SIDEX: triangle inradius or smaller mid-width of a quad (v0 functors.cu:752-763)
        const R s0 = side[0], s1 = side[1], s2 = side[2], s3 = side[3];
        if (s3 > R(0)) {
            sidex = A::fmin(A::mul(A::c(0.5), A::add(s0, s2)), A::mul(A::c(0.5), A::add(s1, s3)));
        } else {
            R ss = A::mul(A::c(0.5), A::add(A::add(s0, s1), s2));
            sidex = A::sqrt(A::div(A::mul(A::mul(A::sub(ss, s0), A::sub(ss, s1)), A::sub(ss, s2)), ss));
        }
        dta = area;
    } else {
        dta = A::div(A::c((double)m.DT), area);
    }
    StepParams p{(double)m.HM1, (double)m.HM2, (double)m.JL, (double)m.DT, 0, 0};
    dta = cell_dta<A, VARIANT>(ci.h, ci.u, dta, sidex, p);
    CellUpdateOut<R> o = update_cell<A, VARIANT>(ci, dta, wh, wu, wv, p,
                                                 [&]() { return cell_friction<A>(ci.h, ci.u, ci.v, ci.fnc, p); });
    c.H[pos] = o.h; c.U[pos] = o.u; c.V[pos] = o.v; c.Z[pos] = o.z; c.W[pos] = speed<A>(o.u, o.v);
}

// Launched with programmatic dependent launch: both kernels wait for their
// predecessor's results before they touch the caller's arrays.
template <class... P, class... Args>
static int ref_launch(void (*kernel)(P...), long long threads, void *stream, Args... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((threads + REF_THREADS - 1) / REF_THREADS));
    cfg.blockDim = dim3(REF_THREADS);
    cfg.stream = (cudaStream_t)stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HB_CUDA_RET(cudaLaunchKernelEx(&cfg, kernel, args...));
    return HB_OK;
}

template <class A, class View>
static int launch_flux(const View *m, int kt, int jt, int variant, void *stream) {
    if (!m || m->CELL < 0) return set_error(HB_E_INVALID, "hb_ref_calculate_flux: bad mesh view");
    if (m->CELL == 0) return HB_OK;
    if (jt < 0 || jt >= m->NDAYS) return set_error(HB_E_INVALID, "hb_ref_calculate_flux: jt=%d outside [0,%d)", jt, m->NDAYS);
    return ref_launch(variant == HB_VARIANT_F ? ref_flux_kernel<A, 1> : ref_flux_kernel<A, 0>, 4LL * m->CELL, stream, *m,
                      kt, jt);
}

template <class A, class View>
static int launch_update(const View *m, int variant, void *stream) {
    if (!m || m->CELL < 0) return set_error(HB_E_INVALID, "hb_ref_update_cell: bad mesh view");
    if (m->CELL == 0) return HB_OK;
    using R = typename A::real;
    const auto &s = m->sides;
    const void *slots[] = {s.FLUX0, s.FLUX1, s.FLUX2, s.FLUX3, s.SIDE, s.SLCOS, s.SLSIN};
    bool vec = true;
    for (const void *q : slots) vec = vec && (uintptr_t)q % (4 * sizeof(R)) == 0;
    const bool f = variant == HB_VARIANT_F;
    auto kernel = f ? (vec ? ref_update_kernel<A, 1, true> : ref_update_kernel<A, 1, false>)
                    : (vec ? ref_update_kernel<A, 0, true> : ref_update_kernel<A, 0, false>);
    return ref_launch(kernel, m->CELL, stream, *m);
}

}  // namespace hb

extern "C" int hb_ref_calculate_flux(const hb_ref_mesh_view *mesh, int32_t kt, int32_t jt, int32_t variant, void *stream) {
    return hb::launch_flux<hb::F64Exact>(mesh, kt, jt, variant, stream);
}
extern "C" int hb_ref_update_cell(const hb_ref_mesh_view *mesh, int32_t variant, void *stream) {
    return hb::launch_update<hb::F64Exact>(mesh, variant, stream);
}
extern "C" int hb_ref_calculate_flux_f32(const hb_ref_mesh_view_f32 *mesh, int32_t kt, int32_t jt, int32_t variant, void *stream) {
    return hb::launch_flux<hb::F32Fast>(mesh, kt, jt, variant, stream);
}
extern "C" int hb_ref_update_cell_f32(const hb_ref_mesh_view_f32 *mesh, int32_t variant, void *stream) {
    return hb::launch_update<hb::F32Fast>(mesh, variant, stream);
}
extern "C" int hb_ref_take_device_errors(uint32_t *bits) {
    uint32_t v = 0, zero = 0;
    HB_CUDA_RET(cudaMemcpyFromSymbol(&v, hb::g_ref_errors, sizeof v));
    HB_CUDA_RET(cudaMemcpyToSymbol(hb::g_ref_errors, &zero, sizeof zero));
    if (bits) *bits = v;
    return HB_OK;
}

// Reference-signature overloads (functors.cuh:59-65).  The reference exits the
// process on a CUDA error (common.hpp:57-59); these report on stderr instead.
static void report(int st, const char *what) {
    if (st != HB_OK) fprintf(stderr, "hydrob200: %s failed: %s\n", what, hb_last_error_string());
}
void CalculateFlux(const MeshView &mesh, int kt, int jt, CUstream_st *stream) {
    report(hb_ref_calculate_flux(reinterpret_cast<const hb_ref_mesh_view *>(&mesh), kt, jt, HB_VARIANT_H, stream),
           "CalculateFlux");
}
void UpdateCell(const MeshView &mesh, CUstream_st *stream) {
    report(hb_ref_update_cell(reinterpret_cast<const hb_ref_mesh_view *>(&mesh), HB_VARIANT_H, stream), "UpdateCell");
}
void CalculateFlux(const MeshView &mesh, int kt, int jt) {
    CalculateFlux(mesh, kt, jt, nullptr);
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) fprintf(stderr, "hydrob200: CalculateFlux: %s\n", cudaGetErrorString(e));
}
void UpdateCell(const MeshView &mesh) {
    UpdateCell(mesh, nullptr);
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) fprintf(stderr, "hydrob200: UpdateCell: %s\n", cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------
// hb_ref_step_static: one step with a fixed, library-owned scratch array
// ---------------------------------------------------------------------------
#include <mutex>

namespace hb {

// [HB_REF_STEP_STATIC_MAX_CELLS * 4 slots][4] = {F0, dWU, dWV, SIDE} per slot.
// Host code must not take this name as a device address: it is a host-side
// stand-in; the device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) double g_static_terms[(size_t)HB_REF_STEP_STATIC_MAX_CELLS * 16];

constexpr int MAX_DEVICES = 64;
static std::mutex g_static_mu;
static double *g_static_ptr[MAX_DEVICES];

// device address of g_static_terms on the current device (looked up once per device)
static int static_terms_ptr(double **out) {
    int dev = -1;
    HB_CUDA_RET(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) return set_error(HB_E_INVALID, "hb_ref_step_static: device %d", dev);
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_terms);
        if (e != cudaSuccess || !p)
            return set_error(HB_E_CUDA, "hb_ref_step_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_static_ptr[dev] = static_cast<double *>(p);
    }
    *out = g_static_ptr[dev];
    return HB_OK;
}

// CalculateFluxKernel's writes (FLUX0..3 by the slot's mask, KLAS on breach)
// plus the slot's terms of the cell sums (functors.cu:733-741) into `terms`.
template <int VARIANT>
__global__ void __launch_bounds__(256) static_flux_kernel(hb_ref_mesh_view m, int kt, int jt, double *terms) {
    using A = F64Exact;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 4 * m.CELL) return;
    const int pos = idx >> 2;
    const auto &c = m.cells;
    const auto &sd = m.sides;
    SlotIn<double> in;
    in.own = {c.H[pos], c.U[pos], c.V[pos], c.Z[pos], c.ZBC[pos]};
    const int nc = (int)(sd.NAC[idx] - 1.0);
    in.has_nb = nc != -1;
    in.own_first = pos < nc;
    if (in.has_nb) in.nb = {c.H[nc], c.U[nc], c.V[nc], c.Z[nc], c.ZBC[nc]};
    else in.nb = {0.0, 0.0, 0.0, 0.0, 0.0};
    in.code = klas_code(sd.KLAS[idx]);
    in.cosj = sd.COSF[idx];
    in.sinj = sd.SINF[idx];
    in.side = sd.SIDE[idx];
    StepParams p{m.HM1, m.HM2, m.JL, m.DT, kt, jt};
    auto fetch = [&]() {
        BoundaryIn<double> b;
        const size_t t = (size_t)jt * (size_t)m.CELL + (size_t)pos;
        b.qt = c.QT[t]; b.dqt = c.DQT[t]; b.zt = c.ZT[t]; b.dzt = c.DZT[t];
        b.top = c.BoundaryFeature[pos];
        b.zw = c.ZW + (size_t)pos * (size_t)m.NHQ;
        b.qw = c.QW + (size_t)pos * (size_t)m.NHQ;
        b.nhq1 = c.NHQ1[pos];
        b.nhq = m.NHQ;
        return b;
    };
    SlotOut<double> o;
    flux_slot<A, VARIANT>(in, p, fetch, o);
    if (o.undefined) atomicOr(&g_ref_errors, ERRBIT_UNDEFINED);
    if (o.klas_to_zero) sd.KLAS[idx] = 0.0;
    // fluxes this slot does not write keep their values (functors.cu:525-565)
    if (o.mask & 1) sd.FLUX0[idx] = o.f[0]; else o.f[0] = sd.FLUX0[idx];
    if (o.mask & 2) sd.FLUX1[idx] = o.f[1]; else o.f[1] = sd.FLUX1[idx];
    if (o.mask & 4) sd.FLUX2[idx] = o.f[2]; else o.f[2] = sd.FLUX2[idx];
    if (o.mask & 8) sd.FLUX3[idx] = o.f[3]; else o.f[3] = sd.FLUX3[idx];
    const double fr1 = A::add(o.f[1], o.f[3]);
    const double slcos = sd.SLCOS[idx], slsin = sd.SLSIN[idx];
    double *t = terms + 4 * (size_t)idx;
    t[0] = o.f[0];
    t[1] = A::dot(slcos, fr1, -slsin, o.f[2], M_WU);
    t[2] = A::dot(slsin, fr1, slcos, o.f[2], M_WV);
    t[3] = in.side;
}

// UpdateCellKernel (functors.cu:717-784) with the sums taken from `terms`.
template <int VARIANT>
__global__ void __launch_bounds__(256) static_update_kernel(hb_ref_mesh_view m, const double *terms) {
    using A = F64Exact;
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= m.CELL) return;
    const auto &c = m.cells;
    const auto &sd = m.sides;
    double wh = 0.0, wu = 0.0, wv = 0.0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const double *t = terms + 16 * (size_t)pos + 4 * j;
        wh = A::madd(t[3], t[0], wh, M_WH);
        wu = A::add(wu, t[1]);
        wv = A::add(wv, t[2]);
    }
    CellUpdateIn<double> ci;
    ci.h = c.H[pos]; ci.u = c.U[pos]; ci.v = c.V[pos]; ci.zbc = c.ZBC[pos]; ci.fnc = c.FNC[pos];
    ci.hlo = 0.0;
    double dta, sidex = 0.0;
    if (VARIANT == 1) {
        const double s0 = sd.SIDE[4 * pos], s1 = sd.SIDE[4 * pos + 1], s2 = sd.SIDE[4 * pos + 2], s3 = sd.SIDE[4 * pos + 3];
        if (s3 > 0.0) {
            sidex = A::fmin(A::mul(0.5, A::add(s0, s2)), A::mul(0.5, A::add(s1, s3)));
        } else {
            double ss = A::mul(0.5, A::add(A::add(s0, s1), s2));
            sidex = A::sqrt(A::div(A::mul(A::mul(A::sub(ss, s0), A::sub(ss, s1)), A::sub(ss, s2)), ss));
        }
        dta = c.AREA[pos];
    } else {
        dta = A::div(m.DT, c.AREA[pos]);
    }
    StepParams p{m.HM1, m.HM2, m.JL, m.DT, 0, 0};
    dta = cell_dta<A, VARIANT>(ci.h, ci.u, dta, sidex, p);
    CellUpdateOut<double> o = update_cell<A, VARIANT>(ci, dta, wh, wu, wv, p,
                                                      [&]() { return cell_friction<A>(ci.h, ci.u, ci.v, ci.fnc, p); });
    c.H[pos] = o.h; c.U[pos] = o.u; c.V[pos] = o.v; c.Z[pos] = o.z; c.W[pos] = speed<A>(o.u, o.v);
}

}  // namespace hb

extern "C" int hb_ref_step_static(const hb_ref_mesh_view *m, int32_t kt, int32_t jt, int32_t variant, void *stream) {
    if (!m || m->CELL < 0) return hb::set_error(HB_E_INVALID, "hb_ref_step_static: bad mesh view");
    if (m->CELL > HB_REF_STEP_STATIC_MAX_CELLS)
        return hb::set_error(HB_E_TOO_LARGE, "hb_ref_step_static: %d cells, the fixed scratch holds %d", m->CELL,
                             HB_REF_STEP_STATIC_MAX_CELLS);
    if (m->CELL == 0) return HB_OK;
    if (jt < 0 || jt >= m->NDAYS)
        return hb::set_error(HB_E_INVALID, "hb_ref_step_static: jt=%d outside [0,%d)", jt, m->NDAYS);
    double *terms = nullptr;
    int st = hb::static_terms_ptr(&terms);
    if (st != HB_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    const int fb = (4 * m->CELL + 255) / 256, ub = (m->CELL + 255) / 256;
    if (variant == HB_VARIANT_F) {
        hb::static_flux_kernel<1><<<fb, 256, 0, s>>>(*m, kt, jt, terms);
        hb::static_update_kernel<1><<<ub, 256, 0, s>>>(*m, terms);
    } else {
        hb::static_flux_kernel<0><<<fb, 256, 0, s>>>(*m, kt, jt, terms);
        hb::static_update_kernel<0><<<ub, 256, 0, s>>>(*m, terms);
    }
    HB_CUDA_RET(cudaGetLastError());
    return HB_OK;
}
