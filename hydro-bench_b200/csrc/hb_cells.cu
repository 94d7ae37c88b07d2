// hb_cells.cu -- the one-launch step of small fp64 meshes (cell_kernel): when
// it is used, its slot table, and its launches.
#include <vector>

#include "hb_handle.hpp"

namespace {

// The one-launch step takes single fp64 meshes whose CTAs are all resident at
// once (edge layout, default launch shape): about 33,000 triangles on a B200.
// It halves the latencies of a step but computes every edge twice, and its
// second wave costs as much as its first.  us per step, 40-step graphs, one
// launch / two kernels (the dam break after 1,500 steps), variant H:
//   cells      24,021      32,000      40,000      60,000
//   channel   4.5 / 7.0   4.6 / 8.1   7.7*/ 8.2   8.7*/ 7.8
//   mixed     5.2 / 7.8   7.7*/ 8.0   8.1*/ 8.5  10.1*/ 10.8
//   dam break 6.3 / 8.7   6.9 / 9.0     -  / 9.3     -  / 10.0
// (* two waves; a mesh with quads has fewer cells to a CTA)
bool fits_at_once(const hb_handle *h, size_t ctas) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->opt.device) != cudaSuccess) return false;
    return ctas <= (size_t)sms * hb::CELL_CTAS;
}

// The slot table is formed on the device: on the host, creating a handle took
// 0.15 ms more at 1,500 cells, 0.7 at 6,675 and 1.1 (of 6.8) at 24,021.
// Device slot -> its record r; the other slot of a pair: -2 - r.
__global__ void slot_record_kernel(const int4 *rix, int nrec, int32_t *record) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrec) return;
    const int4 ix = rix[r];
    record[ix.z] = r;
    if (ix.w >= 0) record[ix.w] = -2 - r;
}
// The slot records of one CTA of cell_kernel, one thread per place (-1 in
// `record`: a triangle's zero-length slot, which has none).  Its boundary
// slots, the slowest ones, come last, so that they share as few warps as
// possible with the others.
__global__ void __launch_bounds__(4 * hb::CELL_MAX)
    slot_table_kernel(hb::DevMesh<hb::F64Exact> m, const int4 *seg, const int32_t *record, double *table) {
    __shared__ int count[2][hb::CELL_MAX / 8];   // inner and boundary slots of each warp
    const int4 d = seg[blockIdx.x];
    const int place = threadIdx.x, warp = place >> 5;
    const int q = place < 4 * d.y ? record[4 * (size_t)d.x + place] : -1;
    const bool real = q != -1, other = q < -1;
    const int r = other ? -2 - q : q;
    // a pair's other slot: negated normal, same length, not the lower-numbered side
    const uint8_t meta = !real ? 0 : other ? (uint8_t)(hb::CODE_ZERO | hb::META_HAS_NB) : m.rmeta[r];
    const int kind = (meta & hb::META_CODE) != hb::CODE_ZERO;
    const unsigned mine[2] = {__ballot_sync(0xffffffffu, real && !kind), __ballot_sync(0xffffffffu, real && kind)};
    if ((place & 31) < 2) count[place & 31][warp] = __popc(mine[place & 31]);
    __syncthreads();
    if (!real) return;
    int at = __popc(mine[kind] & ((1u << (place & 31)) - 1u));
    for (int w = 0; w < hb::CELL_MAX / 8; w++) {
        if (w < warp) at += count[kind][w];
        if (kind) at += count[0][w];
    }
    const int4 ix = m.rix[r];
    const hb::Vec4<double> g = hb::ldg4(m.rgeo + 4 * (size_t)r);
    const unsigned long long w = hb::SlotRef::pack(other ? ix.x : ix.y, place, meta, r);
    hb::stg4(table + 4 * (size_t)(d.z + at), other ? -g.x : g.x, other ? -g.y : g.y, g.z,
             __longlong_as_double((long long)w));
}

template <int VARIANT, bool COEF>
int launch_cells_t(int ncseg, const hb::DevMesh<hb::F64Exact> &m, int k0, int n, int write_last, int tick,
                   cudaStream_t st) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ncseg);
    cfg.blockDim = dim3(hb::CELL_THREADS);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    for (int k = 0; k < n; k++)
        HB_CUDA_RET(cudaLaunchKernelEx(&cfg, hb::cell_kernel<hb::F64Exact, VARIANT, COEF>, m, k0 + k,
                                       (int)(write_last && k == n - 1), k == n - 1 ? tick : 0));
    return HB_OK;
}

}  // namespace

bool hb_cells_used(const hb_handle *h) {
    return h->ncseg > 0 && h->launch_config == hb::DEFAULT_EDGE_CONFIG;
}

int hb_cells_build(hb_handle *h, const std::vector<uint8_t> &cmask) {
    hb::DevMesh<hb::F64Exact> &m = h->m64;
    if (h->opt.precision != HB_FP64 || h->opt.layout != HB_LAYOUT_EDGE || h->opt.persistent || h->segmented() ||
        !fits_at_once(h, (size_t)h->C / hb::CELL_MAX) || m.nrecords >= hb::SlotRef::MAX_RECORD)
        return HB_OK;
    // the CTAs' runs of cells
    std::vector<int4> seg;
    int4 cur = make_int4(0, 0, 0, 0);
    for (int c = 0; c < h->C; c++) {
        const int n = __builtin_popcount(cmask[c]);
        if (cur.w + n > hb::CELL_SLOTS || cur.y == hb::CELL_MAX) {
            seg.push_back(cur);
            cur = make_int4(c, 0, cur.z + cur.w, 0);
        }
        cur.y++;
        cur.w += n;
    }
    seg.push_back(cur);
    if (!fits_at_once(h, seg.size())) return HB_OK;
    // One allocation: the slot records (32-byte aligned), then the CTAs' entries.
    const size_t records = 4 * (size_t)(cur.z + cur.w);
    double *sp;
    TRY(dev_alloc(h, &sp, records + 2 * seg.size()));
    int4 *cp = reinterpret_cast<int4 *>(sp + records);
    HB_CUDA_RET(cudaMemcpy(cp, seg.data(), seg.size() * sizeof(int4), cudaMemcpyHostToDevice));
    // The staging buffer (40 bytes per cell) holds the slots' records (16) meanwhile.
    int32_t *record = reinterpret_cast<int32_t *>(h->d_stage);
    HB_CUDA_RET(cudaMemset(record, 0xFF, 4 * (size_t)h->C * sizeof(int32_t)));
    slot_record_kernel<<<(m.nrecords + 255) / 256, 256>>>(m.rix, m.nrecords, record);
    HB_CUDA_RET(cudaGetLastError());
    slot_table_kernel<<<(unsigned)seg.size(), 4 * hb::CELL_MAX>>>(m, cp, record, sp);
    HB_CUDA_RET(cudaGetLastError());
    HB_CUDA_RET(cudaDeviceSynchronize());
    m.sgeo = sp;
    m.cseg = cp;
    h->ncseg = (int)seg.size();
    return HB_OK;
}

int hb_cells_launch(hb_handle *h, const hb::DevMesh<hb::F64Exact> &m, int k0, int n, int write_last, int tick,
                    bool coef, cudaStream_t st) {
    if (h->opt.variant == HB_VARIANT_F) {
        if (coef) return hb::set_error(HB_E_INVALID, "update coefficients: variant H only");
        return launch_cells_t<1, false>(h->ncseg, m, k0, n, write_last, tick, st);
    }
    return coef ? launch_cells_t<0, true>(h->ncseg, m, k0, n, write_last, tick, st) : launch_cells_t<0, false>(h->ncseg, m, k0, n, write_last, tick, st);
}
