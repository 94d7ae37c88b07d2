// hb_cells.cu -- the one-launch step of small fp64 meshes (cell_kernel): when
// it is used, its slot table, and its launches.
#include <cstring>
#include <vector>

#include "hb_handle.hpp"

namespace {

// The one-launch step takes single fp64 meshes whose CTAs are all resident at
// once (edge layout, default launch shape): about 33,000 triangles on a B200.
// It halves the latencies of a step but computes every edge twice, and its
// second wave costs as much as its first.  us per step, 40-step graphs, one
// launch / two kernels, variant H:
//   cells      24,021      32,000      40,000      60,000
//   channel   4.6 / 6.8   4.6 / 7.7   7.7 / 7.7   8.7*/ 8.7
//   mixed     5.2 / 7.9   7.7*/ 7.7   8.1*/ 8.0  10.1*/ 10.1
//   dam break 6.7 / 8.8   6.8 / 8.9     -  / 9.1     -  / 11.4
// (* two waves)
bool fits_at_once(const hb_handle *h, size_t ctas) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->opt.device) != cudaSuccess) return false;
    return ctas <= (size_t)sms * hb::CELL_CTAS;
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

int hb_cells_build(hb_handle *h, const std::vector<int4> &rix, const std::vector<uint8_t> &rmeta,
                   const std::vector<double> &rgeo) {
    if (h->opt.precision != HB_FP64 || h->opt.layout != HB_LAYOUT_EDGE || h->opt.persistent || h->segmented() ||
        !fits_at_once(h, (size_t)h->C / hb::CELL_MAX) || rix.size() >= (size_t)hb::SlotRef::MAX_RECORD)
        return HB_OK;
    hb::DevMesh<hb::F64Exact> &m = h->m64;
    const int nrec = (int)rix.size();
    // slot -> its record; the other slot of a pair's record r is ~r - 1 (-1: a
    // triangle's zero-length slot, which has no record)
    std::vector<int32_t> record(4 * (size_t)h->C, -1);
    for (int r = 0; r < nrec; r++) {
        record[rix[r].z] = r;
        if (rix[r].w >= 0) record[rix[r].w] = -2 - r;
    }
    // the CTAs' runs of cells
    std::vector<int4> seg;
    int4 cur = make_int4(0, 0, 0, 0);
    for (int c = 0; c < h->C; c++) {
        int n = 0;
        for (int j = 0; j < 4; j++) n += record[4 * (size_t)c + j] != -1;
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
    // A CTA's boundary slots, the slowest ones, come last, so that they share
    // as few warps as possible with the others.
    std::vector<double> table;
    table.reserve(4 * (size_t)(cur.z + cur.w) + 2 * seg.size());
    for (const int4 &d : seg)
        for (int boundary = 0; boundary < 2; boundary++)
            for (int place = 0; place < 4 * d.y; place++) {
                const int q = record[4 * (size_t)d.x + place];
                if (q == -1) continue;
                const bool other = q < 0;
                const int r = other ? -2 - q : q;
                // a pair's other slot: negated normal, same length, not the lower-numbered side
                const uint8_t meta = other ? (uint8_t)(hb::CODE_ZERO | hb::META_HAS_NB) : rmeta[r];
                if (boundary != ((meta & hb::META_CODE) != hb::CODE_ZERO)) continue;
                const double *g = &rgeo[4 * (size_t)r];
                const uint64_t w = hb::SlotRef::pack(other ? rix[r].x : rix[r].y, place, meta, r);
                double v;
                memcpy(&v, &w, sizeof v);
                table.insert(table.end(), {other ? -g[0] : g[0], other ? -g[1] : g[1], g[2], v});
            }
    const size_t records = table.size();
    table.resize(records + 2 * seg.size());
    memcpy(table.data() + records, seg.data(), seg.size() * sizeof(int4));
    double *sp;
    TRY(dev_upload(h, &sp, table));
    const int4 *cp = reinterpret_cast<const int4 *>(sp + records);
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
