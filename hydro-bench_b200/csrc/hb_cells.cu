// hb_cells.cu -- the one-launch step of small fp64 meshes (cell_kernel): when
// it is used, its slot table, and its launches.
#include <cstring>
#include <vector>

#include "hb_handle.hpp"

namespace {

// The one-launch step takes single fp64 meshes of at most this many cells (edge
// layout, default launch shape).  It halves the latencies of a step but
// computes every edge twice.  us per step on a B200, 40- or 100-step graphs,
// one launch / two kernels, variant H:
//   cells      6,675      24,021     60,000      100,000      120,000      140,000
//   channel   4.3 / 8.4  5.0 / 9.1  8.6 / 12.4  13.7 / 14.6  14.7 / 15.7  17.6 / 17.1
//   mixed     4.4 / 8.8  5.6 / 9.9  10.4/ 13.6  14.6 / 15.4  16.8 / 17.3  19.0 / 17.9
//   dam break 5.3*/ 9.5  5.6 / 10.5 8.5 / 15.0  11.6 / 16.1  12.7 / 17.9  15.3 / 19.2
// (* before the update warp.)  The line lies where channels and mixed meshes cross.
constexpr int CELLS_MAX = 120000;

template <int VARIANT, bool COEF>
int launch_cells_t(int ncseg, const hb::DevMesh<hb::F64Exact> &m, int k0, int n, int write_last, cudaStream_t st) {
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
                                       (int)(write_last && k == n - 1)));
    return HB_OK;
}

}  // namespace

bool hb_cells_used(const hb_handle *h) {
    return h->ncseg > 0 && h->launch_config == hb::DEFAULT_EDGE_CONFIG;
}

int hb_cells_build(hb_handle *h, const std::vector<int4> &rix, const std::vector<uint8_t> &rmeta,
                   const std::vector<double> &rgeo) {
    if (h->opt.precision != HB_FP64 || h->opt.layout != HB_LAYOUT_EDGE || h->opt.persistent || h->segmented() ||
        h->C > CELLS_MAX)
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
    // one allocation: the slot records (32-byte aligned), then the CTAs' entries
    std::vector<double> table;
    table.reserve(18 * (size_t)h->C + 64);
    std::vector<int4> seg;
    int4 cur = make_int4(0, 0, 0, 0);
    for (int c = 0; c < h->C; c++) {
        int n = 0;
        for (int j = 0; j < 4; j++) n += record[4 * (size_t)c + j] != -1;
        if (cur.w + n > hb::CELL_SLOTS || cur.y == hb::CELL_MAX) {
            seg.push_back(cur);
            cur = make_int4(c, 0, cur.z + cur.w, 0);
        }
        for (int j = 0; j < 4; j++) {
            const int q = record[4 * (size_t)c + j];
            if (q == -1) continue;
            const bool other = q < 0;
            const int r = other ? -2 - q : q;
            // a pair's other slot: negated normal, same length, not the lower-numbered side
            const double *g = &rgeo[4 * (size_t)r];
            const uint64_t w = hb::SlotRef::pack(other ? rix[r].x : rix[r].y, 4 * cur.y + j,
                                                 other ? (uint8_t)(hb::CODE_ZERO | hb::META_HAS_NB) : rmeta[r], r);
            double d;
            memcpy(&d, &w, sizeof d);
            table.insert(table.end(), {other ? -g[0] : g[0], other ? -g[1] : g[1], g[2], d});
        }
        cur.y++;
        cur.w += n;
    }
    seg.push_back(cur);
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

int hb_cells_launch(hb_handle *h, const hb::DevMesh<hb::F64Exact> &m, int k0, int n, int write_last, bool coef,
                    cudaStream_t st) {
    if (h->opt.variant == HB_VARIANT_F) {
        if (coef) return hb::set_error(HB_E_INVALID, "update coefficients: variant H only");
        return launch_cells_t<1, false>(h->ncseg, m, k0, n, write_last, st);
    }
    return coef ? launch_cells_t<0, true>(h->ncseg, m, k0, n, write_last, st) : launch_cells_t<0, false>(h->ncseg, m, k0, n, write_last, st);
}
