// modal_batch.cu -- the modal stencil kernel over the instances of a batch: one launch per
// degree, one tile of one instance per CTA. Batches whose instances are all linear with constant
// coefficients (modal_applies) run here; others keep the quadrature tiles of batch.cu.
#include "modal_batch.h"

#include <algorithm>

#include "handle.h"
#include "modal_kernel.cuh"

namespace bosss {

struct ModalInst {
    EvalArgs a;
    ModalTile tl;
    long long dom_off, cod_off;
};

namespace {

template <int K, bool SIP, int MODE>
__global__ void __launch_bounds__(ModalCfg<3, K>::NT, ModalCfg<3, K>::MINB)
k_modal_batch(const __grid_constant__ Tables1D tab, const ModalInst* __restrict__ inst, const ModalItem* __restrict__ items, const double* U, const double* V,
              double* out, double alpha, double beta) {
    extern __shared__ double smem[];
    __shared__ ModalInst si;
    const ModalItem w = items[blockIdx.x];
    static_assert(sizeof(ModalInst) % 8 == 0, "copied as doubles");
    for (int i = threadIdx.x; i < (int)(sizeof(ModalInst) / 8); i += ModalCfg<3, K>::NT)
        reinterpret_cast<double*>(&si)[i] = reinterpret_cast<const double*>(inst + w.inst)[i];
    __syncthreads();
    const double* in = MODE == MODE_RES ? U + si.dom_off : V + (MODE == MODE_VJP ? si.cod_off : si.dom_off);
    double* o = out + (MODE == MODE_VJP ? si.dom_off : si.cod_off);
    modal_tile<3, K, SIP, MODE, false>(si.a, tab, si.tl, w.tile, in, o, alpha, beta, smem);
}

template <int K, bool SIP, int MODE>
cudaError_t launch_one(const Tables1D& tab, const ModalInst* inst, const ModalItem* items, int n, const double* U, const double* V,
                       double* out, double alpha, double beta, cudaStream_t s) {
    static unsigned long long done = 0ull;
    const size_t smem = ModalCfg<3, K>::SMEM;
    cudaError_t e = modal_attr(k_modal_batch<K, SIP, MODE>, smem, done);
    if (e != cudaSuccess || n <= 0) return e;
    k_modal_batch<K, SIP, MODE><<<n, ModalCfg<3, K>::NT, smem, s>>>(tab, inst, items, U, V, out, alpha, beta);
    return cudaGetLastError();
}

template <int K, bool SIP>
cudaError_t launch_mode(int mode, const Tables1D& tab, const ModalInst* inst, const ModalItem* items, int n, const double* U, const double* V,
                        double* out, double alpha, double beta, cudaStream_t s) {
    if (mode == MODE_RES) return launch_one<K, SIP, MODE_RES>(tab, inst, items, n, U, V, out, alpha, beta, s);
    if (mode == MODE_JVP) return launch_one<K, SIP, MODE_JVP>(tab, inst, items, n, U, V, out, alpha, beta, s);
    return launch_one<K, SIP, MODE_VJP>(tab, inst, items, n, U, V, out, alpha, beta, s);
}

template <bool SIP>
cudaError_t launch_degree(int K, int mode, const Tables1D& tab, const ModalInst* inst, const ModalItem* items, int n, const double* U,
                          const double* V, double* out, double alpha, double beta, cudaStream_t s) {
    switch (K) {
        case 1: return launch_mode<1, SIP>(mode, tab, inst, items, n, U, V, out, alpha, beta, s);
        case 2: return launch_mode<2, SIP>(mode, tab, inst, items, n, U, V, out, alpha, beta, s);
        case 3: return launch_mode<3, SIP>(mode, tab, inst, items, n, U, V, out, alpha, beta, s);
        default: return launch_mode<4, SIP>(mode, tab, inst, items, n, U, V, out, alpha, beta, s);
    }
}

}  // namespace

struct ModalBatch {
    struct Run {
        int K, first, count;
        Tables1D tab;   // of any instance of the degree (L_m(1), L_m'(1) depend on it alone)
    };
    bool sip = false;
    std::vector<Run> runs;   // highest degree first
    ModalInst* d_inst = nullptr;
    ModalItem* d_items = nullptr;
};

void modal_batch_destroy(ModalBatch* m) {
    if (!m) return;
    cudaFree(m->d_inst);
    cudaFree(m->d_items);
    delete m;
}

int modal_batch_create(const std::vector<bosss_handle*>& hs, const long long* dom_off, const long long* cod_off,
                       ModalBatch** out) {
    *out = nullptr;
    for (const bosss_handle* h : hs)
        if (h->D != 3 || h->K < 1 || h->K > 4 || !modal_applies(h->phys, h->base.ph, h->K, h->Q)) return BOSSS_OK;
    ModalBatch* m = new ModalBatch();
    m->sip = hs[0]->phys == PHYS_SIP;
    std::vector<ModalInst> inst(hs.size());
    std::vector<ModalItem> items;
    for (size_t i = 0; i < hs.size(); ++i) {
        inst[i].a = hs[i]->base;
        inst[i].tl = modal_tiling(hs[i]->base, 3, hs[i]->K, hs.size() > 1);
        inst[i].dom_off = dom_off[i];
        inst[i].cod_off = cod_off[i];
    }
    for (int K = 4; K >= 1; --K) {
        ModalBatch::Run r{K, (int)items.size(), 0, Tables1D{}};
        for (size_t i = 0; i < hs.size(); ++i) {
            if (hs[i]->K != K) continue;
            r.tab = hs[i]->base.tab;
            const ModalTile& t = inst[i].tl;
            for (int k = 0; k < t.t[0] * t.t[1] * t.t[2]; ++k) items.push_back(ModalItem{(int)i, k});
        }
        r.count = (int)items.size() - r.first;
        if (r.count > 0) m->runs.push_back(r);
    }
    cudaError_t e = cudaMalloc(&m->d_inst, sizeof(ModalInst) * inst.size());
    if (e == cudaSuccess) e = cudaMalloc(&m->d_items, sizeof(ModalItem) * items.size());
    if (e == cudaSuccess) e = cudaMemcpy(m->d_inst, inst.data(), sizeof(ModalInst) * inst.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->d_items, items.data(), sizeof(ModalItem) * items.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        modal_batch_destroy(m);
        return fail(BOSSS_ERR_CUDA, std::string("batch setup: ") + cudaGetErrorString(e));
    }
    *out = m;
    return BOSSS_OK;
}

int modal_batch_run(const ModalBatch* m, int mode, double alpha, double beta, const double* U, const double* V,
                    double* out, cudaStream_t s) {
    for (const auto& r : m->runs)
        CUDA_TRY(m->sip ? launch_degree<true>(r.K, mode, r.tab, m->d_inst, m->d_items + r.first, r.count, U, V, out, alpha, beta, s)
                        : launch_degree<false>(r.K, mode, r.tab, m->d_inst, m->d_items + r.first, r.count, U, V, out, alpha, beta, s));
    return BOSSS_OK;
}

}  // namespace bosss
