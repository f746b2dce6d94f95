// bsg_grad: Hellmann-Feynman gradient of eigenvalues with respect to every
// uncoupled matrix element (the transposed-jump contraction of the two-body
// densities, src/bdenslib4.f90:129-729; the tile body is grad_tile.cuh).
//
// One launch covers every (system, states, row tile) item and one the NN
// operators' (system, state, rows) items: bsg_grad is the one-system case of
// grad_many, bsg_batch_grad (batch.cu) the many-system one.  Sums are 128-bit
// fixed point updated with integer atomics, each addend formed the same way
// however many systems and states there are, so the gradient is bitwise
// repeatable and a system's is the same alone or inside a batch.

#include <algorithm>
#include <string>
#include <vector>

#include "grad_tile.cuh"

namespace bsg {

struct GradDesc {
    RowArgs a;
    GradArgs g;
    const double *psi;
    int64_t dim, gstride;   // to the next state's vector and accumulators
};
struct GradItem {
    int32_t desc;   // (system, first state)
    int32_t tile;
};
// kGradNNRows rows (fewer at an operator's end) of one NN operator
struct GradNNItem {
    int32_t desc;   // (system, state)
    int32_t nop;
    int32_t at, n;  // its rows: rows[at .. at + n)
};

__global__ void k_fix_to_double(const unsigned long long *__restrict__ acc, double *__restrict__ out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = fix_value(acc + 2 * i);
}

// [n x ns] row-major -> n rows of columns ld apart; a warp takes 32 states, whose
// lines stay in L1 between the columns
__global__ void k_rows_to_cols(const double *__restrict__ x, int64_t n, int ns, double *__restrict__ y, int64_t ld) {
    const int lane = threadIdx.x & 31;
    for (int64_t r = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32 + lane; r < n;
         r += (int64_t)gridDim.x * blockDim.x)
        for (int k = 0; k < ns; ++k) y[(int64_t)k * ld + r] = __ldg(x + r * ns + k);
}

// three CTAs to an SM: at 128 registers (two) five states of sd 6p6n took 1.72 ms
// through the whole call, at 80 with some spills 1.57
template <int ITEMS, int NS>
__global__ void __launch_bounds__(kGradWarps * 32, 3) k_grad_items(const GradDesc *__restrict__ desc,
                                                                const GradItem *__restrict__ items, int mstride) {
    double *Aw, *stage;
    grad_smem(mstride, NS, Aw, stage);
    const GradItem it = items[blockIdx.x];
    const GradDesc *D = desc + it.desc;
    grad_tile<ITEMS, NS>(D->a, D->g, D->psi, D->dim, D->gstride, D->a.tiles[it.tile], Aw, mstride, stage);
}

// NN: dnn[op_r] += ph_r * sum over the item's rows of psi[row+pos] psi[row+in_r],
// a warp per 32 output positions.  An operator's records are the same in every
// row that has it, so each is read once for kGradNNRows rows and its label is
// updated once, not once a row: the updates (two atomics on one of a few hundred
// labels for each matrix element) were 0.8 ms of the 1.32 ms of a call for one
// state of sd 6p6n, now 0.59.  What is left is the gathers, kGradNNRows in flight.
constexpr int kGradNNRows = 16;
__global__ void __launch_bounds__(kGradWarps * 32) k_grad_nn(const GradDesc *__restrict__ desc,
                                                             const GradNNItem *__restrict__ items,
                                                             const int32_t *__restrict__ rows) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const GradNNItem it = items[blockIdx.x];
    const GradDesc *D = desc + it.desc;
    const RowArgs &a = D->a;
    const GradArgs &g = D->g;
    const double *__restrict__ psi = D->psi;
    const NOp op = a.nops[it.nop];
    const int32_t *__restrict__ ptr = a.nptr + op.ptr_base;
    __shared__ int64_t off[kGradNNRows];
    if (threadIdx.x < kGradNNRows) off[threadIdx.x] = a.row_off[rows[it.at + min((int)threadIdx.x, it.n - 1)]];
    __syncthreads();
    for (int pos = warp * 32 + lane; pos < op.nout; pos += kGradWarps * 32) {
        const int k0 = ptr[pos], k1 = ptr[pos + 1];
        double pout[kGradNNRows];
#pragma unroll
        for (int r = 0; r < kGradNNRows; ++r) pout[r] = r < it.n ? psi[off[r] + pos] : 0.0;
        for (int k = k0; k < k1; ++k) {
            const int64_t rec = op.rec_base + k;
            const double *__restrict__ in = psi + a.nnrec[rec].in;
            double v[2] = {0.0, 0.0};
#pragma unroll
            for (int r = 0; r < kGradNNRows; ++r)
                if (r < it.n) v[r & 1] += pout[r] * in[off[r]];
            fix_add(g.nn + 2 * (size_t)(g.nnrec_op[rec] - 1), (double)g.nnrec_ph[rec] * (v[0] + v[1]));
        }
    }
}

namespace {
constexpr int kGradItems = 4;  // 128-position tiles
// states in one pass over the records, at most.  Whole calls with at most 3, 4 and 5:
// pf 3p4n five states 10.4, 10.6, 9.3 ms, ten 20.1, 19.2, 17.8, twelve 22.9, 22.0, 22.0;
// pf 3p3n five 2.53, 2.51, 2.31, ten 4.46, 4.39, 4.18; sd 6p6n five 1.69, 1.70, 1.57,
// ten 3.03, 2.93, 2.81, eight 2.48, 2.33, 2.31; sd 5p5n five 1.31, 1.31, 1.21.  For 1,
// 2, 3, 6 and 8 states 4 and 5 give the same groups or times within 2 %.
constexpr int kGradStates = 5;
// no more shared memory than leaves two CTAs on an SM
constexpr size_t kGradSmem = 113 * 1024;
// and enough CTAs for the chip: of a small system each state has its own
constexpr int64_t kGradCtas = 148 * 4;
// row-major states on their way to columns: 64 MB at a time
constexpr int64_t kGradPiece = (int64_t)8 << 20;

template <int NS>
cudaError_t launch_items(const DevBuf &descb, const GradItem *items, size_t n, int mstride, cudaStream_t s) {
    const size_t smem = grad_smem_bytes(mstride, NS);
    cudaError_t e = cudaFuncSetAttribute(k_grad_items<kGradItems, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    k_grad_items<kGradItems, NS><<<(unsigned)n, kGradWarps * 32, smem, s>>>((const GradDesc *)descb.p, items, mstride);
    return cudaGetLastError();
}
}  // namespace

int grad_many(bsg_ctx *const *ctxs, int nsys, const double *const *evecs, int nstates, double *const *dpp,
              double *const *dnn, double *const *dpn, double *const *dspe_p, double *const *dspe_n, cudaStream_t s,
              std::string &err, double *kernel_ms, bool rows) {
    auto fail = [&](int code, const std::string &m) {
        err = m;
        return code;
    };
    if (nsys < 1 || nstates < 1 || !evecs || !dpp || !dnn || !dpn) return fail(BSG_ERR_ARG, "null argument");
    for (int i = 0; i < nsys; ++i)
        if (ctxs[i]->threebody)
            return fail(BSG_ERR_UNSUPPORTED, "the adjoint covers two-body contexts only (hmatpp, hmatnn, hmatpn)");
    // per (system, state): psi offset, accumulator offsets; per system: sizes
    std::vector<int64_t> psi_off(nsys), acc_off((size_t)nsys * nstates);
    std::vector<int64_t> nlab(nsys);
    int64_t npsi = 0, nacc = 0;
    int32_t max_nbd = 0;
    std::vector<const TileSet *> ts(nsys);
    int64_t ntiles = 0;
    for (int s2 = 0; s2 < nsys; ++s2) {
        bsg_ctx *c = ctxs[s2];
        if (!evecs[s2] || !dpp[s2] || !dnn[s2] || !dpn[s2]) return fail(BSG_ERR_ARG, "null output for a system");
        const bool spe = c->t.call_spe && dspe_p && dspe_n && dspe_p[s2] && dspe_n[s2];
        c->last_status = BSG_OK;
        ts[s2] = get_tiles(c, 32 * kGradItems);
        if (!ts[s2]) return fail(c->last_status ? c->last_status : BSG_ERR_NOMEM, "tiles: " + c->last_error);
        max_nbd = std::max(max_nbd, c->args.max_nbd);
        ntiles += ts[s2]->ntiles;
        psi_off[s2] = npsi;
        npsi += c->dim * nstates;
        nlab[s2] = c->t.nmatpp + c->t.nmatnn + c->t.nmatpn + (spe ? c->t.nsd_p + c->t.nsd_n : 0);
        for (int k = 0; k < nstates; ++k) {
            acc_off[(size_t)s2 * nstates + k] = nacc;
            nacc += nlab[s2];
        }
    }
    // 8 per-warp FP64 bin tables and staging within 227 KB of shared memory
    if (max_nbd > 3392) return fail(BSG_ERR_UNSUPPORTED, "a neutron sector jump has more than 3392 distinct (b,d) pairs");
    const int mstride = (max_nbd + 1) & ~1;
    // the states of a system in groups of about the same size, at most ng in one
    int ng = std::min(nstates, kGradStates);
    while (ng > 1 && (grad_smem_bytes(mstride, ng) > kGradSmem || ntiles * ((nstates + ng - 1) / ng) < kGradCtas)) --ng;
    const int ngroups = (nstates + ng - 1) / ng;
    // items by group size (two sizes at most), heaviest tiles first (the tile
    // lists are already in that order per system); the groups of a tile next to
    // each other, so that concurrent CTAs share records
    std::vector<GradItem> items[kGradStates + 1];
    for (int s2 = 0; s2 < nsys; ++s2)
        for (int t = 0; t < ts[s2]->ntiles; ++t)
            for (int q = 0; q < ngroups; ++q) {
                const int k0 = nstates * q / ngroups, k1 = nstates * (q + 1) / ngroups;
                items[k1 - k0].push_back(GradItem{s2 * nstates + k0, t});
            }
    // per system the rows of each NN operator, cut into items
    std::vector<GradNNItem> nnitems;
    std::vector<int32_t> nnrows;
    for (int s2 = 0; s2 < nsys; ++s2) {
        const bsg_ctx *c = ctxs[s2];
        const size_t base = nnrows.size(), cnt = c->h_nn.size();
        if (base + cnt > INT32_MAX) return fail(BSG_ERR_UNSUPPORTED, "more than 2^31 rows of NN operators");
        nnrows.resize(base + cnt);
        int32_t nops = 0;
        for (const NNContrib &x : c->h_nn) nops = std::max(nops, x.nop + 1);
        std::vector<int32_t> at((size_t)nops + 1, 0);
        for (const NNContrib &x : c->h_nn) ++at[x.nop + 1];
        for (int32_t o = 0; o < nops; ++o) {
            for (int32_t b = 0; b < at[o + 1]; b += kGradNNRows)
                for (int k = 0; k < nstates; ++k)
                    nnitems.push_back(GradNNItem{s2 * nstates + k, o, (int32_t)base + at[o] + b,
                                                 std::min(kGradNNRows, at[o + 1] - b)});
            at[o + 1] += at[o];
        }
        for (int64_t slot = 0; slot + 1 < (int64_t)c->h_nn_ptr.size(); ++slot)
            for (int32_t x = c->h_nn_ptr[slot]; x < c->h_nn_ptr[slot + 1]; ++x)
                nnrows[base + at[c->h_nn[x].nop]++] = (int32_t)(slot / kRowWarps);
    }
    bsg_ctx *c0 = ctxs[0];
    DevBuf psi, tmp, acc, out, descb, itemb, nnb, nnrb;
    auto cleanup = [&]() { pool_free(c0, {&psi, &tmp, &acc, &out, &descb, &itemb, &nnb, &nnrb}, s); };
    int st;
    if (nstates == 1) rows = false;   // the same layout
    // row-major states come in so many basis states at a time, so that they do
    // not lie on the device twice
    const int64_t piece = std::max<int64_t>(1, kGradPiece / nstates);
    int64_t maxdim = 0;
    for (int s2 = 0; s2 < nsys; ++s2) maxdim = std::max(maxdim, ctxs[s2]->dim);
    if ((st = pool_alloc(c0, psi, sizeof(double) * (size_t)npsi, s)) ||
        (rows && (st = pool_alloc(c0, tmp, sizeof(double) * (size_t)(std::min(piece, maxdim) * nstates), s))) ||
        (st = pool_alloc(c0, acc, 16 * (size_t)nacc, s)) || (st = pool_alloc(c0, out, sizeof(double) * (size_t)nacc, s))) {
        cleanup();
        return fail(st, "device allocation: " + c0->last_error);
    }
    std::vector<GradDesc> desc((size_t)nsys * nstates);
    for (int s2 = 0; s2 < nsys; ++s2) {
        bsg_ctx *c = ctxs[s2];
        const bool spe = c->t.call_spe && dspe_p && dspe_n && dspe_p[s2] && dspe_n[s2];
        for (int k = 0; k < nstates; ++k) {
            GradDesc &d = desc[(size_t)s2 * nstates + k];
            d.a = c->args;
            d.a.tiles = (const Tile *)ts[s2]->buf.p;
            d.a.ntiles = ts[s2]->ntiles;
            unsigned long long *base = (unsigned long long *)acc.p + 2 * acc_off[(size_t)s2 * nstates + k];
            d.g.pp_op = (const int32_t *)c->pp_op.p;
            d.g.pp_ph = (const int8_t *)c->pp_ph.p;
            d.g.nnrec_op = (const int32_t *)c->nnrec_op.p;
            d.g.nnrec_ph = (const int8_t *)c->nnrec_ph.p;
            d.g.pp = base;
            d.g.nn = d.g.pp + 2 * c->t.nmatpp;
            d.g.pn = d.g.nn + 2 * c->t.nmatnn;
            d.g.spe_p = spe ? d.g.pn + 2 * c->t.nmatpn : nullptr;
            d.g.spe_n = spe ? d.g.spe_p + 2 * c->t.nsd_p : nullptr;
            d.psi = (const double *)psi.p + psi_off[s2] + (int64_t)k * c->dim;
            d.dim = c->dim;
            d.gstride = 2 * nlab[s2];
        }
    }
    std::vector<GradItem> all;
    for (const auto &v : items) all.insert(all.end(), v.begin(), v.end());
    if ((st = pool_upload(c0, descb, desc.data(), sizeof(GradDesc) * desc.size(), s)) ||
        (st = pool_upload(c0, itemb, all.data(), sizeof(GradItem) * all.size(), s)) ||
        (st = pool_upload(c0, nnb, nnitems.data(), sizeof(GradNNItem) * nnitems.size(), s)) ||
        (st = pool_upload(c0, nnrb, nnrows.data(), sizeof(int32_t) * nnrows.size(), s))) {
        cleanup();
        return fail(st, "upload: " + c0->last_error);
    }
    cudaError_t e = cudaSuccess;
    for (int s2 = 0; s2 < nsys && e == cudaSuccess; ++s2) {
        const int64_t dim = ctxs[s2]->dim;
        double *to = (double *)psi.p + psi_off[s2];
        if (!rows) e = cudaMemcpyAsync(to, evecs[s2], sizeof(double) * dim * nstates, cudaMemcpyHostToDevice, s);
        for (int64_t r = 0; rows && r < dim && e == cudaSuccess; r += piece) {
            const int64_t n = std::min(piece, dim - r);
            e = cudaMemcpyAsync(tmp.p, evecs[s2] + r * nstates, sizeof(double) * n * nstates, cudaMemcpyHostToDevice, s);
            if (e != cudaSuccess) break;
            k_rows_to_cols<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(
                (const double *)tmp.p, n, nstates, to + r, dim);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(acc.p, 0, acc.bytes, s);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    const GradItem *ip = (const GradItem *)itemb.p;
    for (int n = 1; n <= kGradStates; ++n) {
        const size_t cnt = items[n].size();
        if (e == cudaSuccess && cnt) switch (n) {
            case 1: e = launch_items<1>(descb, ip, cnt, mstride, s); break;
            case 2: e = launch_items<2>(descb, ip, cnt, mstride, s); break;
            case 3: e = launch_items<3>(descb, ip, cnt, mstride, s); break;
            case 4: e = launch_items<4>(descb, ip, cnt, mstride, s); break;
            default: e = launch_items<5>(descb, ip, cnt, mstride, s);
            }
        ip += cnt;
    }
    if (e == cudaSuccess && !nnitems.empty()) {
        k_grad_nn<<<(unsigned)nnitems.size(), kGradWarps * 32, 0, s>>>((const GradDesc *)descb.p,
                                                                       (const GradNNItem *)nnb.p, (const int32_t *)nnrb.p);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && nacc > 0) {
        k_fix_to_double<<<(unsigned)std::min<int64_t>((nacc + 255) / 256, 4096), 256, 0, s>>>(
            (const unsigned long long *)acc.p, (double *)out.p, nacc);
        e = cudaGetLastError();
    }
    cudaEventRecord(e1, s);
    // one copy back, then per system state-major blocks [state][label]
    std::vector<double> host((size_t)nacc);
    if (e == cudaSuccess && nacc > 0)
        e = cudaMemcpyAsync(host.data(), out.p, sizeof(double) * (size_t)nacc, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    for (int s2 = 0; s2 < nsys && e == cudaSuccess; ++s2) {
        bsg_ctx *c = ctxs[s2];
        const bool spe = c->t.call_spe && dspe_p && dspe_n && dspe_p[s2] && dspe_n[s2];
        for (int k = 0; k < nstates; ++k) {
            const double *o = host.data() + acc_off[(size_t)s2 * nstates + k];
            auto cp = [&](double *dst, int64_t cnt) {
                std::copy(o, o + cnt, dst);
                o += cnt;
            };
            cp(dpp[s2] + k * c->t.nmatpp, c->t.nmatpp);
            cp(dnn[s2] + k * c->t.nmatnn, c->t.nmatnn);
            cp(dpn[s2] + k * c->t.nmatpn, c->t.nmatpn);
            if (spe) {
                cp(dspe_p[s2] + k * c->t.nsd_p, c->t.nsd_p);
                cp(dspe_n[s2] + k * c->t.nsd_n, c->t.nsd_n);
            }
        }
    }
    if (kernel_ms && e == cudaSuccess) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        *kernel_ms = ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cleanup();
    if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? BSG_ERR_NOMEM : BSG_ERR_CUDA,
                                      std::string("adjoint: ") + cudaGetErrorString(e));
    return BSG_OK;
}

}  // namespace bsg

using namespace bsg;

static int grad_one(bsg_ctx *ctx, const double *evecs, int nstates, double *dpp, double *dnn, double *dpn, double *dspe_p,
                    double *dspe_n, bool rows) {
    if (!ctx) return BSG_ERR_ARG;
    if (!evecs || nstates < 1 || !dpp || !dnn || !dpn)
        return set_err(ctx, BSG_ERR_ARG, "bsg_grad: null argument or nstates < 1");
    int st = cuda_check(ctx, cudaSetDevice(ctx->device), "cudaSetDevice");
    if (st) return st;
    bsg_ctx *cs[1] = {ctx};
    const double *ev[1] = {evecs};
    double *p[1] = {dpp}, *nn[1] = {dnn}, *pn[1] = {dpn}, *sp[1] = {dspe_p}, *sn[1] = {dspe_n};
    std::string err;
    double ms = 0.0;
    st = grad_many(cs, 1, ev, nstates, p, nn, pn, sp, sn, ctx->stream, err, &ms, rows);
    if (st) return set_err(ctx, st, "bsg_grad: " + err);
    ctx->stats.grad_ms = ms;
    return BSG_OK;
}

extern "C" int bsg_grad(bsg_ctx *ctx, const double *evecs, int nstates, double *dpp, double *dnn, double *dpn,
                        double *dspe_p, double *dspe_n) {
    return grad_one(ctx, evecs, nstates, dpp, dnn, dpn, dspe_p, dspe_n, false);
}

extern "C" int bsg_grad_rows(bsg_ctx *ctx, const double *evecs, int nstates, double *dpp, double *dnn, double *dpn,
                             double *dspe_p, double *dspe_n) {
    return grad_one(ctx, evecs, nstates, dpp, dnn, dpn, dspe_p, dspe_n, true);
}
