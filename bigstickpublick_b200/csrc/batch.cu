// Batched Hamiltonians: many independent systems of uneven dimension.
//
// bsg_batch_applyh  the systems with jump groups in one launch, one CTA per
//                   (system, row), heaviest first, with the single-system row
//                   body (rowgroup.cuh); the others in one persistent launch:
//                   CTAs pull (system, row tile) work items, heaviest first,
//                   from an atomic counter, with the single-system tile body
//                   (applyh_tile.cuh).  No device-side waits.
// bsg_batch_lanczos lock-step scalar Lanczos over all systems in the
//                   reference's order: alpha and W -= alpha v_i first, then
//                   one classical Gram-Schmidt pass against the earlier
//                   history, with the reference's beta safeguards (second
//                   full pass, random restart) decided per system on the
//                   device.  Every kernel of one iteration reads the
//                   iteration index from device memory, so the iteration is
//                   captured once as a CUDA graph and replayed.  Afterwards
//                   the projected tridiagonal matrices are solved on the
//                   device (bisection + inverse iteration) and the Ritz
//                   vectors formed.
//
// The reference runs one Hamiltonian per process; its Lanczos is lanczos_p
// (src/blanczosmain.f90:1413-1793) with the matvec of
// src/bapplyhlibOMP.f90:882.  Systems are independent: no cross-system
// communication of any kind.

#include <algorithm>
#include <thread>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <numeric>
#include <type_traits>
#include <vector>

#include "rowgroup.cuh"
#include "lanczos_kernels.h"
#include "rowgroup.h"

namespace bsg {

struct BatchSys {
    RowArgs a;
    GroupArgs g;        // grouped contexts, with their shared-memory layout
    int32_t parts[2], accel[2], bufel[2];
};
// a system's vectors in one call.  The descriptors above are written when the
// batch's items are built and only read by the launches; what differs from call
// to call lies in that call's own table, so that calls on several streams or
// host threads do not meet.
struct BatchVec {
    const void *vin;
    void *vout;
};
// device table of a call: the persistent kernel's work counter, then the vectors
constexpr size_t kBatchVecOff = 16;
// a batch keeps this many tables: so many calls may be in flight before one
// waits (on its stream) for the launches of an earlier call
constexpr int kBatchTables = 8;
struct BatchItem {
    int32_t sys;
    int32_t tile;
};
// Lanczos bookkeeping per system (device)
struct BLz {
    int64_t dim;
    int64_t off;        // offset of the system in the concatenated vectors
    double *hist;       // (niter+1) columns of dim
    double *partial;    // (niter+1) x nch dot partials
    double *coef;       // niter+1 Gram-Schmidt coefficients
    double *sqp;        // nch norm partials
    double *alpha, *beta;  // niter each
    double *nrm2;       // norm after the second pass (1 entry)
    int32_t *flag;      // bit 0: second pass, bit 1: random restart
    int32_t nch, pad;
};
struct BChunk {
    int32_t sys, local;
    int32_t row0, len;
};

constexpr int kChunk = 2048;

template <typename T, int ITEMS, bool SACC = false>
__device__ __forceinline__ void rows_batch_body(const BatchSys *__restrict__ sys, const BatchVec *__restrict__ vec,
                                                const BatchItem *__restrict__ items, int nitems,
                                                int *__restrict__ counter, int mstride) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_item;
    const int warp = threadIdx.x >> 5;
    float *__restrict__ Mw = reinterpret_cast<float *>(smem) + (size_t)warp * mstride;
    T *__restrict__ part = reinterpret_cast<T *>(smem + align16(sizeof(float) * (size_t)kWarps * mstride));
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int it = s_item;
        __syncthreads();
        if (it >= nitems) return;
        const BatchItem w = items[it];
        const BatchSys *S = sys + w.sys;
        row_tile<T, 1, ITEMS, false, kStore, false, SACC>(S->a, S->a.tiles[w.tile], (const T *)vec[w.sys].vin,
                                                          (T *)vec[w.sys].vout, 1, 0, Mw, part);
        __syncthreads();
    }
}

template <typename T, int ITEMS>
__global__ void __launch_bounds__(kWarps * 32) k_rows_batch(const BatchSys *__restrict__ sys,
                                                            const BatchVec *__restrict__ vec,
                                                            const BatchItem *__restrict__ items, int nitems,
                                                            int *__restrict__ counter, int mstride) {
    rows_batch_body<T, ITEMS>(sys, vec, items, nitems, counter, mstride);
}

// FP32: capped at 40 registers so that 6 CTAs of 256 threads stay resident
// per SM; the system descriptors come from global memory, and the compiler's
// own choice (64 registers, 4 CTAs) was measured slower than the spills the
// cap costs.  From 2 items per lane up the running sums stay in shared memory
// during the record walks (row_tile's SACC): spill loads of the 4-item kernel
// 180 -> 112 bytes, the 256-system matvec 5.98 -> 5.79 ms, bitwise the same.
// With 4 or 8 items the cap is 32 registers (8 CTAs per SM), as for the
// single-system kernel: more spills, but at the autotuned 4 items x 8 CTAs
// 5.75 -> 5.63 ms (the 4-CTA grid settings got slower; the autotuner does not
// pick them).
template <int ITEMS>
__global__ void __launch_bounds__(kWarps * 32, ITEMS >= 4 ? 8 : 6) k_rows_batch_f32(const BatchSys *__restrict__ sys,
                                                                   const BatchVec *__restrict__ vec,
                                                                   const BatchItem *__restrict__ items, int nitems,
                                                                   int *__restrict__ counter, int mstride) {
    rows_batch_body<float, ITEMS, (ITEMS >= 2)>(sys, vec, items, nitems, counter, mstride);
}

// grouped contexts: one CTA per (system, row), heaviest first; the system's
// descriptor is staged in shared memory
template <typename T>
__global__ void __launch_bounds__(256, 4) k_rowgroup_batch(const BatchSys *__restrict__ sys,
                                                            const BatchVec *__restrict__ vec,
                                                            const BatchItem *__restrict__ items) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ BatchSys S;
    const BatchItem w = items[blockIdx.x];
    for (int k = threadIdx.x; k < (int)(sizeof(BatchSys) / 4); k += blockDim.x)
        reinterpret_cast<int *>(&S)[k] = reinterpret_cast<const int *>(sys + w.sys)[k];
    __syncthreads();
    const Tile t = S.a.tiles[w.tile];
    constexpr int P = sizeof(T) == 8 ? 1 : 0;
    row_group<T, 1, kStore>(S.a, S.g, S.parts[P], t.row, t.npos, (const T *)vec[w.sys].vin, 1, (T *)vec[w.sys].vout,
                            nullptr, reinterpret_cast<T *>(smem), S.accel[P], S.bufel[P]);
}

template <typename T, int ITEMS>
constexpr auto batch_rows_kernel() {
    if constexpr (std::is_same<T, float>::value)
        return k_rows_batch_f32<ITEMS>;
    else
        return k_rows_batch<T, ITEMS>;
}

// Y[j*nk + l] = Z[l*m + j]: Ritz coefficients from the inverse iteration's
// column-major layout to the layout of the basis transform
__global__ void k_transpose_small(const double *__restrict__ Z, int m, int nk, double *__restrict__ Y) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m * nk; e += gridDim.x * blockDim.x) {
        const int j = e / nk, l = e - j * nk;
        Y[e] = Z[(size_t)l * m + j];
    }
}
cudaError_t transpose_small(const double *Z, int m, int nk, double *Y, cudaStream_t s) {
    const int total = m * nk;
    k_transpose_small<<<(total + 255) / 256, 256, 0, s>>>(Z, m, nk, Y);
    return cudaGetLastError();
}

// ---- lock-step Lanczos kernels (iteration index `it` read from device)
template <typename T>
__global__ void k_bpack(const BLz *__restrict__ L, const BChunk *__restrict__ ch, int nch, const int *__restrict__ itp,
                        T *__restrict__ X) {
    const int it = *itp;
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const BChunk k = ch[c];
        const BLz s = L[k.sys];
        const double *v = s.hist + (int64_t)it * s.dim + k.row0;
        for (int r = threadIdx.x; r < k.len; r += blockDim.x) X[s.off + k.row0 + r] = (T)v[r];
    }
}

// Pass 1 (br_remove_prev_overlap, src/breorthog.f90:683-711): unpack Y into
// W (fp64) and the chunk partials of <v_it, W>.
template <typename T>
__global__ void __launch_bounds__(256) k_bdot1(const BLz *__restrict__ L, const BChunk *__restrict__ ch, int nch,
                                               const int *__restrict__ itp, const T *__restrict__ Y,
                                               double *__restrict__ W) {
    __shared__ double red[8];
    const int it = *itp;
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const BChunk k = ch[c];
        const BLz s = L[k.sys];
        const double *v = s.hist + (int64_t)it * s.dim + k.row0;
        double acc = 0.0;
        for (int r = threadIdx.x; r < k.len; r += blockDim.x) {
            const double w = (double)Y[s.off + k.row0 + r];
            W[s.off + k.row0 + r] = w;
            acc = fma(v[r], w, acc);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += red[w];
            s.sqp[k.local] = t;  // reuse the norm partial slots for <v_it, W>
        }
    }
}

// alpha[it] = sum of the chunk partials (one warp per system)
__global__ void k_bred1(BLz *__restrict__ L, int nsys, const int *__restrict__ itp) {
    const int it = *itp;
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (s >= nsys) return;
    const BLz b = L[s];
    double acc = 0.0;
    for (int c = lane; c < b.nch; c += 32) acc += b.sqp[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) b.alpha[it] = acc;
}

__device__ __forceinline__ uint64_t bmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Gram-Schmidt dots (br_orthogonalize, src/breorthog.f90:831-891).
// mode 0 (every system): first W -= alpha v_it, then dots with j < it.
// mode 1 (systems whose flag is set): on a random restart W is first replaced
// by a seeded random chunk; dots with j <= it.
__global__ void __launch_bounds__(256) k_bdots2(const BLz *__restrict__ L, const BChunk *__restrict__ ch, int nch,
                                                const int *__restrict__ itp, double *__restrict__ W, int mode,
                                                uint64_t seed) {
    __shared__ double sw[kChunk];
    const int it = *itp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const BChunk k = ch[c];
        const BLz s = L[k.sys];
        const int fl = *s.flag;
        if (mode == 1 && !(fl & 1)) continue;
        __syncthreads();
        const double *v = s.hist + (int64_t)it * s.dim + k.row0;
        const double a = s.alpha[it];
        for (int r = threadIdx.x; r < k.len; r += blockDim.x) {
            double w;
            if (mode == 0) {
                w = W[s.off + k.row0 + r] - a * v[r];
            } else if (fl & 2) {
                const uint64_t h = bmix64(seed ^ bmix64(((uint64_t)k.sys << 40) ^ ((uint64_t)it << 24) ^ (uint64_t)(k.row0 + r)));
                w = ((double)(h >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
            } else {
                w = W[s.off + k.row0 + r];
            }
            sw[r] = w;
            W[s.off + k.row0 + r] = w;
        }
        __syncthreads();
        const int jmax = (mode == 0) ? it : it + 1;
        for (int j = warp; j < jmax; j += 8) {
            const double *h = s.hist + (int64_t)j * s.dim + k.row0;
            double acc = 0.0;
            for (int r = lane; r < k.len; r += 32) acc = fma(h[r], sw[r], acc);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) s.partial[(int64_t)j * s.nch + k.local] = acc;
        }
    }
}

// coef[j] for j < jmax (jmax = it or it+1 by mode); one warp per (system, j)
__global__ void k_breduce(BLz *__restrict__ L, int nsys, const int *__restrict__ itp, int mode) {
    const int it = *itp;
    const int jmax = (mode == 0) ? it : it + 1;
    if (jmax == 0) return;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int s = gw / jmax, j = gw - s * jmax;
    if (s >= nsys) return;
    const BLz b = L[s];
    if (mode == 1 && !(*b.flag & 1)) return;
    double acc = 0.0;
    for (int c = lane; c < b.nch; c += 32) acc += b.partial[(int64_t)j * b.nch + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) b.coef[j] = acc;
}

// W -= sum_{j<jmax} hist_j coef_j ; norm partials per chunk
__global__ void __launch_bounds__(256) k_bsub(const BLz *__restrict__ L, const BChunk *__restrict__ ch, int nch,
                                              const int *__restrict__ itp, double *__restrict__ W, int mode) {
    __shared__ double red[8];
    const int it = *itp;
    const int jmax = (mode == 0) ? it : it + 1;
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const BChunk k = ch[c];
        const BLz s = L[k.sys];
        if (mode == 1 && !(*s.flag & 1)) continue;
        double sq = 0.0;
        for (int r = threadIdx.x; r < k.len; r += blockDim.x) {
            double acc = 0.0;
            for (int j = 0; j < jmax; ++j) acc = fma(s.hist[(int64_t)j * s.dim + k.row0 + r], s.coef[j], acc);
            const double w = W[s.off + k.row0 + r] - acc;
            W[s.off + k.row0 + r] = w;
            sq = fma(w, w, sq);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += red[w];
            s.sqp[k.local] = t;
        }
    }
}

// mode 0: beta[it] = |W| and the safeguards of src/blanczosmain.f90:1634-1660
// (flag bit 0: beta < 0.1 beta_prev -> second full pass; bit 1: beta < 1e-4
// beta_prev -> random restart, beta[it] keeps the small value).
// mode 1: nrm2 = |W| after the second pass.
__global__ void k_bnorm(BLz *__restrict__ L, int nsys, const int *__restrict__ itp, int mode) {
    const int it = *itp;
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (s >= nsys) return;
    const BLz b = L[s];
    if (mode == 1 && !(*b.flag & 1)) return;
    double acc = 0.0;
    for (int c = lane; c < b.nch; c += 32) acc += b.sqp[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
        const double nrm = sqrt(acc);
        if (mode == 0) {
            b.beta[it] = nrm;
            int fl = 0;
            if (it > 0) {
                const double prev = b.beta[it - 1];
                if (nrm < 1e-4 * prev) fl = 3;
                else if (nrm < 0.1 * prev) fl = 1;
            }
            *b.flag = fl;
        } else {
            *b.nrm2 = nrm;
        }
    }
}

// hist_{it+1} = W / norm (zero when the Krylov space is exhausted)
__global__ void k_bscale(const BLz *__restrict__ L, const BChunk *__restrict__ ch, int nch, const int *__restrict__ itp,
                         const double *__restrict__ W) {
    const int it = *itp;
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const BChunk k = ch[c];
        const BLz s = L[k.sys];
        const double b = (*s.flag & 1) ? *s.nrm2 : s.beta[it];
        const double inv = (b > 1e-300) ? 1.0 / b : 0.0;
        double *dst = s.hist + (int64_t)(it + 1) * s.dim + k.row0;
        for (int r = threadIdx.x; r < k.len; r += blockDim.x) dst[r] = W[s.off + k.row0 + r] * inv;
    }
}

__global__ void k_bstep(int *itp) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *itp += 1;
}

}  // namespace bsg

using namespace bsg;

struct bsg_batch {
    int n = 0;
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string last_error;
    std::vector<bsg_ctx *> ctx;
    std::vector<int64_t> dims, off;
    int64_t total = 0;
    int items = 4;            // ITEMS of the batched row kernel (tile width 32*items)
    int ctas_per_sm = 4;
    int mstride = 4;
    DevBuf sys, work, workg;
    int nitems = 0;
    int nitemsg = 0;          // (system, row) items of the grouped contexts
    int nsm = 148;
    bool tuned = false;
    // the calls' tables, taken in turn; an event after the launches of the last
    // call that used each
    DevBuf ring;
    size_t ring_stride = 0;
    std::mutex ring_mu;
    int ring_at = 0;
    cudaEvent_t ring_ev[kBatchTables] = {};
};

namespace {
// SplitMix64 finalizer (Steele, Lea and Flood 2014) for host-side seeded pivots
inline uint64_t host_mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
}  // namespace

namespace {

int berr(bsg_batch *b, int code, const std::string &m) {
    b->last_error = m;
    return code;
}

int build_items(bsg_batch *b, int items) {
    std::vector<BatchItem> all, allg;
    std::vector<int64_t> wt, wtg;
    std::vector<BatchSys> sys(b->n);
    for (int s = 0; s < b->n; ++s) {
        bsg_ctx *c = b->ctx[s];
        const int tp = c->grouped ? kRowTile : 32 * items;
        const TileSet *ts = get_tiles(c, tp);
        if (!ts) return berr(b, BSG_ERR_NOMEM, "tile build failed: " + c->last_error);
        sys[s].a = c->args;
        sys[s].a.tiles = (const Tile *)ts->buf.p;
        sys[s].a.ntiles = ts->ntiles;
        sys[s].a.accumulate = 0;
        sys[s].g = c->group;
        for (int p = 0; p < 2 && c->grouped; ++p) {
            const GroupShape x = group_shape(c, p ? 8 : 4, 1);
            sys[s].parts[p] = x.parts;
            sys[s].accel[p] = x.accel;
            sys[s].bufel[p] = x.bufel;
        }
        std::vector<Tile> tl;
        build_tile_list(c, tp, tl);
        for (size_t t = 0; t < tl.size(); ++t) {
            (c->grouped ? allg : all).push_back(BatchItem{s, (int32_t)t});
            (c->grouped ? wtg : wt).push_back((int64_t)c->h_work[tl[t].row] * tl[t].npos / std::max(1, c->h_rowlen[tl[t].row]) + 1);
        }
    }
    auto heaviest = [](const std::vector<BatchItem> &v, const std::vector<int64_t> &w) {
        std::vector<size_t> ord(v.size());
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](size_t x, size_t y) { return w[x] > w[y]; });
        std::vector<BatchItem> sorted(v.size());
        for (size_t i = 0; i < ord.size(); ++i) sorted[i] = v[ord[i]];
        return sorted;
    };
    const std::vector<BatchItem> sorted = heaviest(all, wt), sortedg = heaviest(allg, wtg);
    int st;
    bsg_ctx *c0 = b->ctx[0];
    if ((st = upload(c0, b->sys, sys.data(), sizeof(BatchSys) * sys.size())) ||
        (st = upload(c0, b->work, sorted.data(), sizeof(BatchItem) * sorted.size())) ||
        (st = upload(c0, b->workg, sortedg.data(), sizeof(BatchItem) * sortedg.size())))
        return berr(b, st, c0->last_error);
    b->nitems = (int)sorted.size();
    b->nitemsg = (int)sortedg.size();
    b->items = items;
    return BSG_OK;
}

// the host image of a call's table (null: no memory)
std::unique_ptr<unsigned char[]> call_table(const bsg_batch *b, const void *const *vin, void *const *vout, size_t &bytes) {
    bytes = kBatchVecOff + sizeof(BatchVec) * (size_t)b->n;
    std::unique_ptr<unsigned char[]> t(new (std::nothrow) unsigned char[bytes]());
    for (int k = 0; t && k < b->n; ++k) {
        const BatchVec v{vin[k], vout[k]};
        std::memcpy(t.get() + kBatchVecOff + sizeof(BatchVec) * (size_t)k, &v, sizeof v);
    }
    return t;
}

// the same on the device for as long as the caller's buffer lives, written
// before the function returns
int place_table(bsg_batch *b, DevBuf &d, const void *const *vin, void *const *vout) {
    size_t bytes = 0;
    const auto t = call_table(b, vin, vout, bytes);
    const int st = t ? dev_alloc(b->ctx[0], d, bytes) : BSG_ERR_NOMEM;
    if (st) return berr(b, st, "batch vector table: no memory");
    if (cudaMemcpyAsync(d.p, t.get(), bytes, cudaMemcpyHostToDevice, b->stream) != cudaSuccess ||
        cudaStreamSynchronize(b->stream) != cudaSuccess)
        return berr(b, BSG_ERR_CUDA, "batch vector table upload failed");
    return BSG_OK;
}

template <typename T>
int launch_batch_group(bsg_batch *b, const void *table, cudaStream_t s) {
    if (b->nitemsg == 0) return BSG_OK;
    size_t smem = 0;
    for (bsg_ctx *c : b->ctx)
        if (c->grouped) smem = std::max(smem, group_shape(c, sizeof(T), 1).bytes(sizeof(T)));
    auto kern = k_rowgroup_batch<T>;
    cudaError_t e = smem > kGroupSmemMax ? cudaErrorInvalidValue
                                         : cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGroupSmemMax);
    if (e == cudaSuccess) {
        kern<<<(unsigned)b->nitemsg, 256, smem, s>>>((const BatchSys *)b->sys.p,
                                                       (const BatchVec *)((const char *)table + kBatchVecOff),
                                                       (const BatchItem *)b->workg.p);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return berr(b, BSG_ERR_CUDA, std::string("batched applyH: ") + cudaGetErrorString(e));
    return BSG_OK;
}

template <typename T, int ITEMS>
int launch_tiles_t(bsg_batch *b, void *table, cudaStream_t s) {
    if (b->nitems == 0) return BSG_OK;
    const size_t smem = align16(sizeof(float) * (size_t)kWarps * b->mstride) + sizeof(T) * (size_t)kWarps * 32 * ITEMS;
    auto kern = batch_rows_kernel<T, ITEMS>();
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaMemsetAsync(table, 0, sizeof(int), s);
    if (e == cudaSuccess) {
        const int grid = std::max(1, std::min(b->nitems, b->nsm * b->ctas_per_sm));
        kern<<<grid, kWarps * 32, smem, s>>>((const BatchSys *)b->sys.p,
                                             (const BatchVec *)((const char *)table + kBatchVecOff),
                                             (const BatchItem *)b->work.p, b->nitems, (int *)table, b->mstride);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return berr(b, BSG_ERR_CUDA, std::string("batched applyH: ") + cudaGetErrorString(e));
    return BSG_OK;
}

// the members without jump groups.  table: the call's own (place_table's
// layout), in use until the launches end
int launch_tiles(bsg_batch *b, int prec, void *table, cudaStream_t s) {
    if (prec == BSG_PREC_FP32) {
        switch (b->items) {
        case 1: return launch_tiles_t<float, 1>(b, table, s);
        case 2: return launch_tiles_t<float, 2>(b, table, s);
        case 8: return launch_tiles_t<float, 8>(b, table, s);
        default: return launch_tiles_t<float, 4>(b, table, s);
        }
    }
    switch (b->items) {
    case 1: return launch_tiles_t<double, 1>(b, table, s);
    case 2: return launch_tiles_t<double, 2>(b, table, s);
    case 8: return launch_tiles_t<double, 8>(b, table, s);
    default: return launch_tiles_t<double, 4>(b, table, s);
    }
}

int launch_batch(bsg_batch *b, int prec, void *table, cudaStream_t s) {
    const int st = prec == BSG_PREC_FP32 ? launch_batch_group<float>(b, table, s) : launch_batch_group<double>(b, table, s);
    return st ? st : launch_tiles(b, prec, table, s);
}

}  // namespace

extern "C" {

int bsg_batch_create(int n, const bsg_tables *const *tables, const bsg_config *cfg, bsg_batch **out) {
    if (!out || n < 1 || !tables) return BSG_ERR_ARG;
    *out = nullptr;
    bsg_batch *b = new (std::nothrow) bsg_batch();
    if (!b) return BSG_ERR_NOMEM;
    b->n = n;
    b->device = cfg ? cfg->device : 0;
    int st = BSG_OK;
    // the systems' set-ups (validation, derived layouts, uploads) are
    // independent: host threads take them in turn
    std::vector<bsg_ctx *> made(n, nullptr);
    std::vector<int> stv(n, BSG_OK);
    {
        std::atomic<int> next{0};
        auto worker = [&]() {
            for (int s = next++; s < n; s = next++) stv[s] = bsg_create(tables[s], cfg, &made[s]);
        };
        const int nth = (int)std::max(1u, std::min<unsigned>(16u, std::min<unsigned>((unsigned)n, std::thread::hardware_concurrency())));
        std::vector<std::thread> pool;
        for (int t = 1; t < nth; ++t) pool.emplace_back(worker);
        worker();
        for (auto &th : pool) th.join();
    }
    for (int s = 0; s < n; ++s)
        if (stv[s] != BSG_OK && !st) {
            st = stv[s];
            b->last_error = "system " + std::to_string(s) + ": bsg_create failed";
        }
    if (st) {
        for (bsg_ctx *c : made)
            if (c) bsg_destroy(c);
        delete b;
        return st;
    }
    for (int s = 0; s < n; ++s) {
        bsg_ctx *c = made[s];
        b->ctx.push_back(c);
        b->dims.push_back(c->dim);
        b->off.push_back(b->total);
        b->total += c->dim;
        b->mstride = std::max(b->mstride, (c->args.max_nbd + 3) & ~3);
    }
    if (!st) {
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, b->device) == cudaSuccess) b->nsm = prop.multiProcessorCount;
        if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) st = BSG_ERR_CUDA;
    }
    if (!st) {
        b->ring_stride = (kBatchVecOff + sizeof(BatchVec) * (size_t)n + 255) & ~(size_t)255;
        st = dev_alloc(b->ctx[0], b->ring, b->ring_stride * kBatchTables);
    }
    for (int k = 0; k < kBatchTables && !st; ++k)
        if (cudaEventCreateWithFlags(&b->ring_ev[k], cudaEventDisableTiming) != cudaSuccess) st = BSG_ERR_CUDA;
    if (!st) st = build_items(b, 4);
    if (st) {
        bsg_batch_destroy(b);
        return st;
    }
    *out = b;
    return BSG_OK;
}

int bsg_batch_destroy(bsg_batch *b) {
    if (!b) return BSG_ERR_ARG;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    dev_free(b->sys);
    dev_free(b->work);
    dev_free(b->workg);
    dev_free(b->ring);
    for (cudaEvent_t e : b->ring_ev)
        if (e) cudaEventDestroy(e);
    for (bsg_ctx *c : b->ctx) bsg_destroy(c);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return BSG_OK;
}

int bsg_batch_grad(bsg_batch *b, const double *const *evecs, int nstates, double *const *dpp, double *const *dnn,
                   double *const *dpn, double *const *dspe_p, double *const *dspe_n, double *kernel_ms) {
    if (!b) return BSG_ERR_ARG;
    cudaSetDevice(b->device);
    std::string err;
    const int st = grad_many(b->ctx.data(), b->n, evecs, nstates, dpp, dnn, dpn, dspe_p, dspe_n, b->stream, err,
                             kernel_ms);
    if (st) return berr(b, st, "bsg_batch_grad: " + err);
    return BSG_OK;
}

int bsg_batch_last_error(const bsg_batch *b, char *buf, size_t len) {
    if (!b || !buf || !len) return BSG_ERR_ARG;
    std::snprintf(buf, len, "%s", b->last_error.c_str());
    return BSG_OK;
}

int bsg_batch_dims(const bsg_batch *b, int64_t *dims) {
    if (!b || !dims) return BSG_ERR_ARG;
    for (int s = 0; s < b->n; ++s) dims[s] = b->dims[s];
    return BSG_OK;
}

int bsg_batch_system(const bsg_batch *b, int s, bsg_ctx **ctx) {
    if (!b || !ctx || s < 0 || s >= b->n) return BSG_ERR_ARG;
    *ctx = b->ctx[s];
    return BSG_OK;
}

int bsg_batch_applyh(bsg_batch *b, const void *const *vin, void *const *vout, int prec, void *stream) {
    if (!b || !vin || !vout || (prec != BSG_PREC_FP32 && prec != BSG_PREC_FP64)) return BSG_ERR_ARG;
    cudaSetDevice(b->device);
    // stream: the caller's cudaStream_t; NULL is the legacy default stream
    cudaStream_t s = (cudaStream_t)stream;
    // a graph would copy the table from host memory that is gone when it runs
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return berr(b, BSG_ERR_CUDA, "bsg_batch_applyh cannot run while the stream is captured");
    }
    size_t bytes = 0;
    const auto t = call_table(b, vin, vout, bytes);
    if (!t) return berr(b, BSG_ERR_NOMEM, "bsg_batch_applyh: no host memory");
    std::lock_guard<std::mutex> lock(b->ring_mu);
    const int k = b->ring_at;
    b->ring_at = (k + 1) % kBatchTables;
    void *table = (char *)b->ring.p + b->ring_stride * (size_t)k;
    // after the launches that last read this place, on whatever stream; the
    // copy from pageable memory has left `t` when the call returns
    cudaError_t e = cudaStreamWaitEvent(s, b->ring_ev[k], 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(table, t.get(), bytes, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return berr(b, BSG_ERR_CUDA, std::string("batch vector table: ") + cudaGetErrorString(e));
    const int st = launch_batch(b, prec, table, s);
    e = cudaEventRecord(b->ring_ev[k], s);
    if (!st && e != cudaSuccess) return berr(b, BSG_ERR_CUDA, std::string("batch event: ") + cudaGetErrorString(e));
    return st;
}

// autotuner: time the persistent launch for each tile width and CTA residency,
// keep the fastest (vectors are scratch, fp32).  The jump groups' launch has no
// choice to make: a batch whose members all have groups keeps its setting.
int bsg_batch_autotune(bsg_batch *b, int *items_out, int *ctas_out, double *best_ms_out) {
    if (!b) return BSG_ERR_ARG;
    cudaSetDevice(b->device);
    DevBuf x, y, tab;
    bsg_ctx *c0 = b->ctx[0];
    int st;
    if ((st = dev_alloc(c0, x, sizeof(float) * b->total)) || (st = dev_alloc(c0, y, sizeof(float) * b->total))) {
        dev_free(x);
        return berr(b, st, "autotune scratch allocation failed");
    }
    cudaMemset(x.p, 0, sizeof(float) * b->total);
    std::vector<const void *> vi(b->n);
    std::vector<void *> vo(b->n);
    for (int s = 0; s < b->n; ++s) {
        vi[s] = (const float *)x.p + b->off[s];
        vo[s] = (float *)y.p + b->off[s];
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 1e300;
    int bi = b->items, bc = b->ctas_per_sm;
    // mean of three launches after one warm-up
    auto timed = [&](auto launch) -> double {
        launch();
        cudaEventRecord(e0, b->stream);
        for (int r = 0; r < 3; ++r) launch();
        cudaEventRecord(e1, b->stream);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        return ms / 3;
    };
    // 2 CTAs per SM never won on the measured batches
    const int cand_items[] = {1, 2, 4, 8};
    const int cand_ctas[] = {4, 8};
    st = place_table(b, tab, vi.data(), vo.data());
    for (int it : cand_items) {
        if (st || b->nitems == 0 || (st = build_items(b, it))) break;
        for (int cps : cand_ctas) {
            b->ctas_per_sm = cps;
            const double ms = timed([&]() { launch_tiles(b, BSG_PREC_FP32, tab.p, b->stream); });
            if (ms < best) {
                best = ms;
                bi = it;
                bc = cps;
            }
        }
    }
    if (!st && b->nitems) {
        b->ctas_per_sm = bc;
        st = build_items(b, bi);
    }
    // the whole call with that setting
    if (!st) best = timed([&]() { launch_batch(b, BSG_PREC_FP32, tab.p, b->stream); });
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    dev_free(x);
    dev_free(y);
    dev_free(tab);
    if (st) return st;
    b->tuned = true;
    if (items_out) *items_out = bi;
    if (ctas_out) *ctas_out = bc;
    if (best_ms_out) *best_ms_out = best;
    return BSG_OK;
}

int bsg_batch_set_tuning(bsg_batch *b, int items, int ctas_per_sm) {
    if (!b || (items != 1 && items != 2 && items != 4 && items != 8) || ctas_per_sm < 1 || ctas_per_sm > 16)
        return BSG_ERR_ARG;
    cudaSetDevice(b->device);
    b->ctas_per_sm = ctas_per_sm;
    return build_items(b, items);
}

// lock-step Lanczos over all systems: fixed p->niter iterations, uniform
// pivot per system (or seeded random ones, p->pivot == 1), lowest p->nkeep eigenvalues per
// system into evals[s*nkeep + k]; evecs: NULL or n host pointers of
// dim_s*nkeep doubles (column-major).
int bsg_batch_lanczos(bsg_batch *b, const bsg_lanczos_params *p, double *evals, double *const *evecs,
                      bsg_report *rep) {
    if (!b || !p || !evals) return BSG_ERR_ARG;
    if (p->niter < 2 || p->nkeep < 1 || p->nkeep > 128 ||
        (p->matvec_prec != BSG_PREC_FP32 && p->matvec_prec != BSG_PREC_FP64))
        return berr(b, BSG_ERR_ARG, "bsg_batch_lanczos: bad parameters");
    cudaSetDevice(b->device);
    const int niter = p->niter, n = b->n;
    for (int s = 0; s < n; ++s)
        if (b->dims[s] <= niter) return berr(b, BSG_ERR_ARG, "bsg_batch_lanczos: niter must be below every dimension");
    cudaStream_t s0 = b->stream;
    bsg_ctx *c0 = b->ctx[0];
    const int esz = p->matvec_prec == BSG_PREC_FP32 ? 4 : 8;
    // chunks and per-system bookkeeping
    std::vector<BChunk> chunks;
    std::vector<BLz> lz(n);
    int64_t histsz = 0, partsz = 0, sqsz = 0;
    for (int s = 0; s < n; ++s) {
        const int nch = (int)((b->dims[s] + kChunk - 1) / kChunk);
        for (int c = 0; c < nch; ++c)
            chunks.push_back(BChunk{s, c, c * kChunk, (int32_t)std::min<int64_t>(kChunk, b->dims[s] - (int64_t)c * kChunk)});
        lz[s].dim = b->dims[s];
        lz[s].off = b->off[s];
        lz[s].nch = nch;
        histsz += (int64_t)(niter + 1) * b->dims[s];
        partsz += (int64_t)(niter + 1) * nch;
        sqsz += nch;
    }
    DevBuf hist, X, Y, W, part, coef, sqp, ab, itd, chd, lzd, fl, tab;
    int st;
    size_t fr = 0, tot = 0;
    const size_t need = (size_t)histsz * 8 + (size_t)b->total * (2 * esz + 8);
    cudaMemGetInfo(&fr, &tot);
    if (need > fr) {
        pool_trim(b->device);
        cudaMemGetInfo(&fr, &tot);
    }
    if (need > fr)
        return berr(b, BSG_ERR_NOMEM, "bsg_batch_lanczos: histories do not fit in device memory");
    if ((st = dev_alloc(c0, hist, 8 * (size_t)histsz)) || (st = dev_alloc(c0, X, (size_t)esz * b->total)) ||
        (st = dev_alloc(c0, Y, (size_t)esz * b->total)) || (st = dev_alloc(c0, W, 8 * (size_t)b->total)) ||
        (st = dev_alloc(c0, part, 8 * (size_t)partsz)) || (st = dev_alloc(c0, coef, 8 * (size_t)n * (niter + 1))) ||
        (st = dev_alloc(c0, sqp, 8 * (size_t)sqsz)) || (st = dev_alloc(c0, ab, 8 * (size_t)2 * n * niter)) ||
        (st = dev_alloc(c0, itd, sizeof(int) * 4)) || (st = dev_alloc(c0, fl, 16 * (size_t)n))) {
        DevBuf *bs[] = {&hist, &X, &Y, &W, &part, &coef, &sqp, &ab, &itd, &fl};
        for (DevBuf *x : bs) dev_free(*x);
        return berr(b, st, "bsg_batch_lanczos: allocation failed");
    }
    {
        int64_t ho = 0, po = 0, so = 0;
        for (int s = 0; s < n; ++s) {
            lz[s].hist = (double *)hist.p + ho;
            lz[s].partial = (double *)part.p + po;
            lz[s].coef = (double *)coef.p + (int64_t)s * (niter + 1);
            lz[s].sqp = (double *)sqp.p + so;
            lz[s].alpha = (double *)ab.p + (int64_t)s * niter;
            lz[s].beta = (double *)ab.p + (int64_t)n * niter + (int64_t)s * niter;
            lz[s].nrm2 = (double *)fl.p + s;
            lz[s].flag = (int32_t *)((double *)fl.p + n) + s;
            ho += (int64_t)(niter + 1) * b->dims[s];
            po += (int64_t)(niter + 1) * lz[s].nch;
            so += lz[s].nch;
        }
    }
    st = upload(c0, chd, chunks.data(), sizeof(BChunk) * chunks.size());
    if (!st) st = upload(c0, lzd, lz.data(), sizeof(BLz) * lz.size());
    // pivots: uniform 1/sqrt(dim) per system (initialize_lanczos_vector
    // option 0), or (p->pivot == 1) a seeded pseudo-random normalized vector
    // per system: SplitMix64 of (seed, system, index) through Box-Muller, so
    // that no symmetry of the uniform vector restricts the Krylov space
    for (int s = 0; s < n && !st; ++s) {
        std::vector<double> v(b->dims[s], 1.0 / std::sqrt((double)b->dims[s]));
        if (p->pivot == 1) {
            double nrm = 0.0;
            for (int64_t i = 0; i < b->dims[s]; ++i) {
                const uint64_t h = host_mix64(p->seed ^ host_mix64(((uint64_t)s << 40) ^ (uint64_t)i));
                const uint64_t h2 = host_mix64(h);
                const double u1 = ((double)(h >> 11) + 1.0) * (1.0 / 9007199254740992.0);
                const double u2 = (double)(h2 >> 11) * (1.0 / 9007199254740992.0);
                v[i] = std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
                nrm += v[i] * v[i];
            }
            const double inv = 1.0 / std::sqrt(nrm);
            for (double &x : v) x *= inv;
        }
        if (cudaMemcpyAsync(lz[s].hist, v.data(), 8 * v.size(), cudaMemcpyHostToDevice, s0) != cudaSuccess ||
            cudaStreamSynchronize(s0) != cudaSuccess)
            st = BSG_ERR_CUDA;
    }
    // matvec vectors: X + off (in), Y + off (out)
    if (!st) {
        std::vector<const void *> vi(n);
        std::vector<void *> vo(n);
        for (int s = 0; s < n; ++s) {
            vi[s] = (const char *)X.p + (size_t)esz * b->off[s];
            vo[s] = (char *)Y.p + (size_t)esz * b->off[s];
        }
        st = place_table(b, tab, vi.data(), vo.data());
    }
    if (!st && cudaMemsetAsync(itd.p, 0, sizeof(int), s0) != cudaSuccess) st = BSG_ERR_CUDA;
    if (!st && cudaMemsetAsync(fl.p, 0, 16 * (size_t)n, s0) != cudaSuccess) st = BSG_ERR_CUDA;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int nchunks = (int)chunks.size();
    const int G = std::max(1, std::min(nchunks, b->nsm * 8));
    // ---- capture one iteration
    if (!st) {
        cudaStreamSynchronize(s0);
        cudaError_t e = cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            const int *itp = (const int *)itd.p;
            if (esz == 4)
                k_bpack<float><<<G, 256, 0, s0>>>((const BLz *)lzd.p, (const BChunk *)chd.p, nchunks, itp, (float *)X.p);
            else
                k_bpack<double><<<G, 256, 0, s0>>>((const BLz *)lzd.p, (const BChunk *)chd.p, nchunks, itp, (double *)X.p);
            int lst = launch_batch(b, p->matvec_prec, tab.p, s0);
            const BLz *Lc = (const BLz *)lzd.p;
            BLz *Lm = (BLz *)lzd.p;
            const BChunk *Cc = (const BChunk *)chd.p;
            if (esz == 4)
                k_bdot1<float><<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (const float *)Y.p, (double *)W.p);
            else
                k_bdot1<double><<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (const double *)Y.p, (double *)W.p);
            const int sysblk = (n * 32 + 255) / 256;
            const int pairblk = (n * (niter + 1) * 32 + 255) / 256;
            k_bred1<<<sysblk, 256, 0, s0>>>(Lm, n, itp);
            k_bdots2<<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (double *)W.p, 0, p->seed);
            k_breduce<<<pairblk, 256, 0, s0>>>(Lm, n, itp, 0);
            k_bsub<<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (double *)W.p, 0);
            k_bnorm<<<sysblk, 256, 0, s0>>>(Lm, n, itp, 0);
            // second full pass / random restart for flagged systems
            k_bdots2<<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (double *)W.p, 1, p->seed);
            k_breduce<<<pairblk, 256, 0, s0>>>(Lm, n, itp, 1);
            k_bsub<<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (double *)W.p, 1);
            k_bnorm<<<sysblk, 256, 0, s0>>>(Lm, n, itp, 1);
            k_bscale<<<G, 256, 0, s0>>>(Lc, Cc, nchunks, itp, (const double *)W.p);
            k_bstep<<<1, 32, 0, s0>>>((int *)itd.p);
            e = cudaStreamEndCapture(s0, &graph);
            if (lst) st = lst;
            if (e == cudaSuccess && !st) e = cudaGraphInstantiate(&gexec, graph, 0);
        }
        if (e != cudaSuccess && !st) st = berr(b, BSG_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    }
    float loop_ms = 0.f;
    if (!st) {
        cudaEventRecord(e0, s0);
        for (int it = 0; it < niter && !st; ++it)
            if (cudaGraphLaunch(gexec, s0) != cudaSuccess) st = berr(b, BSG_ERR_CUDA, "graph launch failed");
        cudaEventRecord(e1, s0);
        if (cudaEventSynchronize(e1) != cudaSuccess) st = berr(b, BSG_ERR_CUDA, "batched Lanczos failed");
        cudaEventElapsedTime(&loop_ms, e0, e1);
    }
    // ---- projected tridiagonal matrices: eigenpairs on the device.  Every
    // system's solve is queued on one stream without host round trips (alpha
    // and beta are read where the loop left them, eigenvalues and Ritz vectors
    // collect in device arrays); one synchronization, then the copies out.
    float eig_ms = 0.f;
    if (!st) {
        std::vector<double> abh((size_t)2 * n * niter);
        if (cudaMemcpy(abh.data(), ab.p, 8 * abh.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
            st = berr(b, BSG_ERR_CUDA, "batched Lanczos: reading alpha/beta failed");
        const int nk = std::min(p->nkeep, niter);
        const bool vecs = evecs != nullptr;
        int64_t tot_dim = 0;
        for (int s = 0; s < n; ++s) tot_dim += b->dims[s];
        DevBuf evd, Z, wk, Yd, outv;
        if (!st && ((st = dev_alloc(c0, evd, 8 * (size_t)n * nk)) || (st = dev_alloc(c0, Z, 8 * (size_t)niter * nk)) ||
                    (st = dev_alloc(c0, wk, 8 * (size_t)6 * niter * nk)) || (st = dev_alloc(c0, Yd, 8 * (size_t)niter * nk)) ||
                    (vecs && (st = dev_alloc(c0, outv, 8 * (size_t)tot_dim * nk))))) {
            st = berr(b, st, "eigen workspace allocation failed");
        }
        cudaEventRecord(e0, s0);
        cudaError_t e = cudaSuccess;
        int64_t off = 0;
        for (int s = 0; s < n && !st && e == cudaSuccess; ++s) {
            const double *A = abh.data() + (size_t)s * niter, *B = abh.data() + (size_t)n * niter + (size_t)s * niter;
            double glo = 1e300, ghi = -1e300;
            for (int i = 0; i < niter; ++i) {
                const double r = (i > 0 ? std::fabs(B[i - 1]) : 0.0) + (i + 1 < niter ? std::fabs(B[i]) : 0.0);
                glo = std::min(glo, A[i] - r);
                ghi = std::max(ghi, A[i] + r);
            }
            const double scale = std::max(std::fabs(glo), std::fabs(ghi));
            glo -= 1e-12 * scale + 1e-300;
            ghi += 1e-12 * scale + 1e-300;
            const double *ald = (const double *)ab.p + (size_t)s * niter;
            const double *btd = (const double *)ab.p + (size_t)n * niter + (size_t)s * niter;
            double *evs = (double *)evd.p + (size_t)s * nk;
            e = bisect_arrow(niter, 0, ald, btd, nk, glo, ghi, evs, s0);
            if (e == cudaSuccess && vecs && evecs[s]) {
                e = inverse_iter_arrow(niter, 0, ald, btd, evs, nk, scale, (double *)Z.p, (double *)wk.p, s0);
                if (e == cudaSuccess) e = transpose_small((const double *)Z.p, niter, nk, (double *)Yd.p, s0);
                if (e == cudaSuccess)
                    e = transform(lz[s].hist, niter, (const double *)Yd.p, nk, nk, (double *)outv.p + off * nk,
                                  b->dims[s], b->dims[s], b->dims[s], s0);
            }
            off += b->dims[s];
        }
        std::vector<double> w((size_t)n * nk);
        if (!st && e == cudaSuccess) e = cudaMemcpyAsync(w.data(), evd.p, 8 * w.size(), cudaMemcpyDeviceToHost, s0);
        if (!st && e == cudaSuccess) e = cudaStreamSynchronize(s0);
        off = 0;
        for (int s = 0; s < n && !st && e == cudaSuccess; ++s) {
            if (vecs && evecs[s])
                e = cudaMemcpy(evecs[s], (const double *)outv.p + off * nk, 8 * (size_t)b->dims[s] * nk,
                               cudaMemcpyDeviceToHost);
            off += b->dims[s];
        }
        if (!st && e != cudaSuccess) st = berr(b, BSG_ERR_CUDA, std::string("batched eigen-solve: ") + cudaGetErrorString(e));
        if (!st)
            for (int s = 0; s < n; ++s)
                for (int k = 0; k < p->nkeep; ++k) evals[(size_t)s * p->nkeep + k] = k < nk ? w[(size_t)s * nk + k] : NAN;
        cudaEventRecord(e1, s0);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&eig_ms, e0, e1);
        DevBuf *bs2[] = {&evd, &Z, &wk, &Yd, &outv};
        for (DevBuf *x : bs2) dev_free(*x);
    }
    if (rep) {
        std::memset(rep, 0, sizeof(*rep));
        rep->iterations = niter;
        rep->total_iterations = niter;
        rep->matvecs = niter;
        rep->converged = st ? 0 : 1;
        rep->t_total_ms = loop_ms + eig_ms;
        rep->t_matvec_ms = loop_ms;  // whole captured iteration (matvec + reorthogonalization)
        rep->t_eig_ms = eig_ms;
    }
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    DevBuf *bs[] = {&hist, &X, &Y, &W, &part, &coef, &sqp, &ab, &itd, &chd, &lzd, &fl, &tab};
    for (DevBuf *x : bs) dev_free(*x);
    return st;
}

}  // extern "C"
