// Row-tile body of the adjoint (Hellmann-Feynman gradient), shared by the
// single-system bsg_grad and the batched bsg_batch_grad.
//
// dE_k/dhmat(label) = sum over every appearance of the label in H of
// phase * psi_k(out) * psi_k(in): the traversal of the two-body densities
// applyh{PP,NN,PN}bundled_den (src/bdenslib4.f90:129-729, dmat(op) +=
// vout(f)*vin(i)*phase) with both vectors equal to the eigenvector, run over
// the matvec's row tiles and (row, warp) slots (NN: over the rows of each
// operator, k_grad_nn), so every f/b appearance, hermitian half and 1/2 on
// diagonal pair labels counts as in the matvec.
//
// Determinism: every global sum is a 128-bit two's-complement fixed-point
// number with 64 fraction bits, updated with 64-bit integer atomics (low word,
// carry into the high word).  Integer addition is associative, so the result
// does not depend on the order in which CTAs arrive; doubles convert exactly
// down to 2^-64.  Per-warp PN bins are summed in lane order.
#pragma once

#include "bsg_internal.h"

namespace bsg {

constexpr int kGradWarps = kRowWarps;

struct GradArgs {
    const int32_t *pp_op;         // hmatpp label of each PP contribution
    const int8_t *pp_ph;          // its jump phase
    const int32_t *nnrec_op;      // hmatnn label of each NN record
    const int8_t *nnrec_ph;       // its jump phase
    // fixed-point accumulators, (lo, hi) words per label: acc[2i], acc[2i+1]
    unsigned long long *pp, *nn, *pn, *spe_p, *spe_n;
};

// acc += v exactly (to 2^-64), order-independent
__device__ __forceinline__ void fix_add(unsigned long long *acc, double v) {
    if (v == 0.0) return;
    const double fl = floor(v);
    const double fr = v - fl;  // [0, 1), exact for |v| < 2^52
    const unsigned long long lo = __double2ull_rz(fr * 18446744073709551616.0);
    const unsigned long long hi = (unsigned long long)(long long)fl;
    const unsigned long long old = atomicAdd(acc, lo);
    atomicAdd(acc + 1, hi + (old + lo < old ? 1ull : 0ull));
}

__device__ __forceinline__ double fix_value(const unsigned long long *acc) {
    return (double)(long long)acc[1] + (double)acc[0] * 5.421010862427522170e-20;  // 2^-64
}

__device__ __forceinline__ double grad_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One tile of one output row for NS states: the records, their labels and the
// lanes that meet in a bin are the same for every state, so they are read and
// matched once.  Each state's sums run in the order that they have alone.
// What bounds it: the latency of record -> gather -> match -> bin per step, and
// the atomics of the labels.  sd 6p6n (dim 93,710), five states in one pass
// against one each: see kGradStates.
// psi: the first state's vector, the next ones dim apart; g: the first state's
// accumulators, the next ones gstride words apart.  Aw: this warp's FP64 bins
// for the distinct (b,d) pairs of a PN operator (NS times mstride doubles);
// stage: its lanes' products (NS times 33 doubles, a pad against conflicts).
template <int ITEMS, int NS>
__device__ __forceinline__ void grad_tile(const RowArgs &a, const GradArgs &g, const double *__restrict__ psi,
                                          int64_t dim, int64_t gstride, const Tile tile, double *__restrict__ Aw,
                                          int mstride, double *__restrict__ stage) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = tile.row;
    const int64_t roff = a.row_off[row];
    const int slot = row * kGradWarps + warp;
    int pos[ITEMS];
    bool valid[ITEMS];
    double pout[NS][ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int local = lane + 32 * i;
        pos[i] = tile.pos0 + local;
        valid[i] = local < tile.npos;
#pragma unroll
        for (int s = 0; s < NS; ++s) pout[s][i] = valid[i] ? psi[s * dim + roff + pos[i]] : 0.0;
    }
    // ---- PP: dpp[op] += ph * sum_pos psi[row+pos] psi[q+pos]
    for (int c = a.pp_ptr[slot]; c < a.pp_ptr[slot + 1]; ++c) {
        const PPContrib pc = a.pp[c];
        double v[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) v[s] = 0.0;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (valid[i] && pos[i] >= pc.lo && pos[i] <= pc.hi) {
#pragma unroll
                for (int s = 0; s < NS; ++s) v[s] += pout[s][i] * psi[s * dim + pc.q_off + pos[i]];
            }
        unsigned long long *acc = g.pp + 2 * (size_t)(g.pp_op[c] - 1);
        const double ph = (double)g.pp_ph[c];
#pragma unroll
        for (int s = 0; s < NS; ++s) v[s] = grad_warp_sum(v[s]);
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (lane == s) fix_add(acc + s * gstride, ph * v[s]);
    }
    // ---- PN: dpn[cpn(b,a)+dpn(d,c)] += php * phn * psi[row+pos] psi[q+in]
    // Records are walked in warp-wide steps, the next step's record on its way
    // meanwhile; in each step the lanes that hit the same (b,d) bin are added in
    // lane order, the states shared out among these lanes.
    const unsigned below = (1u << lane) - 1;
    for (int c = a.pn_ptr[slot]; c < a.pn_ptr[slot + 1]; ++c) {
        const PNContrib pc = a.pn[c];
        const NOp op = a.nops[pc.nop];
#pragma unroll
        for (int s = 0; s < NS; ++s)
            for (int k = lane; k < op.nbd; k += 32) Aw[s * mstride + k] = 0.0;
        __syncwarp();
        const int32_t *__restrict__ ptr = a.nptr + op.ptr_base;
        const PNRec *__restrict__ rec = a.pnrec + op.rec_base;
        const double *__restrict__ q = psi + pc.q_off;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            int k0 = 0, n = 0;
            if (valid[i] && pos[i] < op.nout) {
                k0 = ptr[pos[i]];
                n = ptr[pos[i] + 1] - k0;
            }
            const int nmax = __reduce_max_sync(0xffffffffu, n);
            PNRec r{};
            if (n > 0) r = rec[k0];
            for (int j = 0; j < nmax; ++j) {
                int key = -1;
                if (j < n) {
                    key = r.k;
#pragma unroll
                    for (int s = 0; s < NS; ++s)
                        stage[s * 33 + lane] = pout[s][i] * q[s * dim + r.in] * (double)r.ph;
                    if (j + 1 < n) r = rec[k0 + j + 1];
                }
                const unsigned grp = __match_any_sync(0xffffffffu, key);
                __syncwarp();
                if (key >= 0) {
                    const int size = __popc(grp);
                    for (int s = __popc(grp & below); s < NS; s += size) {
                        double v = 0.0;
                        for (unsigned m = grp; m; m &= m - 1) v += stage[s * 33 + __ffs(m) - 1];
                        Aw[s * mstride + key] += v;
                    }
                }
                __syncwarp();
            }
        }
        for (int k = lane; k < op.nbd; k += 32) {
            const BDPair bd = a.bd[op.bd_base + k];
            unsigned long long *acc = g.pn + 2 * (size_t)(a.cpn[bd.b + pc.aoff] + a.dpn[bd.d + pc.coff] - 1);
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const double v = Aw[s * mstride + k];
                if (v != 0.0) fix_add(acc + s * gstride, (double)pc.php * v);
            }
        }
        __syncwarp();
    }
    // ---- SPE: d/dpspe_h(ip) and d/dnspe_h(in) of sum psi^2 (pspe + nspe)
    if (g.spe_p) {
        for (int c = a.spe_ptr[slot]; c < a.spe_ptr[slot + 1]; ++c) {
            const SPEContrib sc = a.spe[c];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                double v = 0.0;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    if (valid[i] && pos[i] >= sc.lo && pos[i] <= sc.hi) {
                        const double p2 = pout[s][i] * pout[s][i];
                        v += p2;
                        fix_add(g.spe_n + s * gstride + 2 * (size_t)(sc.n0 + (pos[i] - sc.lo)), p2);
                    }
                }
                v = grad_warp_sum(v);
                if (lane == 0) fix_add(g.spe_p + s * gstride + 2 * (size_t)row, v);
            }
        }
    }
}

// shared memory of one adjoint CTA: the warps' bins, then their products
__host__ __device__ constexpr size_t grad_smem_bytes(int mstride, int ns) {
    return sizeof(double) * (size_t)kGradWarps * ns * ((size_t)(mstride > 0 ? mstride : 2) + 33);
}

__device__ __forceinline__ void grad_smem(int mstride, int ns, double *&Aw, double *&stage) {
    extern __shared__ __align__(16) double smem_grad[];
    const int warp = threadIdx.x >> 5;
    const int ms = mstride > 0 ? mstride : 2;
    Aw = smem_grad + (size_t)warp * ns * ms;
    stage = smem_grad + (size_t)kGradWarps * ns * ms + (size_t)warp * ns * 33;
}

}  // namespace bsg
