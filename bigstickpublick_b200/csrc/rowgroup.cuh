// Whole-row body of applyH on jump groups, shared by the single-system and
// the batched kernel.
//
// One CTA owns one output row (proton SD p).  The proton jumps p'_j -> p that
// use the same neutron operator are taken J = 4, 2 or 1 at a time: the CTA
// stages their J input rows interleaved, X[n'][j], and their J matrix-element
// rows interleaved, V[k][j], in shared memory, and then walks the operator's
// records once for all of them,
//     out[n] += sum_r s_r (V[k_r][0] X[n'_r][0] + ... + V[k_r][J-1] X[n'_r][J-1]).
// What a record costs is one coalesced 4-byte load and two vector loads from
// shared memory; walked once per jump it cost a record load, a gathered load
// through L1 and a shared load for every jump.
//
// Measured on one B200 (before: the row-tile kernel, which walks the records
// once per jump): pf 4p4n 1.52 -> 0.93 ms FP32, 2.13 -> 1.43 ms FP64; pf 6p6n
// 133 -> 83 ms; sd 6p6n 62 -> 47 us; three-body pf 3p4n 8.4 -> 3.7 ms.  Bound by
// the L1 / shared-memory data path: 82 % of its wavefronts at pf 4p4n FP32, half
// of them the two 16-byte gathers of a record (4 wavefronts at least, about 5
// with conflicts).
//
// Lane l of a warp holds positions 32 s + l, one slice s at a time; every
// position has one owner, so there is no reduction over warps and the order of
// the sum is fixed: bitwise repeatable.
#pragma once

#include "applyh_tile.cuh"

namespace bsg {

// N consecutive elements (aligned to their size, 16 bytes at most) as one or
// two vector accesses
template <typename T, int N>
struct alignas(sizeof(T) * N > 16 ? 16 : sizeof(T) * N) Pack {
    T a[N];
};
template <typename T, int N>
__device__ __forceinline__ Pack<T, N> ldg_pack(const T *p) {
    Pack<T, N> r;
    if constexpr (N == 1) {
        r.a[0] = __ldg(p);
    } else if constexpr (sizeof(T) * N == 8) {
        const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
        r.a[0] = v.x;
        r.a[1] = v.y;
    } else if constexpr (sizeof(T) == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
        r.a[0] = v.x;
        r.a[1] = v.y;
        r.a[2] = v.z;
        r.a[3] = v.w;
    } else {
        const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
        r.a[0] = v.x;
        r.a[1] = v.y;
    }
    return r;
}

__device__ __forceinline__ float flip_sign(float x, unsigned bit31) {
    return __uint_as_float(__float_as_uint(x) ^ bit31);
}
__device__ __forceinline__ double flip_sign(double x, unsigned bit31) {
    return __hiloint2double(__double2hiint(x) ^ (int)bit31, __double2loint(x));
}

// the warps of one part of a CTA: one warp, or all of the CTA (group_shape)
struct Part {
    int id, g, w, lane;    // part, its warps, this warp among them
    __device__ __forceinline__ void sync() const {
        if (g == 1)
            __syncwarp();
        else
            __syncthreads();
    }
};

// one group of J jumps [c, c + J) on one neutron operator, NV vectors at once
template <typename T, int J, int NV>
__device__ __forceinline__ void group_walk(const RowArgs &a, const GroupArgs &g, const Part &pt, const int c, const NOp &op,
                                           const T *__restrict__ vin, const int64_t ld, const int nin, Pack<T, NV> *acc,
                                           T *buf) {
    using VJ = Pack<T, J>;            // the jumps' matrix elements of one label pair
    using XV = Pack<T, NV>;
    // X[n] holds the jumps side by side up to 16 bytes; wider, every jump has
    // an array of its own (32-byte entries would use every other bank group)
    constexpr int JX = sizeof(T) * J * NV > 16 ? 1 : J, NA = J / JX;
    using XJ = Pack<T, JX * NV>;
    const int xs = nin + 1;
    XJ *X = reinterpret_cast<XJ *>(buf);
    VJ *V = reinterpret_cast<VJ *>(X + NA * xs);
    const int tid = pt.w * 32 + pt.lane, nt = pt.g * 32;
    const T *__restrict__ src[J];
    const float *__restrict__ vrow[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const longlong2 q = __ldg(reinterpret_cast<const longlong2 *>(g.jumps) + c + j);
        src[j] = vin + q.x * ld;
        vrow[j] = g.vtab + q.y;
    }
    for (int k = tid; k < op.nbd; k += nt) {
        VJ v;
#pragma unroll
        for (int j = 0; j < J; ++j) v.a[j] = (T)__ldg(vrow[j] + k);
        V[k] = v;
    }
#pragma unroll 2
    for (int n = tid; n < nin; n += nt) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            XJ x;
#pragma unroll
            for (int j = 0; j < JX; ++j) {
                const XV v = ldg_pack<T, NV>(src[i * JX + j] + n * ld);
#pragma unroll
                for (int q = 0; q < NV; ++q) x.a[j * NV + q] = v.a[q];
            }
            X[i * xs + n] = x;
        }
    }
    if (tid < NA) X[tid * xs + nin] = XJ{};   // what the unused record places read
    pt.sync();
    const int32_t *__restrict__ so = a.slice_off + op.slice_base;
    const uint32_t *__restrict__ recs = a.sell32 + op.sell_base + pt.lane;
    const int ns = (op.nout + 31) >> 5;
    for (int sl = pt.w; sl < ns; sl += pt.g) {
        const int o0 = __ldg(so + sl), o1 = __ldg(so + sl + 1);
        const uint32_t *__restrict__ col = recs + o0;
        XV s{};
        auto add = [&](uint32_t r) {
            XJ x[NA];
#pragma unroll
            for (int i = 0; i < NA; ++i) x[i] = X[i * xs + (r & 0xffffu)];
            const VJ v = V[(r >> 16) & 0x7fffu];
            const unsigned sign = r & 0x80000000u;
            if constexpr (NV == 1) {
                T t = x[0].a[0] * v.a[0];
#pragma unroll
                for (int j = 1; j < J; ++j) t = fma(x[j / JX].a[j % JX], v.a[j], t);
                s.a[0] += flip_sign(t, sign);
            } else {
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const T w = flip_sign(v.a[j], sign);
#pragma unroll
                    for (int q = 0; q < NV; ++q) s.a[q] = fma(x[j / JX].a[(j % JX) * NV + q], w, s.a[q]);
                }
            }
        };
        int n = (o1 - o0) >> 5;
        for (; n >= 4; n -= 4, col += 128) {
            uint32_t r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) r[u] = __ldg(col + 32 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) add(r[u]);
        }
        if (n & 2) {
            const uint32_t r0 = __ldg(col), r1 = __ldg(col + 32);
            add(r0);
            add(r1);
            col += 64;
        }
        if (n & 1) add(__ldg(col));
        XV t = acc[sl * 32 + pt.lane];
#pragma unroll
        for (int q = 0; q < NV; ++q) t.a[q] += s.a[q];
        acc[sl * 32 + pt.lane] = t;
    }
    pt.sync();
}

// the most jumps of a group
template <typename T, int NV> constexpr int kGroupJumps = sizeof(T) == 4 && NV == 1 ? 4 : 2;

// One row, NV vectors (consecutive elements; ld elements between positions).
// smem: per part acc[accel] and the staging buffer [bufel] (elements of T).
// The row's work items lie in 8 slots; part p of P takes 8 / P of them and
// keeps its own sums, added in part order at the end.  P follows from the
// context, T and NV, and so do the jumps of a group, so the order of the sum is
// fixed for these three (the single and the batched kernel share it); a block's
// column, or a block on another base (which allows another NV), rounds otherwise.
template <typename T, int NV, int OUT>
__device__ __forceinline__ void row_group(const RowArgs &a, const GroupArgs &g, const int parts, const int row, const int len,
                                          const T *__restrict__ vin, const int64_t ld_, T *__restrict__ vout,
                                          double *__restrict__ cols, T *smem, const int accel, const int bufel) {
    using XV = Pack<T, NV>;
    const int64_t ld = NV == 1 ? ld_ : (ld_ & ~(int64_t)(NV - 1));   // a multiple of NV
    Part pt;
    pt.lane = threadIdx.x & 31;
    pt.g = (blockDim.x >> 5) / parts;
    pt.id = (threadIdx.x >> 5) / pt.g;
    pt.w = (threadIdx.x >> 5) - pt.id * pt.g;
    XV *acc = reinterpret_cast<XV *>(smem + (size_t)pt.id * (accel + bufel));
    T *buf = smem + (size_t)pt.id * (accel + bufel) + accel;
    const int64_t roff = a.row_off[row];
    const int tid = pt.w * 32 + pt.lane, nt = pt.g * 32;
    const int ns = (len + 31) >> 5;
    for (int sl = pt.w; sl < ns; sl += pt.g) acc[sl * 32 + pt.lane] = XV{};
    const int slots = kRowWarps / parts;
    const int32_t *__restrict__ ip = g.item_ptr + row * kRowWarps + pt.id * slots;
    const int i1 = __ldg(ip + slots);
    for (int i = __ldg(ip); i < i1; ++i) {
        const int4 it = __ldg(reinterpret_cast<const int4 *>(g.items) + i);
        const int kind = it.y >> 16, cnt = it.y & 0xffff;
        if (kind == kItemPN) {
            // PN, PPN, PNN (src/bapplyhlibOMP.f90:1242-1442)
            const NOp op = a.nops[it.z];
            if constexpr (kGroupJumps<T, NV> == 4) {
                if (cnt == 4)
                    group_walk<T, 4, NV>(a, g, pt, it.x, op, vin, ld, it.w, acc, buf);
                else if (cnt == 2)
                    group_walk<T, 2, NV>(a, g, pt, it.x, op, vin, ld, it.w, acc, buf);
                else
                    group_walk<T, 1, NV>(a, g, pt, it.x, op, vin, ld, it.w, acc, buf);
            } else {
                int c = it.x;
                for (; c + 2 <= it.x + cnt; c += 2) group_walk<T, 2, NV>(a, g, pt, c, op, vin, ld, it.w, acc, buf);
                if (c < it.x + cnt) group_walk<T, 1, NV>(a, g, pt, c, op, vin, ld, it.w, acc, buf);
            }
        } else if (kind == kItemPP) {
            // PP and PPP (:1068-1241): up to 32 contributions, lane l holds one
            int64_t q = 0;
            float me = 0.f;
            int lo = 0, hi = len - 1;
            if (pt.lane < cnt) {
                const PPContrib pc = a.pp[it.x + pt.lane];
                q = pc.q_off * ld;
                me = pc.me;
                lo = pc.lo;
                hi = pc.hi;
            }
            const bool whole = __all_sync(0xffffffffu, lo == 0 && hi == len - 1);
            for (int sl = pt.w; sl < ns; sl += pt.g) {
                const int pos = sl * 32 + pt.lane;
                const T *__restrict__ xp = vin + min(pos, len - 1) * ld;
                XV s{};
                if (whole) {
#pragma unroll 8
                    for (int k = 0; k < cnt; ++k) {
                        const T mk = (T)__shfl_sync(0xffffffffu, me, k);
                        const XV x = ldg_pack<T, NV>(xp + __shfl_sync(0xffffffffu, q, k));
#pragma unroll
                        for (int v = 0; v < NV; ++v) s.a[v] += mk * x.a[v];
                    }
                } else {
                    for (int k = 0; k < cnt; ++k) {
                        const int lk = __shfl_sync(0xffffffffu, lo, k), hk = __shfl_sync(0xffffffffu, hi, k);
                        const T mk = (T)__shfl_sync(0xffffffffu, me, k);
                        const int64_t qk = __shfl_sync(0xffffffffu, q, k);
                        if (pos >= lk && pos <= hk) {
                            const XV x = ldg_pack<T, NV>(xp + qk);
#pragma unroll
                            for (int v = 0; v < NV; ++v) s.a[v] += mk * x.a[v];
                        }
                    }
                }
                XV t = acc[pos];
#pragma unroll
                for (int v = 0; v < NV; ++v) t.a[v] += s.a[v];
                acc[pos] = t;
            }
        } else if (kind == kItemNN) {
            // NN and NNN (:1012-1066): share cnt of it.w of every position's
            // records, the row itself staged for the gathers
            const NOp op = a.nops[it.z];
            XV *xs = reinterpret_cast<XV *>(buf);
            for (int e = tid; e < len; e += nt) xs[e] = ldg_pack<T, NV>(vin + (roff + e) * ld);
            if (tid == 0) xs[g.zero_pos] = XV{};   // what the unused record places read
            pt.sync();
            const int32_t *__restrict__ so = a.slice_off + op.slice_base;
            for (int sl = pt.w; sl * 32 < op.nout; sl += pt.g) {
                const int o0 = __ldg(so + sl), n = (__ldg(so + sl + 1) - o0) >> 5;
                int k = n * cnt / it.w;
                const int ke = n * (cnt + 1) / it.w;
                const int2 *__restrict__ col = a.sell + op.sell_base + o0 + pt.lane + 32 * k;
                XV s{};
                auto add = [&](int2 r) {
                    const XV x = xs[r.x];
                    const T m = (T)__int_as_float(r.y);
#pragma unroll
                    for (int v = 0; v < NV; ++v) s.a[v] += m * x.a[v];
                };
                for (; k + 4 <= ke; k += 4, col += 128) {
                    int2 r[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) r[u] = __ldg(col + 32 * u);
#pragma unroll
                    for (int u = 0; u < 4; ++u) add(r[u]);
                }
                for (; k < ke; ++k, col += 32) add(__ldg(col));
                XV t = acc[sl * 32 + pt.lane];
#pragma unroll
                for (int v = 0; v < NV; ++v) t.a[v] += s.a[v];
                acc[sl * 32 + pt.lane] = t;
            }
            pt.sync();
        } else {
            // SPE (:988-1011)
            const SPEContrib sc = a.spe[it.x];
            for (int sl = pt.w; sl < ns; sl += pt.g) {
                const int pos = sl * 32 + pt.lane;
                if (pos >= sc.lo && pos <= sc.hi) {
                    const T e = (T)(sc.pspe + __ldg(a.nspe + sc.n0 + (pos - sc.lo)));
                    const XV x = ldg_pack<T, NV>(vin + (roff + pos) * ld);
#pragma unroll
                    for (int v = 0; v < NV; ++v) acc[pos].a[v] += x.a[v] * e;
                }
            }
        }
    }
    __syncthreads();
    // ---- the parts in order, a single write per element
    for (int e = threadIdx.x; e < len * NV; e += blockDim.x) {
        T s = smem[e];
        for (int p = 1; p < parts; ++p) s += smem[(size_t)p * (accel + bufel) + e];
        if constexpr (OUT == kColumns) {
            // consecutive threads take one column where there is one vector
            cols[(int64_t)(e % NV) * a.cols_ld + roff + e / NV] = (double)s;
        } else {
            T *o = vout + (roff + e / NV) * ld_ + e % NV;
            if constexpr (OUT == kAccumulate)
                *o = *o + s;
            else
                *o = s;
        }
    }
}

}  // namespace bsg
