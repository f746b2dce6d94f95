// applyH on jump groups: kernel, launch and table set-up (rowgroup.cuh has
// the row body and the reason for the form).

#include <algorithm>
#include <type_traits>
#include <vector>

#include "host_parallel.h"
#include "rowgroup.cuh"
#include "rowgroup.h"

namespace bsg {

namespace {

// one CTA per row and NV of the block's vectors, heaviest rows first, a row's
// vectors next to each other (they share the records and, where the vectors
// are interleaved, the sectors).  FORM: up to 256 threads with 64 registers, so that
// 32 warps stay resident per SM; up to 1024 threads; or, for single vectors on many
// rows of a few positions, 256 threads with 40 registers and 48 warps: there a CTA
// waits on one short chain of loads, and more rows at once outweigh the spills
// (60 bytes at most).  Calls with 64 / 40 / 32 registers: sd 6p2n FP64 33.6 / 28.9 /
// 30.7 us, FP32 29.7 / 25.6 / 27.0, pf 5p1n FP64 247 / 214 / 212, FP32 191 / 172 / 169;
// but pf 3p2n (rows of 23) FP32 34.0 / 38.0 / 35.2, sd 4p2n (all rows at once anyway)
// 24.5 / 25.6 / 28.1.
enum RowForm { kSmallCta = 0, kBigCta = 1, kManyCtas = 2 };
template <typename T, int NV, int OUT, int FORM>
__global__ void __launch_bounds__(FORM == kBigCta ? 1024 : 256, FORM == kBigCta ? 1 : (FORM == kManyCtas ? 6 : 4))
    k_rowgroup(const RowArgs a, const GroupArgs g, const int parts, const T *__restrict__ vin, const int64_t ld,
               T *__restrict__ vout, const int accel, const int bufel, const int ngrp) {
    extern __shared__ __align__(16) unsigned char smem[];
    const Tile t = a.tiles[blockIdx.x / ngrp];
    const int64_t v = ngrp == 1 ? 0 : (int64_t)(blockIdx.x % ngrp) * NV;
    row_group<T, NV, OUT>(a, g, parts, t.row, t.npos, vin + v, ld, vout + v,
                          OUT == kColumns ? a.cols_out + v * a.cols_ld : nullptr, reinterpret_cast<T *>(smem), accel, bufel);
}

// CTAs of 256 threads and 64 registers that fit at once
constexpr int64_t kGroupWave = 148 * 4;

struct VKey {
    int32_t nop, aoff, coff;
    float php;
};

// matrix-element rows: hmat(cpn[b + aoff] + dpn[d + coff]) * php for the
// operator's label pairs, as the row kernels tabulate them per jump
__global__ void k_vrows(const RowArgs a, const VKey *__restrict__ key, const int64_t *__restrict__ base, int n,
                        float *__restrict__ v) {
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const VKey k = key[i];
        const NOp op = a.nops[k.nop];
        for (int q = lane; q < op.nbd; q += 32) {
            const BDPair bd = a.bd[op.bd_base + q];
            v[base[i] + q] = a.hmatpn[a.cpn[bd.b + k.aoff] + a.dpn[bd.d + k.coff] - 1] * k.php;
        }
    }
}

template <typename T, int NV, int OUT, int FORM>
int launch_k(bsg_ctx *ctx, const GroupShape &sh, const T *vin, T *vout, int nb, cudaStream_t s, const TileSet *ts,
             double *cols) {
    RowArgs a = ctx->args;
    a.tiles = (const Tile *)ts->buf.p;
    a.ntiles = ts->ntiles;
    a.cols_out = cols;
    a.cols_ld = ctx->dim;
    auto k = k_rowgroup<T, NV, OUT, FORM>;
    // the attribute belongs to the function, not the context: set to the
    // limit once, so that contexts of different sizes do not undo one another's
    size_t &cur = ctx->smem_allowed[(const void *)k];
    if (cur == 0) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGroupSmemMax);
        if (e != cudaSuccess) return cuda_check(ctx, e, "applyh smem attribute");
        cur = kGroupSmemMax;
    }
    k<<<(unsigned)ts->ntiles * (unsigned)(nb / NV), sh.threads, sh.bytes(sizeof(T)), s>>>(
        a, ctx->group, sh.parts, vin, (int64_t)nb, vout, sh.accel, sh.bufel, nb / NV);
    return cuda_check(ctx, cudaGetLastError(), "applyh kernel launch");
}

// rows of at most half a slice, more of them than CTAs of 64 registers fit at once
bool many_short_rows(const bsg_ctx *ctx) { return ctx->median_rowlen <= 16 && ctx->nrows > kGroupWave; }

template <typename T, int NV>
int launch_v(bsg_ctx *ctx, const T *vin, T *vout, int nb, int accumulate, cudaStream_t s, const TileSet *ts, double *cols) {
    const GroupShape sh = group_shape(ctx, sizeof(T), NV);
    auto go = [&](auto f) {
        constexpr int F = decltype(f)::value;
        if (cols) return launch_k<T, NV, kColumns, F>(ctx, sh, vin, vout, nb, s, ts, cols);
        if (accumulate) return launch_k<T, NV, kAccumulate, F>(ctx, sh, vin, vout, nb, s, ts, cols);
        return launch_k<T, NV, kStore, F>(ctx, sh, vin, vout, nb, s, ts, cols);
    };
    if (sh.threads > 256) return go(std::integral_constant<int, kBigCta>{});
    if constexpr (NV == 1)
        if (nb == 1 && many_short_rows(ctx)) return go(std::integral_constant<int, kManyCtas>{});
    return go(std::integral_constant<int, kSmallCta>{});
}

template <typename T>
int launch_t(bsg_ctx *ctx, const T *vin, T *vout, int nb, int accumulate, cudaStream_t s, TileLookup lookup, double *cols) {
    ctx->last_status = BSG_OK;
    const TileSet *ts = lookup ? lookup(ctx, kRowTile) : get_tiles(ctx, kRowTile);
    if (!ts) return ctx->last_status ? ctx->last_status : BSG_ERR_NOMEM;
    if (ts->ntiles == 0) return BSG_OK;
    // as many vectors at once as a 16-byte load takes, where the block's
    // layout and base allow it and the row's sums and staging fit
    auto fits = [&](int nv) {
        return nb % nv == 0 && (reinterpret_cast<uintptr_t>(vin) & (nv * sizeof(T) - 1)) == 0 &&
               group_shape(ctx, sizeof(T), nv).bytes(sizeof(T)) <= kGroupSmemMax;
    };
    if constexpr (sizeof(T) == 4)
        if (fits(4)) return launch_v<T, 4>(ctx, vin, vout, nb, accumulate, s, ts, cols);
    if (fits(2)) return launch_v<T, 2>(ctx, vin, vout, nb, accumulate, s, ts, cols);
    return launch_v<T, 1>(ctx, vin, vout, nb, accumulate, s, ts, cols);
}

}  // namespace

// P parts of G warps: rows short enough that 8 parts of one warp each leave
// room for 4 CTAs, or of 5 slices at most, take those (no barrier but the last;
// sd 6p6n FP32 46.9 us against 67.6 as one part of 4 warps; three-body pf 2p3n,
// 2 CTAs, 225 us against 420 as two parts of 4 warps), longer ones one part of
// as many warps as make 32 per SM (pf 4p4n FP64 1.43 ms at 4 warps, 3.50 as 8
// parts).
GroupShape group_shape(const bsg_ctx *ctx, int esize, int nv) {
    GroupShape r;
    const int64_t j = esize == 4 && nv == 1 ? 4 : 2;
    r.accel = ((ctx->max_rowlen + 31) & ~31) * nv;
    r.bufel = (int)((std::max<int64_t>(j * ctx->group_nbd + j * nv * (ctx->group_nin + 1), (int64_t)nv * (ctx->max_rowlen + 1)) + 3) &
                    ~(int64_t)3);
    const size_t b = r.part_bytes(esize);
    const size_t one = nv == 1 ? b : group_shape(ctx, esize, 1).part_bytes(esize);
    r.parts = (8 * one <= 50 * 1024 || ctx->max_rowlen <= 160) && 8 * b <= kGroupSmemMax ? 8 : 1;
    r.threads = r.parts == 8 ? 256 : (b > 113 * 1024 ? 1024 : (b > 56 * 1024 ? 512 : (b > 28 * 1024 ? 256 : 128)));
    return r;
}

// The row-tile kernel takes a whole block in one walk, the jump groups nb / NV
// walks, so which is faster depends on the block and the rows.  Both timed on one
// B200 over sd 1p1n ... 8p8n and pf 1p1n ... 8p1n, 3p6n; figures are row-tile time /
// jump-group time.
//  - Single vectors: the groups, 1.02 - 2.6 (0.93 - 1.1 on many rows of a few
//    positions, sd 5p1n ... 7p2n FP64 with 48 warps to an SM; a batch of such systems
//    is 1.3 - 2 times faster on the groups, and a member has the bits of the same
//    system alone).
//  - Long rows (one part): the groups, at least 1.13 for FP32 and 1.03 for FP64
//    blocks (rows of 390 to 3,500).
//  - Pairs on rows of at most half a slice, more of them than CTAs fit at once: the
//    row tiles (0.77 - 0.95).  There a CTA is mostly start and end.
//  - Odd blocks and those below one 16-byte load: the groups (the row tiles split
//    odd blocks: 0.97 - 9).
//  - Powers of two from one 16-byte load up, short rows: a median of 64 and less
//    the row tiles (FP64 nb = 8 down to 0.46, FP32 nb = 16 the same) but for pairs;
//    above, the row tiles at two loads (FP32 nb = 8 0.94 - 1.07, FP64 nb = 4 0.90 -
//    1.03) and, where the rows fill the chip twice, at four (pf 4p3n ... 6p3n: FP64
//    nb = 8 0.95 - 0.97, FP32 nb = 16 0.97 - 0.99; pf 3p3n, 1,140 rows, 1.02; sd
//    1.01 - 1.14); the groups elsewhere (FP32 nb = 4 1.05 - 1.5, FP64 nb = 16 1.09 -
//    2).  Spaces of few rows scatter: sd 2p6n (66 rows) loses at FP32 nb = 16 (0.78)
//    what sd 2p8n gains (1.26), sd 3p6n (220) at nb = 4 (0.94) what sd 3p7n (1.21).
bool group_takes(const bsg_ctx *ctx, int nb, int prec) {
    if (!ctx->grouped) return false;
    if (nb == 1 || group_shape(ctx, prec, 1).parts == 1) return true;
    const int nv = 16 / prec;
    if (nb == 2 && many_short_rows(ctx)) return false;
    if (nb < nv || (nb & (nb - 1)) || nb > 16) return true;
    if (ctx->median_rowlen <= 64) return nb == 2;
    return nb != 2 * nv && (nb != 4 * nv || ctx->nrows <= 2 * kGroupWave);
}

int launch_rowgroup(bsg_ctx *ctx, const void *vin, void *vout, int nb, int prec, int accumulate, cudaStream_t s,
                    TileLookup lookup, double *cols) {
    if (prec == BSG_PREC_FP32) return launch_t<float>(ctx, (const float *)vin, (float *)vout, nb, accumulate, s, lookup, cols);
    return launch_t<double>(ctx, (const double *)vin, (double *)vout, nb, accumulate, s, lookup, cols);
}

bool group_eligible(bsg_ctx *ctx, const GroupSource &S, bool pack32) {
    if (!pack32 || S.pn.empty()) return false;
    ctx->group_nbd = ctx->group_nin = 0;
    for (size_t o = 0; o < S.nops.size(); ++o)
        if (S.nops[o].kind == 1) {
            ctx->group_nbd = std::max<int64_t>(ctx->group_nbd, S.nops[o].nbd);
            ctx->group_nin = std::max<int64_t>(ctx->group_nin, S.nop_maxin[o] + 1);
        }
    // unused record places read a zero input and the operator's first element: an
    // infinite one would reach positions that it does not couple.  (A zero element
    // of their own, staged for each group, costs 3 % on three-body pf 2p3n FP64.)
    if (!S.finite) return false;
    // a record has 16 bits for the position, one past the operator's own inputs for
    // the unused places
    if (ctx->max_rowlen > 65535) return false;
    // few long rows (one CTA of a few warps each) do not fill the chip, where
    // the row-tile kernel cuts them (pf 2p4n, 190 rows: FP64 159 us against 88)
    for (int esize : {4, 8}) {
        const GroupShape sh = group_shape(ctx, esize, 1);
        if (sh.bytes(esize) > kGroupSmemMax || (sh.parts == 1 && ctx->nrows < 512)) return false;
    }
    return true;
}

int build_groups(bsg_ctx *ctx, const GroupSource &S, int nthr) {
    const std::vector<NOp> &nops = S.nops;
    auto &pn = S.pn;
    // ---- matrix-element rows: one per distinct (operator, proton labels,
    // phase).  Operators are dealt to NT tasks; each walks all jumps and keeps
    // the keys of its own operators, numbered by themselves
    const int NT = nthr > 1 ? 8 : 1;
    std::vector<std::vector<VKey>> tkeys(NT);
    std::vector<std::vector<int64_t>> tbase(NT);
    std::vector<int64_t> ttot(NT + 1, 0);
    std::vector<GroupJump> jumps(pn.size());
    parallel_for(NT, 1, [&](int64_t task) {
        // the keys of one operator: open addressing on (aoff, coff, phase)
        struct Slot { int32_t aoff, coff, php; int64_t base; };
        std::vector<std::vector<Slot>> tab((nops.size() + NT - 1) / NT);
        std::vector<int32_t> used(tab.size(), 0);
        auto &keys = tkeys[task];
        auto &base = tbase[task];
        int64_t &tot = ttot[task + 1];
        auto find = [](std::vector<Slot> &t, int32_t x, int32_t y, int32_t z) -> Slot & {
            const uint32_t mask = (uint32_t)t.size() - 1;
            uint32_t h = ((uint32_t)x * 2654435761u ^ (uint32_t)y * 2246822519u ^ (uint32_t)z * 3266489917u) >> 7 & mask;
            while (t[h].base >= 0 && !(t[h].aoff == x && t[h].coff == y && t[h].php == z)) h = (h + 1) & mask;
            return t[h];
        };
        for (size_t i = 0; i < pn.size(); ++i) {
            const PNContrib &c = pn[i].second;
            if (c.nop % NT != task) continue;
            auto &t = tab[c.nop / NT];
            if (t.empty()) t.assign(64, Slot{0, 0, 0, -1});
            const int32_t ph = c.php < 0 ? -1 : 1;
            Slot *s = &find(t, c.aoff, c.coff, ph);
            if (s->base < 0) {
                if ((size_t)++used[c.nop / NT] * 2 > t.size()) {
                    std::vector<Slot> old(t.size() * 2, Slot{0, 0, 0, -1});
                    old.swap(t);
                    for (const Slot &q : old)
                        if (q.base >= 0) find(t, q.aoff, q.coff, q.php) = q;
                    s = &find(t, c.aoff, c.coff, ph);
                }
                *s = Slot{c.aoff, c.coff, ph, tot};
                keys.push_back(VKey{c.nop, c.aoff, c.coff, c.php});
                base.push_back(tot);
                tot += nops[c.nop].nbd;
            }
            jumps[i] = GroupJump{c.q_off, s->base};
        }
    }, nthr);
    for (int t = 0; t < NT; ++t) ttot[t + 1] += ttot[t];
    const int64_t vtot = ttot[NT];
    std::vector<VKey> keys;
    std::vector<int64_t> vbase;
    for (int t = 0; t < NT; ++t) {
        keys.insert(keys.end(), tkeys[t].begin(), tkeys[t].end());
        for (int64_t b : tbase[t]) vbase.push_back(b + ttot[t]);
    }
    if (NT > 1)
        parallel_for((int64_t)pn.size(), 1 << 15, [&](int64_t i) { jumps[i].v += ttot[pn[i].second.nop % NT]; }, nthr);
    // ---- work items: per row and operator the jumps in fours, then a two and
    // a one; the PP contributions in 32s; every NN operator in shares of about
    // 24 records a position.  A row's items go to 8 slots, longest first to the
    // least loaded; weights are estimated L1 / shared-memory cycles.
    const bool spread = group_shape(ctx, 4, 1).parts > 1;
    const int64_t nrows = ctx->nrows;
    std::vector<int64_t> rs(nrows + 1, 0);
    for (auto &e : pn) rs[e.first + 1]++;
    for (int64_t r = 0; r < nrows; ++r) rs[r + 1] += rs[r];
    std::vector<int32_t> iptr((size_t)nrows * kRowWarps + 1, 0);
    auto nrec = [&](int32_t o) -> int64_t { return S.nptr[nops[o].ptr_base + nops[o].nout]; };
    struct Wt { int64_t w; GroupItem it; };
    auto row_items = [&](int64_t r, std::vector<Wt> &v) {
        v.clear();
        const int64_t len = ctx->h_rowlen[r];
        for (int64_t i = rs[r]; i < rs[r + 1];) {
            const int32_t o = pn[i].second.nop;
            int64_t e = i;
            while (e < rs[r + 1] && pn[e].second.nop == o) ++e;
            while (i < e) {
                const int j = e - i >= 4 ? 4 : (e - i >= 2 ? 2 : 1);
                v.push_back(Wt{nrec(o) * (j == 4 ? 17 : (j == 2 ? 10 : 9)) + (int64_t)(S.nop_maxin[o] + 1) * (4 + 2 * j) + 600,
                               GroupItem{(int32_t)i, kItemPN << 16 | j, o, S.nop_maxin[o] + 1}});
                i += j;
            }
        }
        const int32_t pp0 = ctx->h_pp_ptr[r * kRowWarps], pp1 = ctx->h_pp_ptr[(r + 1) * kRowWarps];
        for (int32_t c = pp0; c < pp1; c += 32) {
            const int32_t m = std::min(32, pp1 - c);
            v.push_back(Wt{len * m * 5 / 2 + 300, GroupItem{c, kItemPP << 16 | m, 0, 0}});
        }
        for (int32_t c = ctx->h_nn_ptr[r * kRowWarps]; c < ctx->h_nn_ptr[(r + 1) * kRowWarps]; ++c) {
            const int32_t o = ctx->h_nn[c].nop;
            const int32_t sh = !spread ? 1 : (int32_t)std::max<int64_t>(1, std::min<int64_t>(16, nrec(o) / (24 * (int64_t)nops[o].nout + 1) + 1));
            for (int32_t k = 0; k < sh; ++k)
                v.push_back(Wt{nrec(o) * 8 / sh + 600, GroupItem{0, kItemNN << 16 | k, o, sh}});
        }
        for (int32_t c = S.spe_ptr[r * kRowWarps]; c < S.spe_ptr[(r + 1) * kRowWarps]; ++c)
            v.push_back(Wt{len * 4, GroupItem{c, kItemSPE << 16, 0, 0}});
    };
    parallel_for(nrows, 256, [&](int64_t r) {
        thread_local std::vector<Wt> v;
        row_items(r, v);
        iptr[(r + 1) * kRowWarps] = (int32_t)v.size();
    }, nthr);
    {
        int64_t tot = 0;
        for (int64_t r = 0; r < nrows; ++r) {
            tot += iptr[(r + 1) * kRowWarps];
            if (tot > INT32_MAX) return set_err(ctx, BSG_ERR_UNSUPPORTED, "more than 2^31 row items");
            iptr[(r + 1) * kRowWarps] = (int32_t)tot;
        }
    }
    std::vector<GroupItem> items((size_t)iptr[nrows * kRowWarps]);
    parallel_for(nrows, 256, [&](int64_t r) {
        thread_local std::vector<Wt> v;
        thread_local std::vector<std::pair<int64_t, int32_t>> ord;
        thread_local std::vector<uint8_t> slot;
        row_items(r, v);
        slot.assign(v.size(), 0);
        if (spread) {
            ord.resize(v.size());
            for (size_t k = 0; k < v.size(); ++k) ord[k] = {-v[k].w, (int32_t)k};
            std::sort(ord.begin(), ord.end());
            int64_t load[kRowWarps] = {0};
            for (auto &o : ord) {
                int best = 0;
                for (int w = 1; w < kRowWarps; ++w)
                    if (load[w] < load[best]) best = w;
                load[best] += v[o.second].w;
                slot[o.second] = (uint8_t)best;
            }
        } else {
            int64_t tot = 0, at = 0;
            for (auto &x : v) tot += x.w;
            for (size_t k = 0; k < v.size(); ++k) {
                slot[k] = (uint8_t)std::min<int64_t>(kRowWarps - 1, (2 * at + v[k].w) * kRowWarps / (2 * std::max<int64_t>(tot, 1)));
                at += v[k].w;
            }
        }
        int32_t at = iptr[r * kRowWarps];
        for (int w = 0; w < kRowWarps; ++w) {
            if (w) iptr[r * kRowWarps + w] = at;
            for (size_t k = 0; k < v.size(); ++k)
                if (slot[k] == w) items[at++] = v[k].it;
        }
    }, nthr);
    // ---- one allocation: jumps, items, slots, keys and bases, the rows
    auto at16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const size_t b_jump = sizeof(GroupJump) * jumps.size(), b_item = sizeof(GroupItem) * items.size(),
                 b_iptr = at16(4 * iptr.size()), b_key = sizeof(VKey) * keys.size(), b_base = at16(8 * vbase.size());
    int st = dev_alloc(ctx, ctx->g_buf, b_jump + b_item + b_iptr + b_key + b_base + (size_t)vtot * sizeof(float));
    if (st) return st;
    char *p = (char *)ctx->g_buf.p;
    auto put = [&](const void *src, size_t bytes, size_t room) {
        char *at = p;
        if (!st && bytes) st = cuda_check(ctx, cudaMemcpy(at, src, bytes, cudaMemcpyHostToDevice), "upload");
        p += room;
        return at;
    };
    ctx->group.jumps = (const GroupJump *)put(jumps.data(), b_jump, b_jump);
    ctx->group.items = (const GroupItem *)put(items.data(), b_item, b_item);
    ctx->group.item_ptr = (const int32_t *)put(iptr.data(), 4 * iptr.size(), b_iptr);
    const VKey *kd = (const VKey *)put(keys.data(), b_key, b_key);
    const int64_t *bd = (const int64_t *)put(vbase.data(), 8 * vbase.size(), b_base);
    float *vd = (float *)p;
    ctx->group.vtab = vd;
    ctx->group.zero_pos = ctx->max_rowlen;
    if (st) return st;
    // on the default stream, after the uploads
    const int n = (int)keys.size();
    k_vrows<<<std::max(1, std::min(1184, (n + 7) / 8)), 256>>>(ctx->args, kd, bd, n, vd);
    st = cuda_check(ctx, cudaGetLastError(), "matrix-element rows launch");
    if (!st) st = cuda_check(ctx, cudaStreamSynchronize(nullptr), "matrix-element rows sync");
    if (st) return st;
    ctx->stats.derived_bytes += (int64_t)ctx->g_buf.bytes;
    ctx->grouped = true;
    return BSG_OK;
}

void free_groups(bsg_ctx *ctx) {
    dev_free(ctx->g_buf);
    ctx->group = GroupArgs{};
    ctx->grouped = false;
}

}  // namespace bsg
