// Set-up and launch of the jump-group row kernel (rowgroup.cu).
#pragma once

#include <utility>
#include <vector>

#include "bsg_internal.h"

namespace bsg {

// one tile per row
constexpr int kRowTile = 1 << 24;
constexpr size_t kGroupSmemMax = 226 * 1024;

// what the groups are built from: pn sorted by (row, operator)
struct GroupSource {
    const std::vector<NOp> &nops;
    const std::vector<int32_t> &nop_maxin;
    const std::vector<int32_t> &nptr;
    const std::vector<int32_t> &spe_ptr;
    const std::vector<std::pair<int32_t, PNContrib>> &pn;
    bool finite;   // every element of hmatpn (hmatppn, hmatpnn) is
};
// whether the context takes the jump-group kernel
bool group_eligible(bsg_ctx *ctx, const GroupSource &S, bool pack32);
// BSG_ERR_NOMEM, BSG_ERR_UNSUPPORTED (or std::bad_alloc): the context has none
int build_groups(bsg_ctx *ctx, const GroupSource &S, int nthr);
void free_groups(bsg_ctx *ctx);

// shared memory and threads of one CTA on nv vectors
struct GroupShape {
    int accel, bufel;    // of a part: sums and staging, elements of T
    int parts = 1, threads;
    size_t part_bytes(int esize) const { return (size_t)(accel + bufel) * esize; }
    size_t bytes(int esize) const { return part_bytes(esize) * parts; }
};
GroupShape group_shape(const bsg_ctx *ctx, int esize, int nv);

}  // namespace bsg
