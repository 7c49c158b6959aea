// Lifting rows out of the tree, for the product that gathers and updates in one pass.
//
// A row under a parent has fewer entries than the whole row, but it waits for its parent, and a product of a small graph is
// nothing but the chain of those waits.  The tree that the builder emits is the one with the fewest entries, so a row
// hangs under a parent for a saving of one entry as for one of a hundred; on most graphs nearly all savings are of
// the first kind (a copy-model graph of 4 096 rows: 2 800 rows in 12 levels below the first save 12 300 of 86 000 entries).  A
// whole row is its parent's whole row with the row's own entries merged in, so it can be had from the structure alone.
// Here rows whose saving is not worth a wait are hung under the virtual root with all their entries.
// 1 000 rows, 16 columns 11.8 -> 8.2 us, 4 096 rows, 500 columns 38.7 -> 32.0, 400 000 community rows, 47 columns 266 -> 251;
// a structure that does compress (40 000 rows of 152 entries, 17 % saved) lifts the tenth of its rows that saves least and
// measures the same, 201 us (207 with every row lifted).
#include "cbm_lift.h"

#include <algorithm>

namespace cbm {
namespace {

using i32 = int32_t;
using i64 = int64_t;

// What a waiting row and a level of the tree cost beside the entries, in entries.  A wait is some trips to L2 (flag, parent
// row, flag), each as long as a batch of fetches; a level about 1.2 us of the chain, in which the GPU gathers 20 000 to
// 40 000 row pieces of 512 bytes.  For operands of up to 128 columns, that is; wider products choose between the two
// schedules by their width (cbm_b200_plan::tree_pays).
constexpr i64 WAIT_COST = 8, LEVEL_COST = 20000;
constexpr i64 LONGEST = 1 << 20;  // lifted rows stay well below what a schedule can cut into segments

// The row's entries merged into its parent's whole row; false where the result is not a whole row exactly: columns not
// ascending, a column of both that does not cancel, more or fewer entries than counted.
bool merge(const i32* pc, const float* pv, i64 np, const i32* dc, const float* dv, i64 nd, i32* col, float* val, i64 want) {
    i64 i = 0, j = 0, out = 0;
    for (i64 k = 1; k < nd; ++k)
        if (dc[k - 1] >= dc[k]) return false;
    while (i < np || j < nd) {
        if (i < np && j < nd && pc[i] == dc[j]) {
            if (pv[i++] + dv[j++] != 0.0f) return false;
            continue;
        }
        if (out == want) return false;
        const bool from_parent = j == nd || (i < np && pc[i] < dc[j]);
        col[out] = from_parent ? pc[i] : dc[j];
        val[out++] = from_parent ? pv[i++] : dv[j++];
    }
    return out == want;
}

}  // namespace

void lift_rows(i32 n, const std::vector<i32>& order, const std::vector<i32>& parent, const std::vector<i32>& level,
               const i32* crow, const i32* col, const float* val, Lifted& out) {
    const i32 rows = (i32)order.size();
    i32 first = 0;  // the rows before it, breadth-first, are children of the virtual root
    i64 entries = 0;
    for (i32 v : order) entries += crow[v + 1] - crow[v];
    while (first < rows && parent[order[first]] == n) ++first;
    if (first == rows) return;

    // length of every whole row: an entry with a minus takes one of the parent's away
    std::vector<i32> taken((size_t)n, 0);
    std::vector<i64> whole((size_t)n + 1, 0);
#pragma omp parallel for schedule(dynamic, 512) if (entries > 200000)
    for (i32 k = first; k < rows; ++k) {
        const i32 v = order[k];
        i32 minus = 0;
        for (i32 e = crow[v]; e < crow[v + 1]; ++e) minus += val[e] < 0.0f;
        taken[v] = minus;
    }
    for (i32 v : order) {
        const i64 len = crow[v + 1] - crow[v];
        whole[v] = parent[v] == n ? len : whole[parent[v]] + len - 2 * (i64)taken[v];
        if (whole[v] < 0 || whole[v] > n) return;  // not a pattern with signs
    }
    const auto saves = [&](i32 v) { return whole[v] - (crow[v + 1] - crow[v]); };
    const auto lifts = [&](i32 v, i64 limit) { return saves(v) <= limit && whole[v] <= LONGEST; };

    // The saving up to which rows are lifted: the one with which entries, waits and levels together cost least.
    constexpr i64 ALL = (i64)1 << 40, NEVER = -ALL;
    i64 least = 0, limit = NEVER;
    std::vector<i32> lev((size_t)n + 1, 0), needed((size_t)n, -1);
    i32 round = 0;
    for (i32 k = 0; k < first; ++k) lev[order[k]] = 1;
    for (const i64 s : {NEVER, (i64)0, (i64)4, (i64)8, (i64)16, (i64)32, (i64)64, (i64)128, ALL}) {
        i64 extra = 0, waits = 0, buffer = 0;
        i32 depth = 1;
        ++round;
        for (i32 k = first; k < rows; ++k) {
            const i32 v = order[k];
            if (lifts(v, s)) {
                extra += saves(v);
                lev[v] = 1;
                for (i32 u = v; parent[u] != n && needed[u] != round; u = parent[u]) {
                    needed[u] = round;
                    buffer += whole[u];
                }
            } else {
                ++waits;
                lev[v] = lev[parent[v]] + 1;
                depth = std::max(depth, lev[v]);
            }
        }
        // (whole rows that are needed on the way only must not outgrow the structure, as on a chain of nested rows)
        if (buffer > 2 * entries + 65536 || entries + extra + n + 1024 > INT32_MAX) break;
        const i64 cost = entries + extra + WAIT_COST * waits + (depth > 1 ? LEVEL_COST * depth : 0);
        if (s == NEVER || cost < least) {
            least = cost;
            limit = s;
        }
    }
    if (limit == NEVER) return;

    std::vector<i64> place((size_t)n, -1);
    i64 room = 0;
    std::vector<char> lifted((size_t)n, 0);
    for (i32 k = first; k < rows; ++k) {
        const i32 v = order[k];
        if (!lifts(v, limit)) continue;
        lifted[v] = 1;
        ++out.n_lifted;
        for (i32 u = v; parent[u] != n && place[u] < 0; u = parent[u]) place[u] = 0;
    }
    for (i32 k = first; k < rows; ++k)
        if (place[order[k]] == 0) {
            place[order[k]] = room;
            room += whole[order[k]];
        }
    out.col.resize((size_t)room);
    out.val.resize((size_t)room);
    // level by level: a level's rows need only those above them
    bool whole_rows = true;
    for (i32 k0 = first, k1; k0 < rows && whole_rows; k0 = k1) {
        for (k1 = k0; k1 < rows && level[order[k1]] == level[order[k0]];) ++k1;
#pragma omp parallel for schedule(dynamic, 256) reduction(&& : whole_rows) if (k1 - k0 > 4096)
        for (i32 k = k0; k < k1; ++k) {
            const i32 v = order[k], u = parent[v];
            if (place[v] < 0) continue;
            const bool top = parent[u] == n;
            const i32* pc = top ? col + crow[u] : out.col.data() + place[u];
            const float* pv = top ? val + crow[u] : out.val.data() + place[u];
            bool ascending = true;
            for (i64 e = 1; top && e < whole[u]; ++e) ascending = ascending && pc[e - 1] < pc[e];
            whole_rows = whole_rows && ascending &&
                         merge(pc, pv, whole[u], col + crow[v], val + crow[v], crow[v + 1] - crow[v], out.col.data() + place[v],
                               out.val.data() + place[v], whole[v]);
        }
    }
    if (!whole_rows) {
        out = Lifted();
        return;
    }
    out.parent = parent;
    out.level = level;
    out.len.resize((size_t)n);
    out.at.resize((size_t)n);
    for (i32 v = 0; v < n; ++v) {
        out.len[v] = crow[v + 1] - crow[v];
        out.at[v] = crow[v];
    }
    for (i32 k = first; k < rows; ++k) {
        const i32 v = order[k];
        if (lifted[v]) {
            out.parent[v] = n;
            out.level[v] = 1;
            out.len[v] = (i32)whole[v];
            out.at[v] = place[v];
        } else {
            out.level[v] = out.level[parent[v]] + 1;
        }
    }
    out.lifted.swap(lifted);
    for (i32 v : order) out.n_entries += out.len[v];
}

}  // namespace cbm
