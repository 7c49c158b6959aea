// Which rows of a tree a product computes from all of their entries instead of from their parent's row (host).
#pragma once
#include <cstdint>
#include <vector>

namespace cbm {

struct Lifted {
    int32_t n_lifted = 0;                // 0: the tree stays as it is, and nothing below is set
    std::vector<int32_t> parent, level;  // of every row, in the tree with the lifted rows under the virtual root
    std::vector<int32_t> len;            // entries of every row there
    std::vector<int64_t> at;             // their place: in the caller's arrays, or, of a lifted row, in col and val
    std::vector<char> lifted;
    std::vector<int32_t> col;
    std::vector<float> val;
    int64_t n_entries = 0;  // of all rows in `order`
};

// `order`: the rows a plan computes, parents first; parent[v] == n: a child of the virtual root.
void lift_rows(int32_t n, const std::vector<int32_t>& order, const std::vector<int32_t>& parent,
               const std::vector<int32_t>& level, const int32_t* crow, const int32_t* col, const float* val, Lifted& out);

}  // namespace cbm
