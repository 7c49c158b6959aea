// Groups rows that name the same columns (cbm_cluster.cu).
#ifndef CBM_CLUSTER_H
#define CBM_CLUSTER_H

#include <cstdint>

namespace cbm {

// label[v], in [0, n), for each of the n rows of the pattern (crow, col; parent[v] counts as one more column, n = none; columns
// from n on are passed over), found on GPU `device` by label propagation.  Rows of one community come out with one label.  Returns false when
// the GPU could not be used (label is then unspecified); the outcome only steers the order of work.
bool cluster_rows(int32_t n, const int32_t* crow, const int32_t* col, const int32_t* parent, int device, int32_t* label);

}  // namespace cbm

#endif
