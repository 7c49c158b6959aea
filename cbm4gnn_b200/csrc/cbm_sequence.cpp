// Several of the library's calls as one.  On graphs of a few thousand nodes the kernels of a layer are shorter than the
// time a caller's interpreter takes to allocate for, look up and issue each of them; a caller that knows all calls of a
// pass beforehand lists them once and hands over, each time, the list and where its arrays lie now.
#include <string>

#include "cbm_b200.h"
#include "cbm_common.h"

extern "C" int cbm_b200_sequence(const int64_t* calls, int32_t n_calls, const int64_t* bases, int32_t n_bases, void* stream) {
    if (n_calls < 0 || n_bases < 0 || n_bases > 256 || (n_calls && !calls) || (n_bases && !bases))
        return cbm::fail(CBM_B200_ERR_ARG, "sequence: bad arguments");
    bool known = true;
    const auto at = [&](int64_t place) -> float* {  // base number + 256 x offset in bytes; negative: NULL
        if (place < 0) return nullptr;
        if ((place & 255) >= n_bases) {
            known = false;
            return nullptr;
        }
        return reinterpret_cast<float*>(bases[place & 255] + (place >> 8));
    };
    for (int32_t i = 0; i < n_calls; ++i) {
        const int64_t* c = calls + (int64_t)CBM_B200_CALL_WORDS * i;
        const auto whole = [&](int k) { return (int32_t)c[k]; };
        int rc = CBM_B200_OK;
        if (c[0] == CBM_B200_CALL_PRODUCT) {
            auto* plan = reinterpret_cast<cbm_b200_plan*>(c[1]);
            const float* x = at(c[2]);
            float* y = at(c[4]);
            if (known) rc = (c[7] ? cbm_b200_fused_spmm_update : cbm_b200_spmm_update)(plan, x, c[3], y, c[5], whole(6), stream);
        } else if (c[0] == CBM_B200_CALL_MAP) {
            const float *x = at(c[1]), *w = at(c[3]);
            float* y = at(c[5]);
            if (!known) {
            } else if (c[10]) {
                rc = cbm_b200_dense_forward_of_relu(x, c[2], w, c[4], y, c[6], whole(7), whole(8), whole(9), whole(11), stream);
            } else {
                rc = (c[11] ? cbm_b200_dense_forward_relu : cbm_b200_dense_forward)(x, c[2], w, c[4], y, c[6], whole(7), whole(8),
                                                                                 whole(9), stream);
            }
        } else if (c[0] == CBM_B200_CALL_GRAD_INPUT) {
            const float *dy = at(c[1]), *w = at(c[3]), *h = at(c[5]);
            float* dx = at(c[7]);
            if (!known) {
            } else if (h) {
                rc = cbm_b200_dense_grad_input_relu(dy, c[2], w, c[4], h, c[6], dx, c[8], whole(9), whole(10), whole(11), stream);
            } else {
                rc = cbm_b200_dense_grad_input(dy, c[2], w, c[4], dx, c[8], whole(9), whole(10), whole(11), stream);
            }
        } else if (c[0] == CBM_B200_CALL_GRAD_WEIGHT) {
            const float *dy = at(c[1]), *x = at(c[3]);
            float *dw = at(c[5]), *workspace = at(c[11]);
            if (known)
                rc = (c[10] ? cbm_b200_dense_grad_weight_of_relu : cbm_b200_dense_grad_weight)(
                    dy, c[2], x, c[4], dw, c[6], whole(7), whole(8), whole(9), workspace, c[12], stream);
        } else {
            return cbm::fail(CBM_B200_ERR_ARG, "sequence: call " + std::to_string(i) + " is of no known kind");
        }
        if (!known) return cbm::fail(CBM_B200_ERR_ARG, "sequence: call " + std::to_string(i) + " names a base that was not given");
        if (rc) return rc;
    }
    return CBM_B200_OK;
}
