// gj_lookup_btree.cu -- B+tree probe kernels for plain nodes of 4 and 8 separators.
#include "gj_lookup_kernels.cuh"

namespace gj {

template <>
int lookup_call_btree<4>(const gj_index* idx, const lookup_call& c) {
    return plain_nodes_call<4>(idx, c);
}

template <>
int lookup_call_btree<8>(const gj_index* idx, const lookup_call& c) {
    return plain_nodes_call<8>(idx, c);
}

}  // namespace gj
