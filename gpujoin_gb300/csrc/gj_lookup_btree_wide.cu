// gj_lookup_btree_wide.cu -- B+tree probe kernels for plain nodes of 16, 32 and 64 separators.
#include "gj_lookup_kernels.cuh"

namespace gj {

template <>
int lookup_call_btree<16>(const gj_index* idx, const lookup_call& c) {
    return plain_nodes_call<16>(idx, c);
}

template <>
int lookup_call_btree<32>(const gj_index* idx, const lookup_call& c) {
    return plain_nodes_call<32>(idx, c);
}

template <>
int lookup_call_btree<64>(const gj_index* idx, const lookup_call& c) {
    return plain_nodes_call<64>(idx, c);
}

}  // namespace gj
