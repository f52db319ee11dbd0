// batched_split_ref.cu -- the reference-arithmetic instantiations of the batched step kernel
// (batched_kernel.cuh) that step one env with a cluster of thread blocks (CL = true).
// Compiled with the flags of batched_ref.cu, whose kernels they match bit for bit.  The next tet
// record always rides in registers (PIPE): a part has few tets per thread and one block per
// SM, so nothing else hides its load.
#include "batched_kernel.cuh"

namespace ffsrl {

using namespace bk;

kern_f pick_ref_split(int block, unsigned flags) {
#define PK(B)                                                                                          \
    if (block == B)                                                                                    \
        return flags == kLiverFlags ? k_batched<AccFixed, B, 0, true, kLiverFlags, true, true>        \
                                    : k_batched<AccFixed, B, 0, true, 0, true, true>;
    PK(128) PK(256) PK(512)
#undef PK
    return nullptr;
}

}  // namespace ffsrl
