// batched_split.cu -- the fast-arithmetic instantiations of the batched step kernel
// (batched_kernel.cuh) that step one env with a cluster of thread blocks (CL = true).
// Compiled with the flags of batched.cu, whose kernels they match bit for bit.  The next tet
// record always rides in registers (PIPE): a part has few tets per thread and one block per
// SM, so nothing else hides its load.
#include "batched_kernel.cuh"

namespace ffsrl {

using namespace bk;

kern_f pick_fast_split(int block, unsigned flags) {
#define PK(B)                                                                                          \
    if (block == B)                                                                                    \
        return flags == kLiverFlags ? k_batched<AccFixed, B, 0, true, kLiverFlags, false, true>        \
                                    : k_batched<AccFixed, B, 0, true, 0, false, true>;
    PK(128) PK(256) PK(512)
#undef PK
    return nullptr;
}

}  // namespace ffsrl
