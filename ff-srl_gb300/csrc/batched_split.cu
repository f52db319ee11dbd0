// batched_split.cu -- the fast-arithmetic instantiations of the batched step kernel
// (batched_kernel.cuh) that step one env with a cluster of thread blocks (CL = true).
// Compiled with the flags of batched.cu, whose kernels they match bit for bit.  Up to 512
// threads the next tet record rides in registers (PIPE): a part has few tets per thread and
// one block per SM, so nothing else hides its load; 768 leave no registers for it.
#include "batched_kernel.cuh"

namespace ffsrl {

using namespace bk;

kern_f pick_fast_split(int block, unsigned flags) {
#define PK(B, PIPE)                                                                                    \
    if (block == B)                                                                                    \
        return flags == kLiverFlags ? k_batched<AccFixed, B, 0, PIPE, kLiverFlags, false, true>        \
                                    : k_batched<AccFixed, B, 0, PIPE, 0, false, true>;
    PK(128, true) PK(256, true) PK(512, true) PK(768, false)
#undef PK
    return nullptr;
}

}  // namespace ffsrl
