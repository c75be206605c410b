// One group of instances of the tensor-core kernel: compiled once per group with -DTSB_TC_PART=0..10.
#include "conv_tc_kernel.cuh"

namespace tsb {
namespace tc {

#define TSB_TC_INSTANCE(BN_, BK_, SWAP_, MODE_, EPI_, DUAL_)                                                                      \
    template int launch<BN_, BK_, SWAP_, MODE_, EPI_, DUAL_>(const Config &, const CUtensorMap &, const CUtensorMap &,            \
                                                       const CUtensorMap &, const CUtensorMap &, const CUtensorMap &,       \
                                                       const KernelParams &, const EpiParams &, cudaStream_t,               \
                                                       const std::conditional_t<DUAL_, DualParams, NoDual> &);
#define TSB_TC_CONCAT(A, B) A##B
#define TSB_TC_PART_OF(N) TSB_TC_CONCAT(TSB_TC_PART_, N)
TSB_TC_PART_OF(TSB_TC_PART)(TSB_TC_INSTANCE)

}  // namespace tc
}  // namespace tsb
