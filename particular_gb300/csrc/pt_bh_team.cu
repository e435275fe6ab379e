// The group walk's kernels for several warps per group, a unit of their own so that they
// compile beside the others.
#include "pt_bh_group.cuh"

namespace pt {
namespace bh {

GroupKernel group_kernel_team(bool quad, bool guard, bool local, bool rel, int team) {
    return team == 8 ? group_kernel_w<8>(quad, guard, local, rel) : group_kernel_w<4>(quad, guard, local, rel);
}

}  // namespace bh
}  // namespace pt
