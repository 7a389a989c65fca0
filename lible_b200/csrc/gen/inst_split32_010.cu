// Generated by gen_instances.py: split forms of (3,2|1,0), (3,3|0,0).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split32_08_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,2,1,0,float>())
            return launchSplit<3,2,1,0,float>(a, s, n);
        else
            return launchSplit<1,0,3,2,float>(a, s, n);
    }
    cudaError_t launch_split32_09_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,3,0,0,float>())
            return launchSplit<3,3,0,0,float>(a, s, n);
        else
            return launchSplit<0,0,3,3,float>(a, s, n);
    }
}
