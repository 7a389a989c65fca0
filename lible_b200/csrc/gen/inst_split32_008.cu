// Generated by gen_instances.py: split forms of (3,0|3,0), (3,1|0,0), (3,1|1,0).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split32_06_06(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,0,3,0,float>())
            return launchSplit<3,0,3,0,float>(a, s, n);
        else
            return launchSplit<3,0,3,0,float>(a, s, n);
    }
    cudaError_t launch_split32_07_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,1,0,0,float>())
            return launchSplit<3,1,0,0,float>(a, s, n);
        else
            return launchSplit<0,0,3,1,float>(a, s, n);
    }
    cudaError_t launch_split32_07_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,1,1,0,float>())
            return launchSplit<3,1,1,0,float>(a, s, n);
        else
            return launchSplit<1,0,3,1,float>(a, s, n);
    }
}
