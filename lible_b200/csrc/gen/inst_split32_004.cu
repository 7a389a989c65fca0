// Generated by gen_instances.py: split forms of (2,1|1,1), (2,1|2,0), (2,1|2,1).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split32_04_02(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,1,1,1,float>())
            return launchSplit<2,1,1,1,float>(a, s, n);
        else
            return launchSplit<1,1,2,1,float>(a, s, n);
    }
    cudaError_t launch_split32_04_03(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,1,2,0,float>())
            return launchSplit<2,1,2,0,float>(a, s, n);
        else
            return launchSplit<2,0,2,1,float>(a, s, n);
    }
    cudaError_t launch_split32_04_04(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,1,2,1,float>())
            return launchSplit<2,1,2,1,float>(a, s, n);
        else
            return launchSplit<2,1,2,1,float>(a, s, n);
    }
}
