// Generated by gen_instances.py: split forms of (2,0|2,0), (2,1|0,0), (2,1|1,0).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split32_03_03(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,0,2,0,float>())
            return launchSplit<2,0,2,0,float>(a, s, n);
        else
            return launchSplit<2,0,2,0,float>(a, s, n);
    }
    cudaError_t launch_split32_04_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,1,0,0,float>())
            return launchSplit<2,1,0,0,float>(a, s, n);
        else
            return launchSplit<0,0,2,1,float>(a, s, n);
    }
    cudaError_t launch_split32_04_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,1,1,0,float>())
            return launchSplit<2,1,1,0,float>(a, s, n);
        else
            return launchSplit<1,0,2,1,float>(a, s, n);
    }
}
