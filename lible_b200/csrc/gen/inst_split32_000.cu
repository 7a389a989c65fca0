// Generated by gen_instances.py: split forms of (0,0|0,0), (1,0|0,0), (1,0|1,0).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split32_00_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<0,0,0,0,float>())
            return launchSplit<0,0,0,0,float>(a, s, n);
        else
            return launchSplit<0,0,0,0,float>(a, s, n);
    }
    cudaError_t launch_split32_01_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<1,0,0,0,float>())
            return launchSplit<1,0,0,0,float>(a, s, n);
        else
            return launchSplit<0,0,1,0,float>(a, s, n);
    }
    cudaError_t launch_split32_01_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<1,0,1,0,float>())
            return launchSplit<1,0,1,0,float>(a, s, n);
        else
            return launchSplit<1,0,1,0,float>(a, s, n);
    }
}
