// Generated by gen_instances.py: split forms of (2,0|0,0), (2,0|1,0), (2,0|1,1).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split64_03_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,0,0,0,double>())
            return launchSplit<2,0,0,0,double>(a, s, n);
        else
            return launchSplit<0,0,2,0,double>(a, s, n);
    }
    cudaError_t launch_split64_03_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,0,1,0,double>())
            return launchSplit<2,0,1,0,double>(a, s, n);
        else
            return launchSplit<1,0,2,0,double>(a, s, n);
    }
    cudaError_t launch_split64_03_02(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,0,1,1,double>())
            return launchSplit<2,0,1,1,double>(a, s, n);
        else
            return launchSplit<1,1,2,0,double>(a, s, n);
    }
}
