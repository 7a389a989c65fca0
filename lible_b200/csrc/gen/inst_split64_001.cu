// Generated by gen_instances.py: split forms of (1,1|0,0), (1,1|1,0), (1,1|1,1).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split64_02_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<1,1,0,0,double>())
            return launchSplit<1,1,0,0,double>(a, s, n);
        else
            return launchSplit<0,0,1,1,double>(a, s, n);
    }
    cudaError_t launch_split64_02_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<1,1,1,0,double>())
            return launchSplit<1,1,1,0,double>(a, s, n);
        else
            return launchSplit<1,0,1,1,double>(a, s, n);
    }
    cudaError_t launch_split64_02_02(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<1,1,1,1,double>())
            return launchSplit<1,1,1,1,double>(a, s, n);
        else
            return launchSplit<1,1,1,1,double>(a, s, n);
    }
}
