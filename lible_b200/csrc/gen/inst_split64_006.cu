// Generated by gen_instances.py: split forms of (2,2|2,0), (3,0|0,0), (3,0|1,0).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split64_05_03(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<2,2,2,0,double>())
            return launchSplit<2,2,2,0,double>(a, s, n);
        else
            return launchSplit<2,0,2,2,double>(a, s, n);
    }
    cudaError_t launch_split64_06_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,0,0,0,double>())
            return launchSplit<3,0,0,0,double>(a, s, n);
        else
            return launchSplit<0,0,3,0,double>(a, s, n);
    }
    cudaError_t launch_split64_06_01(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,0,1,0,double>())
            return launchSplit<3,0,1,0,double>(a, s, n);
        else
            return launchSplit<1,0,3,0,double>(a, s, n);
    }
}
