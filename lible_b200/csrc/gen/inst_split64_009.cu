// Generated by gen_instances.py: split forms of (3,1|1,1), (3,1|2,0), (3,2|0,0).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split64_07_02(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,1,1,1,double>())
            return launchSplit<3,1,1,1,double>(a, s, n);
        else
            return launchSplit<1,1,3,1,double>(a, s, n);
    }
    cudaError_t launch_split64_07_03(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,1,2,0,double>())
            return launchSplit<3,1,2,0,double>(a, s, n);
        else
            return launchSplit<2,0,3,1,double>(a, s, n);
    }
    cudaError_t launch_split64_08_00(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,2,0,0,double>())
            return launchSplit<3,2,0,0,double>(a, s, n);
        else
            return launchSplit<0,0,3,2,double>(a, s, n);
    }
}
