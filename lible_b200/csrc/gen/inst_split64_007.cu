// Generated by gen_instances.py: split forms of (3,0|1,1), (3,0|2,0), (3,0|2,1).
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_split64_06_02(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,0,1,1,double>())
            return launchSplit<3,0,1,1,double>(a, s, n);
        else
            return launchSplit<1,1,3,0,double>(a, s, n);
    }
    cudaError_t launch_split64_06_03(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,0,2,0,double>())
            return launchSplit<3,0,2,0,double>(a, s, n);
        else
            return launchSplit<2,0,3,0,double>(a, s, n);
    }
    cudaError_t launch_split64_06_04(const QuartetArgs &a, cudaStream_t s, int n)
    {
        if constexpr (hasSplitForm<3,0,2,1,double>())
            return launchSplit<3,0,2,1,double>(a, s, n);
        else
            return launchSplit<2,1,3,0,double>(a, s, n);
    }
}
