// Generated by gen_instances.py: lookup of class kernels.
#include "../eri_launch_fwd.cuh"
#include "../eri_split_kernel.cuh"

namespace lible_b200
{
    cudaError_t launch_fwd64_00_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_01_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_01_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_10(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_10(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_11(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_00_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_01_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_01_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_08_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_08_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_09_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_08_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_09_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_10_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_08_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_09_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_10_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_11_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_00_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_01_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_01_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_02_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_03_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_04_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_05_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_06_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_07_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_08_08_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_08_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_09_09_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_08_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_09_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_10_10_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_08_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_09_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_10_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd64_11_11_f(const QuartetArgs &, cudaStream_t, int);
    static const LaunchFn k_fwd64_00[1] = {&launch_fwd64_00_00};
    static const LaunchFn k_fwd64v_00[1] = {hasShapeVariant<0,0,0,0,double>() ? &launch_fwd64_00_00_v1 : nullptr};
    static const LaunchFn k_fwd64f_00[1] = {hasFlippedShape<0,0,0,0,double>() ? &launch_fwd64_00_00_f : nullptr};
    static const int u_fwd64_0_00[1] = {workUnit<0,0,0,0,double,0>()};
    static const int u_fwd64_1_00[1] = {workUnit<0,0,0,0,double,1>()};
    static const int u_fwd64_2_00[1] = {hasFlippedShape<0,0,0,0,double>() ? workUnit<0,0,0,0,double,0>() : 0};
    static const LaunchFn k_fwd64_01[2] = {&launch_fwd64_01_00, &launch_fwd64_01_01};
    static const LaunchFn k_fwd64v_01[2] = {hasShapeVariant<1,0,0,0,double>() ? &launch_fwd64_01_00_v1 : nullptr, hasShapeVariant<1,0,1,0,double>() ? &launch_fwd64_01_01_v1 : nullptr};
    static const LaunchFn k_fwd64f_01[2] = {hasFlippedShape<1,0,0,0,double>() ? &launch_fwd64_01_00_f : nullptr, hasFlippedShape<1,0,1,0,double>() ? &launch_fwd64_01_01_f : nullptr};
    static const int u_fwd64_0_01[2] = {workUnit<1,0,0,0,double,0>(), workUnit<1,0,1,0,double,0>()};
    static const int u_fwd64_1_01[2] = {workUnit<1,0,0,0,double,1>(), workUnit<1,0,1,0,double,1>()};
    static const int u_fwd64_2_01[2] = {hasFlippedShape<1,0,0,0,double>() ? workUnit<0,0,1,0,double,0>() : 0, hasFlippedShape<1,0,1,0,double>() ? workUnit<1,0,1,0,double,0>() : 0};
    static const LaunchFn k_fwd64_02[3] = {&launch_fwd64_02_00, &launch_fwd64_02_01, &launch_fwd64_02_02};
    static const LaunchFn k_fwd64v_02[3] = {hasShapeVariant<1,1,0,0,double>() ? &launch_fwd64_02_00_v1 : nullptr, hasShapeVariant<1,1,1,0,double>() ? &launch_fwd64_02_01_v1 : nullptr, hasShapeVariant<1,1,1,1,double>() ? &launch_fwd64_02_02_v1 : nullptr};
    static const LaunchFn k_fwd64f_02[3] = {hasFlippedShape<1,1,0,0,double>() ? &launch_fwd64_02_00_f : nullptr, hasFlippedShape<1,1,1,0,double>() ? &launch_fwd64_02_01_f : nullptr, hasFlippedShape<1,1,1,1,double>() ? &launch_fwd64_02_02_f : nullptr};
    static const int u_fwd64_0_02[3] = {workUnit<1,1,0,0,double,0>(), workUnit<1,1,1,0,double,0>(), workUnit<1,1,1,1,double,0>()};
    static const int u_fwd64_1_02[3] = {workUnit<1,1,0,0,double,1>(), workUnit<1,1,1,0,double,1>(), workUnit<1,1,1,1,double,1>()};
    static const int u_fwd64_2_02[3] = {hasFlippedShape<1,1,0,0,double>() ? workUnit<0,0,1,1,double,0>() : 0, hasFlippedShape<1,1,1,0,double>() ? workUnit<1,0,1,1,double,0>() : 0, hasFlippedShape<1,1,1,1,double>() ? workUnit<1,1,1,1,double,0>() : 0};
    static const LaunchFn k_fwd64_03[4] = {&launch_fwd64_03_00, &launch_fwd64_03_01, &launch_fwd64_03_02, &launch_fwd64_03_03};
    static const LaunchFn k_fwd64v_03[4] = {hasShapeVariant<2,0,0,0,double>() ? &launch_fwd64_03_00_v1 : nullptr, hasShapeVariant<2,0,1,0,double>() ? &launch_fwd64_03_01_v1 : nullptr, hasShapeVariant<2,0,1,1,double>() ? &launch_fwd64_03_02_v1 : nullptr, hasShapeVariant<2,0,2,0,double>() ? &launch_fwd64_03_03_v1 : nullptr};
    static const LaunchFn k_fwd64f_03[4] = {hasFlippedShape<2,0,0,0,double>() ? &launch_fwd64_03_00_f : nullptr, hasFlippedShape<2,0,1,0,double>() ? &launch_fwd64_03_01_f : nullptr, hasFlippedShape<2,0,1,1,double>() ? &launch_fwd64_03_02_f : nullptr, hasFlippedShape<2,0,2,0,double>() ? &launch_fwd64_03_03_f : nullptr};
    static const int u_fwd64_0_03[4] = {workUnit<2,0,0,0,double,0>(), workUnit<2,0,1,0,double,0>(), workUnit<2,0,1,1,double,0>(), workUnit<2,0,2,0,double,0>()};
    static const int u_fwd64_1_03[4] = {workUnit<2,0,0,0,double,1>(), workUnit<2,0,1,0,double,1>(), workUnit<2,0,1,1,double,1>(), workUnit<2,0,2,0,double,1>()};
    static const int u_fwd64_2_03[4] = {hasFlippedShape<2,0,0,0,double>() ? workUnit<0,0,2,0,double,0>() : 0, hasFlippedShape<2,0,1,0,double>() ? workUnit<1,0,2,0,double,0>() : 0, hasFlippedShape<2,0,1,1,double>() ? workUnit<1,1,2,0,double,0>() : 0, hasFlippedShape<2,0,2,0,double>() ? workUnit<2,0,2,0,double,0>() : 0};
    static const LaunchFn k_fwd64_04[5] = {&launch_fwd64_04_00, &launch_fwd64_04_01, &launch_fwd64_04_02, &launch_fwd64_04_03, &launch_fwd64_04_04};
    static const LaunchFn k_fwd64v_04[5] = {hasShapeVariant<2,1,0,0,double>() ? &launch_fwd64_04_00_v1 : nullptr, hasShapeVariant<2,1,1,0,double>() ? &launch_fwd64_04_01_v1 : nullptr, hasShapeVariant<2,1,1,1,double>() ? &launch_fwd64_04_02_v1 : nullptr, hasShapeVariant<2,1,2,0,double>() ? &launch_fwd64_04_03_v1 : nullptr, hasShapeVariant<2,1,2,1,double>() ? &launch_fwd64_04_04_v1 : nullptr};
    static const LaunchFn k_fwd64f_04[5] = {hasFlippedShape<2,1,0,0,double>() ? &launch_fwd64_04_00_f : nullptr, hasFlippedShape<2,1,1,0,double>() ? &launch_fwd64_04_01_f : nullptr, hasFlippedShape<2,1,1,1,double>() ? &launch_fwd64_04_02_f : nullptr, hasFlippedShape<2,1,2,0,double>() ? &launch_fwd64_04_03_f : nullptr, hasFlippedShape<2,1,2,1,double>() ? &launch_fwd64_04_04_f : nullptr};
    static const int u_fwd64_0_04[5] = {workUnit<2,1,0,0,double,0>(), workUnit<2,1,1,0,double,0>(), workUnit<2,1,1,1,double,0>(), workUnit<2,1,2,0,double,0>(), workUnit<2,1,2,1,double,0>()};
    static const int u_fwd64_1_04[5] = {workUnit<2,1,0,0,double,1>(), workUnit<2,1,1,0,double,1>(), workUnit<2,1,1,1,double,1>(), workUnit<2,1,2,0,double,1>(), workUnit<2,1,2,1,double,1>()};
    static const int u_fwd64_2_04[5] = {hasFlippedShape<2,1,0,0,double>() ? workUnit<0,0,2,1,double,0>() : 0, hasFlippedShape<2,1,1,0,double>() ? workUnit<1,0,2,1,double,0>() : 0, hasFlippedShape<2,1,1,1,double>() ? workUnit<1,1,2,1,double,0>() : 0, hasFlippedShape<2,1,2,0,double>() ? workUnit<2,0,2,1,double,0>() : 0, hasFlippedShape<2,1,2,1,double>() ? workUnit<2,1,2,1,double,0>() : 0};
    static const LaunchFn k_fwd64_05[6] = {&launch_fwd64_05_00, &launch_fwd64_05_01, &launch_fwd64_05_02, &launch_fwd64_05_03, &launch_fwd64_05_04, &launch_fwd64_05_05};
    static const LaunchFn k_fwd64v_05[6] = {hasShapeVariant<2,2,0,0,double>() ? &launch_fwd64_05_00_v1 : nullptr, hasShapeVariant<2,2,1,0,double>() ? &launch_fwd64_05_01_v1 : nullptr, hasShapeVariant<2,2,1,1,double>() ? &launch_fwd64_05_02_v1 : nullptr, hasShapeVariant<2,2,2,0,double>() ? &launch_fwd64_05_03_v1 : nullptr, hasShapeVariant<2,2,2,1,double>() ? &launch_fwd64_05_04_v1 : nullptr, hasShapeVariant<2,2,2,2,double>() ? &launch_fwd64_05_05_v1 : nullptr};
    static const LaunchFn k_fwd64f_05[6] = {hasFlippedShape<2,2,0,0,double>() ? &launch_fwd64_05_00_f : nullptr, hasFlippedShape<2,2,1,0,double>() ? &launch_fwd64_05_01_f : nullptr, hasFlippedShape<2,2,1,1,double>() ? &launch_fwd64_05_02_f : nullptr, hasFlippedShape<2,2,2,0,double>() ? &launch_fwd64_05_03_f : nullptr, hasFlippedShape<2,2,2,1,double>() ? &launch_fwd64_05_04_f : nullptr, hasFlippedShape<2,2,2,2,double>() ? &launch_fwd64_05_05_f : nullptr};
    static const int u_fwd64_0_05[6] = {workUnit<2,2,0,0,double,0>(), workUnit<2,2,1,0,double,0>(), workUnit<2,2,1,1,double,0>(), workUnit<2,2,2,0,double,0>(), workUnit<2,2,2,1,double,0>(), workUnit<2,2,2,2,double,0>()};
    static const int u_fwd64_1_05[6] = {workUnit<2,2,0,0,double,1>(), workUnit<2,2,1,0,double,1>(), workUnit<2,2,1,1,double,1>(), workUnit<2,2,2,0,double,1>(), workUnit<2,2,2,1,double,1>(), workUnit<2,2,2,2,double,1>()};
    static const int u_fwd64_2_05[6] = {hasFlippedShape<2,2,0,0,double>() ? workUnit<0,0,2,2,double,0>() : 0, hasFlippedShape<2,2,1,0,double>() ? workUnit<1,0,2,2,double,0>() : 0, hasFlippedShape<2,2,1,1,double>() ? workUnit<1,1,2,2,double,0>() : 0, hasFlippedShape<2,2,2,0,double>() ? workUnit<2,0,2,2,double,0>() : 0, hasFlippedShape<2,2,2,1,double>() ? workUnit<2,1,2,2,double,0>() : 0, hasFlippedShape<2,2,2,2,double>() ? workUnit<2,2,2,2,double,0>() : 0};
    static const LaunchFn k_fwd64_06[7] = {&launch_fwd64_06_00, &launch_fwd64_06_01, &launch_fwd64_06_02, &launch_fwd64_06_03, &launch_fwd64_06_04, &launch_fwd64_06_05, &launch_fwd64_06_06};
    static const LaunchFn k_fwd64v_06[7] = {hasShapeVariant<3,0,0,0,double>() ? &launch_fwd64_06_00_v1 : nullptr, hasShapeVariant<3,0,1,0,double>() ? &launch_fwd64_06_01_v1 : nullptr, hasShapeVariant<3,0,1,1,double>() ? &launch_fwd64_06_02_v1 : nullptr, hasShapeVariant<3,0,2,0,double>() ? &launch_fwd64_06_03_v1 : nullptr, hasShapeVariant<3,0,2,1,double>() ? &launch_fwd64_06_04_v1 : nullptr, hasShapeVariant<3,0,2,2,double>() ? &launch_fwd64_06_05_v1 : nullptr, hasShapeVariant<3,0,3,0,double>() ? &launch_fwd64_06_06_v1 : nullptr};
    static const LaunchFn k_fwd64f_06[7] = {hasFlippedShape<3,0,0,0,double>() ? &launch_fwd64_06_00_f : nullptr, hasFlippedShape<3,0,1,0,double>() ? &launch_fwd64_06_01_f : nullptr, hasFlippedShape<3,0,1,1,double>() ? &launch_fwd64_06_02_f : nullptr, hasFlippedShape<3,0,2,0,double>() ? &launch_fwd64_06_03_f : nullptr, hasFlippedShape<3,0,2,1,double>() ? &launch_fwd64_06_04_f : nullptr, hasFlippedShape<3,0,2,2,double>() ? &launch_fwd64_06_05_f : nullptr, hasFlippedShape<3,0,3,0,double>() ? &launch_fwd64_06_06_f : nullptr};
    static const int u_fwd64_0_06[7] = {workUnit<3,0,0,0,double,0>(), workUnit<3,0,1,0,double,0>(), workUnit<3,0,1,1,double,0>(), workUnit<3,0,2,0,double,0>(), workUnit<3,0,2,1,double,0>(), workUnit<3,0,2,2,double,0>(), workUnit<3,0,3,0,double,0>()};
    static const int u_fwd64_1_06[7] = {workUnit<3,0,0,0,double,1>(), workUnit<3,0,1,0,double,1>(), workUnit<3,0,1,1,double,1>(), workUnit<3,0,2,0,double,1>(), workUnit<3,0,2,1,double,1>(), workUnit<3,0,2,2,double,1>(), workUnit<3,0,3,0,double,1>()};
    static const int u_fwd64_2_06[7] = {hasFlippedShape<3,0,0,0,double>() ? workUnit<0,0,3,0,double,0>() : 0, hasFlippedShape<3,0,1,0,double>() ? workUnit<1,0,3,0,double,0>() : 0, hasFlippedShape<3,0,1,1,double>() ? workUnit<1,1,3,0,double,0>() : 0, hasFlippedShape<3,0,2,0,double>() ? workUnit<2,0,3,0,double,0>() : 0, hasFlippedShape<3,0,2,1,double>() ? workUnit<2,1,3,0,double,0>() : 0, hasFlippedShape<3,0,2,2,double>() ? workUnit<2,2,3,0,double,0>() : 0, hasFlippedShape<3,0,3,0,double>() ? workUnit<3,0,3,0,double,0>() : 0};
    static const LaunchFn k_fwd64_07[8] = {&launch_fwd64_07_00, &launch_fwd64_07_01, &launch_fwd64_07_02, &launch_fwd64_07_03, &launch_fwd64_07_04, &launch_fwd64_07_05, &launch_fwd64_07_06, &launch_fwd64_07_07};
    static const LaunchFn k_fwd64v_07[8] = {hasShapeVariant<3,1,0,0,double>() ? &launch_fwd64_07_00_v1 : nullptr, hasShapeVariant<3,1,1,0,double>() ? &launch_fwd64_07_01_v1 : nullptr, hasShapeVariant<3,1,1,1,double>() ? &launch_fwd64_07_02_v1 : nullptr, hasShapeVariant<3,1,2,0,double>() ? &launch_fwd64_07_03_v1 : nullptr, hasShapeVariant<3,1,2,1,double>() ? &launch_fwd64_07_04_v1 : nullptr, hasShapeVariant<3,1,2,2,double>() ? &launch_fwd64_07_05_v1 : nullptr, hasShapeVariant<3,1,3,0,double>() ? &launch_fwd64_07_06_v1 : nullptr, hasShapeVariant<3,1,3,1,double>() ? &launch_fwd64_07_07_v1 : nullptr};
    static const LaunchFn k_fwd64f_07[8] = {hasFlippedShape<3,1,0,0,double>() ? &launch_fwd64_07_00_f : nullptr, hasFlippedShape<3,1,1,0,double>() ? &launch_fwd64_07_01_f : nullptr, hasFlippedShape<3,1,1,1,double>() ? &launch_fwd64_07_02_f : nullptr, hasFlippedShape<3,1,2,0,double>() ? &launch_fwd64_07_03_f : nullptr, hasFlippedShape<3,1,2,1,double>() ? &launch_fwd64_07_04_f : nullptr, hasFlippedShape<3,1,2,2,double>() ? &launch_fwd64_07_05_f : nullptr, hasFlippedShape<3,1,3,0,double>() ? &launch_fwd64_07_06_f : nullptr, hasFlippedShape<3,1,3,1,double>() ? &launch_fwd64_07_07_f : nullptr};
    static const int u_fwd64_0_07[8] = {workUnit<3,1,0,0,double,0>(), workUnit<3,1,1,0,double,0>(), workUnit<3,1,1,1,double,0>(), workUnit<3,1,2,0,double,0>(), workUnit<3,1,2,1,double,0>(), workUnit<3,1,2,2,double,0>(), workUnit<3,1,3,0,double,0>(), workUnit<3,1,3,1,double,0>()};
    static const int u_fwd64_1_07[8] = {workUnit<3,1,0,0,double,1>(), workUnit<3,1,1,0,double,1>(), workUnit<3,1,1,1,double,1>(), workUnit<3,1,2,0,double,1>(), workUnit<3,1,2,1,double,1>(), workUnit<3,1,2,2,double,1>(), workUnit<3,1,3,0,double,1>(), workUnit<3,1,3,1,double,1>()};
    static const int u_fwd64_2_07[8] = {hasFlippedShape<3,1,0,0,double>() ? workUnit<0,0,3,1,double,0>() : 0, hasFlippedShape<3,1,1,0,double>() ? workUnit<1,0,3,1,double,0>() : 0, hasFlippedShape<3,1,1,1,double>() ? workUnit<1,1,3,1,double,0>() : 0, hasFlippedShape<3,1,2,0,double>() ? workUnit<2,0,3,1,double,0>() : 0, hasFlippedShape<3,1,2,1,double>() ? workUnit<2,1,3,1,double,0>() : 0, hasFlippedShape<3,1,2,2,double>() ? workUnit<2,2,3,1,double,0>() : 0, hasFlippedShape<3,1,3,0,double>() ? workUnit<3,0,3,1,double,0>() : 0, hasFlippedShape<3,1,3,1,double>() ? workUnit<3,1,3,1,double,0>() : 0};
    static const LaunchFn k_fwd64_08[9] = {&launch_fwd64_08_00, &launch_fwd64_08_01, &launch_fwd64_08_02, &launch_fwd64_08_03, &launch_fwd64_08_04, &launch_fwd64_08_05, &launch_fwd64_08_06, &launch_fwd64_08_07, &launch_fwd64_08_08};
    static const LaunchFn k_fwd64v_08[9] = {hasShapeVariant<3,2,0,0,double>() ? &launch_fwd64_08_00_v1 : nullptr, hasShapeVariant<3,2,1,0,double>() ? &launch_fwd64_08_01_v1 : nullptr, hasShapeVariant<3,2,1,1,double>() ? &launch_fwd64_08_02_v1 : nullptr, hasShapeVariant<3,2,2,0,double>() ? &launch_fwd64_08_03_v1 : nullptr, hasShapeVariant<3,2,2,1,double>() ? &launch_fwd64_08_04_v1 : nullptr, hasShapeVariant<3,2,2,2,double>() ? &launch_fwd64_08_05_v1 : nullptr, hasShapeVariant<3,2,3,0,double>() ? &launch_fwd64_08_06_v1 : nullptr, hasShapeVariant<3,2,3,1,double>() ? &launch_fwd64_08_07_v1 : nullptr, hasShapeVariant<3,2,3,2,double>() ? &launch_fwd64_08_08_v1 : nullptr};
    static const LaunchFn k_fwd64f_08[9] = {hasFlippedShape<3,2,0,0,double>() ? &launch_fwd64_08_00_f : nullptr, hasFlippedShape<3,2,1,0,double>() ? &launch_fwd64_08_01_f : nullptr, hasFlippedShape<3,2,1,1,double>() ? &launch_fwd64_08_02_f : nullptr, hasFlippedShape<3,2,2,0,double>() ? &launch_fwd64_08_03_f : nullptr, hasFlippedShape<3,2,2,1,double>() ? &launch_fwd64_08_04_f : nullptr, hasFlippedShape<3,2,2,2,double>() ? &launch_fwd64_08_05_f : nullptr, hasFlippedShape<3,2,3,0,double>() ? &launch_fwd64_08_06_f : nullptr, hasFlippedShape<3,2,3,1,double>() ? &launch_fwd64_08_07_f : nullptr, hasFlippedShape<3,2,3,2,double>() ? &launch_fwd64_08_08_f : nullptr};
    static const int u_fwd64_0_08[9] = {workUnit<3,2,0,0,double,0>(), workUnit<3,2,1,0,double,0>(), workUnit<3,2,1,1,double,0>(), workUnit<3,2,2,0,double,0>(), workUnit<3,2,2,1,double,0>(), workUnit<3,2,2,2,double,0>(), workUnit<3,2,3,0,double,0>(), workUnit<3,2,3,1,double,0>(), workUnit<3,2,3,2,double,0>()};
    static const int u_fwd64_1_08[9] = {workUnit<3,2,0,0,double,1>(), workUnit<3,2,1,0,double,1>(), workUnit<3,2,1,1,double,1>(), workUnit<3,2,2,0,double,1>(), workUnit<3,2,2,1,double,1>(), workUnit<3,2,2,2,double,1>(), workUnit<3,2,3,0,double,1>(), workUnit<3,2,3,1,double,1>(), workUnit<3,2,3,2,double,1>()};
    static const int u_fwd64_2_08[9] = {hasFlippedShape<3,2,0,0,double>() ? workUnit<0,0,3,2,double,0>() : 0, hasFlippedShape<3,2,1,0,double>() ? workUnit<1,0,3,2,double,0>() : 0, hasFlippedShape<3,2,1,1,double>() ? workUnit<1,1,3,2,double,0>() : 0, hasFlippedShape<3,2,2,0,double>() ? workUnit<2,0,3,2,double,0>() : 0, hasFlippedShape<3,2,2,1,double>() ? workUnit<2,1,3,2,double,0>() : 0, hasFlippedShape<3,2,2,2,double>() ? workUnit<2,2,3,2,double,0>() : 0, hasFlippedShape<3,2,3,0,double>() ? workUnit<3,0,3,2,double,0>() : 0, hasFlippedShape<3,2,3,1,double>() ? workUnit<3,1,3,2,double,0>() : 0, hasFlippedShape<3,2,3,2,double>() ? workUnit<3,2,3,2,double,0>() : 0};
    static const LaunchFn k_fwd64_09[10] = {&launch_fwd64_09_00, &launch_fwd64_09_01, &launch_fwd64_09_02, &launch_fwd64_09_03, &launch_fwd64_09_04, &launch_fwd64_09_05, &launch_fwd64_09_06, &launch_fwd64_09_07, &launch_fwd64_09_08, &launch_fwd64_09_09};
    static const LaunchFn k_fwd64v_09[10] = {hasShapeVariant<3,3,0,0,double>() ? &launch_fwd64_09_00_v1 : nullptr, hasShapeVariant<3,3,1,0,double>() ? &launch_fwd64_09_01_v1 : nullptr, hasShapeVariant<3,3,1,1,double>() ? &launch_fwd64_09_02_v1 : nullptr, hasShapeVariant<3,3,2,0,double>() ? &launch_fwd64_09_03_v1 : nullptr, hasShapeVariant<3,3,2,1,double>() ? &launch_fwd64_09_04_v1 : nullptr, hasShapeVariant<3,3,2,2,double>() ? &launch_fwd64_09_05_v1 : nullptr, hasShapeVariant<3,3,3,0,double>() ? &launch_fwd64_09_06_v1 : nullptr, hasShapeVariant<3,3,3,1,double>() ? &launch_fwd64_09_07_v1 : nullptr, hasShapeVariant<3,3,3,2,double>() ? &launch_fwd64_09_08_v1 : nullptr, hasShapeVariant<3,3,3,3,double>() ? &launch_fwd64_09_09_v1 : nullptr};
    static const LaunchFn k_fwd64f_09[10] = {hasFlippedShape<3,3,0,0,double>() ? &launch_fwd64_09_00_f : nullptr, hasFlippedShape<3,3,1,0,double>() ? &launch_fwd64_09_01_f : nullptr, hasFlippedShape<3,3,1,1,double>() ? &launch_fwd64_09_02_f : nullptr, hasFlippedShape<3,3,2,0,double>() ? &launch_fwd64_09_03_f : nullptr, hasFlippedShape<3,3,2,1,double>() ? &launch_fwd64_09_04_f : nullptr, hasFlippedShape<3,3,2,2,double>() ? &launch_fwd64_09_05_f : nullptr, hasFlippedShape<3,3,3,0,double>() ? &launch_fwd64_09_06_f : nullptr, hasFlippedShape<3,3,3,1,double>() ? &launch_fwd64_09_07_f : nullptr, hasFlippedShape<3,3,3,2,double>() ? &launch_fwd64_09_08_f : nullptr, hasFlippedShape<3,3,3,3,double>() ? &launch_fwd64_09_09_f : nullptr};
    static const int u_fwd64_0_09[10] = {workUnit<3,3,0,0,double,0>(), workUnit<3,3,1,0,double,0>(), workUnit<3,3,1,1,double,0>(), workUnit<3,3,2,0,double,0>(), workUnit<3,3,2,1,double,0>(), workUnit<3,3,2,2,double,0>(), workUnit<3,3,3,0,double,0>(), workUnit<3,3,3,1,double,0>(), workUnit<3,3,3,2,double,0>(), workUnit<3,3,3,3,double,0>()};
    static const int u_fwd64_1_09[10] = {workUnit<3,3,0,0,double,1>(), workUnit<3,3,1,0,double,1>(), workUnit<3,3,1,1,double,1>(), workUnit<3,3,2,0,double,1>(), workUnit<3,3,2,1,double,1>(), workUnit<3,3,2,2,double,1>(), workUnit<3,3,3,0,double,1>(), workUnit<3,3,3,1,double,1>(), workUnit<3,3,3,2,double,1>(), workUnit<3,3,3,3,double,1>()};
    static const int u_fwd64_2_09[10] = {hasFlippedShape<3,3,0,0,double>() ? workUnit<0,0,3,3,double,0>() : 0, hasFlippedShape<3,3,1,0,double>() ? workUnit<1,0,3,3,double,0>() : 0, hasFlippedShape<3,3,1,1,double>() ? workUnit<1,1,3,3,double,0>() : 0, hasFlippedShape<3,3,2,0,double>() ? workUnit<2,0,3,3,double,0>() : 0, hasFlippedShape<3,3,2,1,double>() ? workUnit<2,1,3,3,double,0>() : 0, hasFlippedShape<3,3,2,2,double>() ? workUnit<2,2,3,3,double,0>() : 0, hasFlippedShape<3,3,3,0,double>() ? workUnit<3,0,3,3,double,0>() : 0, hasFlippedShape<3,3,3,1,double>() ? workUnit<3,1,3,3,double,0>() : 0, hasFlippedShape<3,3,3,2,double>() ? workUnit<3,2,3,3,double,0>() : 0, hasFlippedShape<3,3,3,3,double>() ? workUnit<3,3,3,3,double,0>() : 0};
    static const LaunchFn k_fwd64_10[11] = {&launch_fwd64_10_00, &launch_fwd64_10_01, &launch_fwd64_10_02, &launch_fwd64_10_03, &launch_fwd64_10_04, &launch_fwd64_10_05, &launch_fwd64_10_06, &launch_fwd64_10_07, &launch_fwd64_10_08, &launch_fwd64_10_09, &launch_fwd64_10_10};
    static const LaunchFn k_fwd64v_10[11] = {hasShapeVariant<4,0,0,0,double>() ? &launch_fwd64_10_00_v1 : nullptr, hasShapeVariant<4,0,1,0,double>() ? &launch_fwd64_10_01_v1 : nullptr, hasShapeVariant<4,0,1,1,double>() ? &launch_fwd64_10_02_v1 : nullptr, hasShapeVariant<4,0,2,0,double>() ? &launch_fwd64_10_03_v1 : nullptr, hasShapeVariant<4,0,2,1,double>() ? &launch_fwd64_10_04_v1 : nullptr, hasShapeVariant<4,0,2,2,double>() ? &launch_fwd64_10_05_v1 : nullptr, hasShapeVariant<4,0,3,0,double>() ? &launch_fwd64_10_06_v1 : nullptr, hasShapeVariant<4,0,3,1,double>() ? &launch_fwd64_10_07_v1 : nullptr, hasShapeVariant<4,0,3,2,double>() ? &launch_fwd64_10_08_v1 : nullptr, hasShapeVariant<4,0,3,3,double>() ? &launch_fwd64_10_09_v1 : nullptr, hasShapeVariant<4,0,4,0,double>() ? &launch_fwd64_10_10_v1 : nullptr};
    static const LaunchFn k_fwd64f_10[11] = {hasFlippedShape<4,0,0,0,double>() ? &launch_fwd64_10_00_f : nullptr, hasFlippedShape<4,0,1,0,double>() ? &launch_fwd64_10_01_f : nullptr, hasFlippedShape<4,0,1,1,double>() ? &launch_fwd64_10_02_f : nullptr, hasFlippedShape<4,0,2,0,double>() ? &launch_fwd64_10_03_f : nullptr, hasFlippedShape<4,0,2,1,double>() ? &launch_fwd64_10_04_f : nullptr, hasFlippedShape<4,0,2,2,double>() ? &launch_fwd64_10_05_f : nullptr, hasFlippedShape<4,0,3,0,double>() ? &launch_fwd64_10_06_f : nullptr, hasFlippedShape<4,0,3,1,double>() ? &launch_fwd64_10_07_f : nullptr, hasFlippedShape<4,0,3,2,double>() ? &launch_fwd64_10_08_f : nullptr, hasFlippedShape<4,0,3,3,double>() ? &launch_fwd64_10_09_f : nullptr, hasFlippedShape<4,0,4,0,double>() ? &launch_fwd64_10_10_f : nullptr};
    static const int u_fwd64_0_10[11] = {workUnit<4,0,0,0,double,0>(), workUnit<4,0,1,0,double,0>(), workUnit<4,0,1,1,double,0>(), workUnit<4,0,2,0,double,0>(), workUnit<4,0,2,1,double,0>(), workUnit<4,0,2,2,double,0>(), workUnit<4,0,3,0,double,0>(), workUnit<4,0,3,1,double,0>(), workUnit<4,0,3,2,double,0>(), workUnit<4,0,3,3,double,0>(), workUnit<4,0,4,0,double,0>()};
    static const int u_fwd64_1_10[11] = {workUnit<4,0,0,0,double,1>(), workUnit<4,0,1,0,double,1>(), workUnit<4,0,1,1,double,1>(), workUnit<4,0,2,0,double,1>(), workUnit<4,0,2,1,double,1>(), workUnit<4,0,2,2,double,1>(), workUnit<4,0,3,0,double,1>(), workUnit<4,0,3,1,double,1>(), workUnit<4,0,3,2,double,1>(), workUnit<4,0,3,3,double,1>(), workUnit<4,0,4,0,double,1>()};
    static const int u_fwd64_2_10[11] = {hasFlippedShape<4,0,0,0,double>() ? workUnit<0,0,4,0,double,0>() : 0, hasFlippedShape<4,0,1,0,double>() ? workUnit<1,0,4,0,double,0>() : 0, hasFlippedShape<4,0,1,1,double>() ? workUnit<1,1,4,0,double,0>() : 0, hasFlippedShape<4,0,2,0,double>() ? workUnit<2,0,4,0,double,0>() : 0, hasFlippedShape<4,0,2,1,double>() ? workUnit<2,1,4,0,double,0>() : 0, hasFlippedShape<4,0,2,2,double>() ? workUnit<2,2,4,0,double,0>() : 0, hasFlippedShape<4,0,3,0,double>() ? workUnit<3,0,4,0,double,0>() : 0, hasFlippedShape<4,0,3,1,double>() ? workUnit<3,1,4,0,double,0>() : 0, hasFlippedShape<4,0,3,2,double>() ? workUnit<3,2,4,0,double,0>() : 0, hasFlippedShape<4,0,3,3,double>() ? workUnit<3,3,4,0,double,0>() : 0, hasFlippedShape<4,0,4,0,double>() ? workUnit<4,0,4,0,double,0>() : 0};
    static const LaunchFn k_fwd64_11[12] = {&launch_fwd64_11_00, &launch_fwd64_11_01, &launch_fwd64_11_02, &launch_fwd64_11_03, &launch_fwd64_11_04, &launch_fwd64_11_05, &launch_fwd64_11_06, &launch_fwd64_11_07, &launch_fwd64_11_08, &launch_fwd64_11_09, &launch_fwd64_11_10, &launch_fwd64_11_11};
    static const LaunchFn k_fwd64v_11[12] = {hasShapeVariant<5,0,0,0,double>() ? &launch_fwd64_11_00_v1 : nullptr, hasShapeVariant<5,0,1,0,double>() ? &launch_fwd64_11_01_v1 : nullptr, hasShapeVariant<5,0,1,1,double>() ? &launch_fwd64_11_02_v1 : nullptr, hasShapeVariant<5,0,2,0,double>() ? &launch_fwd64_11_03_v1 : nullptr, hasShapeVariant<5,0,2,1,double>() ? &launch_fwd64_11_04_v1 : nullptr, hasShapeVariant<5,0,2,2,double>() ? &launch_fwd64_11_05_v1 : nullptr, hasShapeVariant<5,0,3,0,double>() ? &launch_fwd64_11_06_v1 : nullptr, hasShapeVariant<5,0,3,1,double>() ? &launch_fwd64_11_07_v1 : nullptr, hasShapeVariant<5,0,3,2,double>() ? &launch_fwd64_11_08_v1 : nullptr, hasShapeVariant<5,0,3,3,double>() ? &launch_fwd64_11_09_v1 : nullptr, hasShapeVariant<5,0,4,0,double>() ? &launch_fwd64_11_10_v1 : nullptr, hasShapeVariant<5,0,5,0,double>() ? &launch_fwd64_11_11_v1 : nullptr};
    static const LaunchFn k_fwd64f_11[12] = {hasFlippedShape<5,0,0,0,double>() ? &launch_fwd64_11_00_f : nullptr, hasFlippedShape<5,0,1,0,double>() ? &launch_fwd64_11_01_f : nullptr, hasFlippedShape<5,0,1,1,double>() ? &launch_fwd64_11_02_f : nullptr, hasFlippedShape<5,0,2,0,double>() ? &launch_fwd64_11_03_f : nullptr, hasFlippedShape<5,0,2,1,double>() ? &launch_fwd64_11_04_f : nullptr, hasFlippedShape<5,0,2,2,double>() ? &launch_fwd64_11_05_f : nullptr, hasFlippedShape<5,0,3,0,double>() ? &launch_fwd64_11_06_f : nullptr, hasFlippedShape<5,0,3,1,double>() ? &launch_fwd64_11_07_f : nullptr, hasFlippedShape<5,0,3,2,double>() ? &launch_fwd64_11_08_f : nullptr, hasFlippedShape<5,0,3,3,double>() ? &launch_fwd64_11_09_f : nullptr, hasFlippedShape<5,0,4,0,double>() ? &launch_fwd64_11_10_f : nullptr, hasFlippedShape<5,0,5,0,double>() ? &launch_fwd64_11_11_f : nullptr};
    static const int u_fwd64_0_11[12] = {workUnit<5,0,0,0,double,0>(), workUnit<5,0,1,0,double,0>(), workUnit<5,0,1,1,double,0>(), workUnit<5,0,2,0,double,0>(), workUnit<5,0,2,1,double,0>(), workUnit<5,0,2,2,double,0>(), workUnit<5,0,3,0,double,0>(), workUnit<5,0,3,1,double,0>(), workUnit<5,0,3,2,double,0>(), workUnit<5,0,3,3,double,0>(), workUnit<5,0,4,0,double,0>(), workUnit<5,0,5,0,double,0>()};
    static const int u_fwd64_1_11[12] = {workUnit<5,0,0,0,double,1>(), workUnit<5,0,1,0,double,1>(), workUnit<5,0,1,1,double,1>(), workUnit<5,0,2,0,double,1>(), workUnit<5,0,2,1,double,1>(), workUnit<5,0,2,2,double,1>(), workUnit<5,0,3,0,double,1>(), workUnit<5,0,3,1,double,1>(), workUnit<5,0,3,2,double,1>(), workUnit<5,0,3,3,double,1>(), workUnit<5,0,4,0,double,1>(), workUnit<5,0,5,0,double,1>()};
    static const int u_fwd64_2_11[12] = {hasFlippedShape<5,0,0,0,double>() ? workUnit<0,0,5,0,double,0>() : 0, hasFlippedShape<5,0,1,0,double>() ? workUnit<1,0,5,0,double,0>() : 0, hasFlippedShape<5,0,1,1,double>() ? workUnit<1,1,5,0,double,0>() : 0, hasFlippedShape<5,0,2,0,double>() ? workUnit<2,0,5,0,double,0>() : 0, hasFlippedShape<5,0,2,1,double>() ? workUnit<2,1,5,0,double,0>() : 0, hasFlippedShape<5,0,2,2,double>() ? workUnit<2,2,5,0,double,0>() : 0, hasFlippedShape<5,0,3,0,double>() ? workUnit<3,0,5,0,double,0>() : 0, hasFlippedShape<5,0,3,1,double>() ? workUnit<3,1,5,0,double,0>() : 0, hasFlippedShape<5,0,3,2,double>() ? workUnit<3,2,5,0,double,0>() : 0, hasFlippedShape<5,0,3,3,double>() ? workUnit<3,3,5,0,double,0>() : 0, hasFlippedShape<5,0,4,0,double>() ? workUnit<4,0,5,0,double,0>() : 0, hasFlippedShape<5,0,5,0,double>() ? workUnit<5,0,5,0,double,0>() : 0};
    static const int *const u_fwd64_0[12] = {u_fwd64_0_00, u_fwd64_0_01, u_fwd64_0_02, u_fwd64_0_03, u_fwd64_0_04, u_fwd64_0_05, u_fwd64_0_06, u_fwd64_0_07, u_fwd64_0_08, u_fwd64_0_09, u_fwd64_0_10, u_fwd64_0_11};
    static const int *const u_fwd64_1[12] = {u_fwd64_1_00, u_fwd64_1_01, u_fwd64_1_02, u_fwd64_1_03, u_fwd64_1_04, u_fwd64_1_05, u_fwd64_1_06, u_fwd64_1_07, u_fwd64_1_08, u_fwd64_1_09, u_fwd64_1_10, u_fwd64_1_11};
    static const int *const u_fwd64_2[12] = {u_fwd64_2_00, u_fwd64_2_01, u_fwd64_2_02, u_fwd64_2_03, u_fwd64_2_04, u_fwd64_2_05, u_fwd64_2_06, u_fwd64_2_07, u_fwd64_2_08, u_fwd64_2_09, u_fwd64_2_10, u_fwd64_2_11};
    static const LaunchFn *const k_fwd64v[12] = {k_fwd64v_00, k_fwd64v_01, k_fwd64v_02, k_fwd64v_03, k_fwd64v_04, k_fwd64v_05, k_fwd64v_06, k_fwd64v_07, k_fwd64v_08, k_fwd64v_09, k_fwd64v_10, k_fwd64v_11};
    static const LaunchFn *const k_fwd64f[12] = {k_fwd64f_00, k_fwd64f_01, k_fwd64f_02, k_fwd64f_03, k_fwd64f_04, k_fwd64f_05, k_fwd64f_06, k_fwd64f_07, k_fwd64f_08, k_fwd64f_09, k_fwd64f_10, k_fwd64f_11};
    static const LaunchFn *const k_fwd64[12] = {k_fwd64_00, k_fwd64_01, k_fwd64_02, k_fwd64_03, k_fwd64_04, k_fwd64_05, k_fwd64_06, k_fwd64_07, k_fwd64_08, k_fwd64_09, k_fwd64_10, k_fwd64_11};
    cudaError_t launch_fwd32_00_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_01_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_01_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_00_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_01_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_01_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_08_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_00_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_01_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_02_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_03_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_04_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_05_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_06_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_07_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_08_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_09_v1(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_00_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_01_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_01_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_02_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_03_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_04_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_05_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_06_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_07_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_08_08_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_00_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_01_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_02_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_03_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_04_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_05_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_06_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_07_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_08_f(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_fwd32_09_09_f(const QuartetArgs &, cudaStream_t, int);
    static const LaunchFn k_fwd32_00[1] = {&launch_fwd32_00_00};
    static const LaunchFn k_fwd32v_00[1] = {hasShapeVariant<0,0,0,0,float>() ? &launch_fwd32_00_00_v1 : nullptr};
    static const LaunchFn k_fwd32f_00[1] = {hasFlippedShape<0,0,0,0,float>() ? &launch_fwd32_00_00_f : nullptr};
    static const int u_fwd32_0_00[1] = {workUnit<0,0,0,0,float,0>()};
    static const int u_fwd32_1_00[1] = {workUnit<0,0,0,0,float,1>()};
    static const int u_fwd32_2_00[1] = {hasFlippedShape<0,0,0,0,float>() ? workUnit<0,0,0,0,float,0>() : 0};
    static const LaunchFn k_fwd32_01[2] = {&launch_fwd32_01_00, &launch_fwd32_01_01};
    static const LaunchFn k_fwd32v_01[2] = {hasShapeVariant<1,0,0,0,float>() ? &launch_fwd32_01_00_v1 : nullptr, hasShapeVariant<1,0,1,0,float>() ? &launch_fwd32_01_01_v1 : nullptr};
    static const LaunchFn k_fwd32f_01[2] = {hasFlippedShape<1,0,0,0,float>() ? &launch_fwd32_01_00_f : nullptr, hasFlippedShape<1,0,1,0,float>() ? &launch_fwd32_01_01_f : nullptr};
    static const int u_fwd32_0_01[2] = {workUnit<1,0,0,0,float,0>(), workUnit<1,0,1,0,float,0>()};
    static const int u_fwd32_1_01[2] = {workUnit<1,0,0,0,float,1>(), workUnit<1,0,1,0,float,1>()};
    static const int u_fwd32_2_01[2] = {hasFlippedShape<1,0,0,0,float>() ? workUnit<0,0,1,0,float,0>() : 0, hasFlippedShape<1,0,1,0,float>() ? workUnit<1,0,1,0,float,0>() : 0};
    static const LaunchFn k_fwd32_02[3] = {&launch_fwd32_02_00, &launch_fwd32_02_01, &launch_fwd32_02_02};
    static const LaunchFn k_fwd32v_02[3] = {hasShapeVariant<1,1,0,0,float>() ? &launch_fwd32_02_00_v1 : nullptr, hasShapeVariant<1,1,1,0,float>() ? &launch_fwd32_02_01_v1 : nullptr, hasShapeVariant<1,1,1,1,float>() ? &launch_fwd32_02_02_v1 : nullptr};
    static const LaunchFn k_fwd32f_02[3] = {hasFlippedShape<1,1,0,0,float>() ? &launch_fwd32_02_00_f : nullptr, hasFlippedShape<1,1,1,0,float>() ? &launch_fwd32_02_01_f : nullptr, hasFlippedShape<1,1,1,1,float>() ? &launch_fwd32_02_02_f : nullptr};
    static const int u_fwd32_0_02[3] = {workUnit<1,1,0,0,float,0>(), workUnit<1,1,1,0,float,0>(), workUnit<1,1,1,1,float,0>()};
    static const int u_fwd32_1_02[3] = {workUnit<1,1,0,0,float,1>(), workUnit<1,1,1,0,float,1>(), workUnit<1,1,1,1,float,1>()};
    static const int u_fwd32_2_02[3] = {hasFlippedShape<1,1,0,0,float>() ? workUnit<0,0,1,1,float,0>() : 0, hasFlippedShape<1,1,1,0,float>() ? workUnit<1,0,1,1,float,0>() : 0, hasFlippedShape<1,1,1,1,float>() ? workUnit<1,1,1,1,float,0>() : 0};
    static const LaunchFn k_fwd32_03[4] = {&launch_fwd32_03_00, &launch_fwd32_03_01, &launch_fwd32_03_02, &launch_fwd32_03_03};
    static const LaunchFn k_fwd32v_03[4] = {hasShapeVariant<2,0,0,0,float>() ? &launch_fwd32_03_00_v1 : nullptr, hasShapeVariant<2,0,1,0,float>() ? &launch_fwd32_03_01_v1 : nullptr, hasShapeVariant<2,0,1,1,float>() ? &launch_fwd32_03_02_v1 : nullptr, hasShapeVariant<2,0,2,0,float>() ? &launch_fwd32_03_03_v1 : nullptr};
    static const LaunchFn k_fwd32f_03[4] = {hasFlippedShape<2,0,0,0,float>() ? &launch_fwd32_03_00_f : nullptr, hasFlippedShape<2,0,1,0,float>() ? &launch_fwd32_03_01_f : nullptr, hasFlippedShape<2,0,1,1,float>() ? &launch_fwd32_03_02_f : nullptr, hasFlippedShape<2,0,2,0,float>() ? &launch_fwd32_03_03_f : nullptr};
    static const int u_fwd32_0_03[4] = {workUnit<2,0,0,0,float,0>(), workUnit<2,0,1,0,float,0>(), workUnit<2,0,1,1,float,0>(), workUnit<2,0,2,0,float,0>()};
    static const int u_fwd32_1_03[4] = {workUnit<2,0,0,0,float,1>(), workUnit<2,0,1,0,float,1>(), workUnit<2,0,1,1,float,1>(), workUnit<2,0,2,0,float,1>()};
    static const int u_fwd32_2_03[4] = {hasFlippedShape<2,0,0,0,float>() ? workUnit<0,0,2,0,float,0>() : 0, hasFlippedShape<2,0,1,0,float>() ? workUnit<1,0,2,0,float,0>() : 0, hasFlippedShape<2,0,1,1,float>() ? workUnit<1,1,2,0,float,0>() : 0, hasFlippedShape<2,0,2,0,float>() ? workUnit<2,0,2,0,float,0>() : 0};
    static const LaunchFn k_fwd32_04[5] = {&launch_fwd32_04_00, &launch_fwd32_04_01, &launch_fwd32_04_02, &launch_fwd32_04_03, &launch_fwd32_04_04};
    static const LaunchFn k_fwd32v_04[5] = {hasShapeVariant<2,1,0,0,float>() ? &launch_fwd32_04_00_v1 : nullptr, hasShapeVariant<2,1,1,0,float>() ? &launch_fwd32_04_01_v1 : nullptr, hasShapeVariant<2,1,1,1,float>() ? &launch_fwd32_04_02_v1 : nullptr, hasShapeVariant<2,1,2,0,float>() ? &launch_fwd32_04_03_v1 : nullptr, hasShapeVariant<2,1,2,1,float>() ? &launch_fwd32_04_04_v1 : nullptr};
    static const LaunchFn k_fwd32f_04[5] = {hasFlippedShape<2,1,0,0,float>() ? &launch_fwd32_04_00_f : nullptr, hasFlippedShape<2,1,1,0,float>() ? &launch_fwd32_04_01_f : nullptr, hasFlippedShape<2,1,1,1,float>() ? &launch_fwd32_04_02_f : nullptr, hasFlippedShape<2,1,2,0,float>() ? &launch_fwd32_04_03_f : nullptr, hasFlippedShape<2,1,2,1,float>() ? &launch_fwd32_04_04_f : nullptr};
    static const int u_fwd32_0_04[5] = {workUnit<2,1,0,0,float,0>(), workUnit<2,1,1,0,float,0>(), workUnit<2,1,1,1,float,0>(), workUnit<2,1,2,0,float,0>(), workUnit<2,1,2,1,float,0>()};
    static const int u_fwd32_1_04[5] = {workUnit<2,1,0,0,float,1>(), workUnit<2,1,1,0,float,1>(), workUnit<2,1,1,1,float,1>(), workUnit<2,1,2,0,float,1>(), workUnit<2,1,2,1,float,1>()};
    static const int u_fwd32_2_04[5] = {hasFlippedShape<2,1,0,0,float>() ? workUnit<0,0,2,1,float,0>() : 0, hasFlippedShape<2,1,1,0,float>() ? workUnit<1,0,2,1,float,0>() : 0, hasFlippedShape<2,1,1,1,float>() ? workUnit<1,1,2,1,float,0>() : 0, hasFlippedShape<2,1,2,0,float>() ? workUnit<2,0,2,1,float,0>() : 0, hasFlippedShape<2,1,2,1,float>() ? workUnit<2,1,2,1,float,0>() : 0};
    static const LaunchFn k_fwd32_05[6] = {&launch_fwd32_05_00, &launch_fwd32_05_01, &launch_fwd32_05_02, &launch_fwd32_05_03, &launch_fwd32_05_04, &launch_fwd32_05_05};
    static const LaunchFn k_fwd32v_05[6] = {hasShapeVariant<2,2,0,0,float>() ? &launch_fwd32_05_00_v1 : nullptr, hasShapeVariant<2,2,1,0,float>() ? &launch_fwd32_05_01_v1 : nullptr, hasShapeVariant<2,2,1,1,float>() ? &launch_fwd32_05_02_v1 : nullptr, hasShapeVariant<2,2,2,0,float>() ? &launch_fwd32_05_03_v1 : nullptr, hasShapeVariant<2,2,2,1,float>() ? &launch_fwd32_05_04_v1 : nullptr, hasShapeVariant<2,2,2,2,float>() ? &launch_fwd32_05_05_v1 : nullptr};
    static const LaunchFn k_fwd32f_05[6] = {hasFlippedShape<2,2,0,0,float>() ? &launch_fwd32_05_00_f : nullptr, hasFlippedShape<2,2,1,0,float>() ? &launch_fwd32_05_01_f : nullptr, hasFlippedShape<2,2,1,1,float>() ? &launch_fwd32_05_02_f : nullptr, hasFlippedShape<2,2,2,0,float>() ? &launch_fwd32_05_03_f : nullptr, hasFlippedShape<2,2,2,1,float>() ? &launch_fwd32_05_04_f : nullptr, hasFlippedShape<2,2,2,2,float>() ? &launch_fwd32_05_05_f : nullptr};
    static const int u_fwd32_0_05[6] = {workUnit<2,2,0,0,float,0>(), workUnit<2,2,1,0,float,0>(), workUnit<2,2,1,1,float,0>(), workUnit<2,2,2,0,float,0>(), workUnit<2,2,2,1,float,0>(), workUnit<2,2,2,2,float,0>()};
    static const int u_fwd32_1_05[6] = {workUnit<2,2,0,0,float,1>(), workUnit<2,2,1,0,float,1>(), workUnit<2,2,1,1,float,1>(), workUnit<2,2,2,0,float,1>(), workUnit<2,2,2,1,float,1>(), workUnit<2,2,2,2,float,1>()};
    static const int u_fwd32_2_05[6] = {hasFlippedShape<2,2,0,0,float>() ? workUnit<0,0,2,2,float,0>() : 0, hasFlippedShape<2,2,1,0,float>() ? workUnit<1,0,2,2,float,0>() : 0, hasFlippedShape<2,2,1,1,float>() ? workUnit<1,1,2,2,float,0>() : 0, hasFlippedShape<2,2,2,0,float>() ? workUnit<2,0,2,2,float,0>() : 0, hasFlippedShape<2,2,2,1,float>() ? workUnit<2,1,2,2,float,0>() : 0, hasFlippedShape<2,2,2,2,float>() ? workUnit<2,2,2,2,float,0>() : 0};
    static const LaunchFn k_fwd32_06[7] = {&launch_fwd32_06_00, &launch_fwd32_06_01, &launch_fwd32_06_02, &launch_fwd32_06_03, &launch_fwd32_06_04, &launch_fwd32_06_05, &launch_fwd32_06_06};
    static const LaunchFn k_fwd32v_06[7] = {hasShapeVariant<3,0,0,0,float>() ? &launch_fwd32_06_00_v1 : nullptr, hasShapeVariant<3,0,1,0,float>() ? &launch_fwd32_06_01_v1 : nullptr, hasShapeVariant<3,0,1,1,float>() ? &launch_fwd32_06_02_v1 : nullptr, hasShapeVariant<3,0,2,0,float>() ? &launch_fwd32_06_03_v1 : nullptr, hasShapeVariant<3,0,2,1,float>() ? &launch_fwd32_06_04_v1 : nullptr, hasShapeVariant<3,0,2,2,float>() ? &launch_fwd32_06_05_v1 : nullptr, hasShapeVariant<3,0,3,0,float>() ? &launch_fwd32_06_06_v1 : nullptr};
    static const LaunchFn k_fwd32f_06[7] = {hasFlippedShape<3,0,0,0,float>() ? &launch_fwd32_06_00_f : nullptr, hasFlippedShape<3,0,1,0,float>() ? &launch_fwd32_06_01_f : nullptr, hasFlippedShape<3,0,1,1,float>() ? &launch_fwd32_06_02_f : nullptr, hasFlippedShape<3,0,2,0,float>() ? &launch_fwd32_06_03_f : nullptr, hasFlippedShape<3,0,2,1,float>() ? &launch_fwd32_06_04_f : nullptr, hasFlippedShape<3,0,2,2,float>() ? &launch_fwd32_06_05_f : nullptr, hasFlippedShape<3,0,3,0,float>() ? &launch_fwd32_06_06_f : nullptr};
    static const int u_fwd32_0_06[7] = {workUnit<3,0,0,0,float,0>(), workUnit<3,0,1,0,float,0>(), workUnit<3,0,1,1,float,0>(), workUnit<3,0,2,0,float,0>(), workUnit<3,0,2,1,float,0>(), workUnit<3,0,2,2,float,0>(), workUnit<3,0,3,0,float,0>()};
    static const int u_fwd32_1_06[7] = {workUnit<3,0,0,0,float,1>(), workUnit<3,0,1,0,float,1>(), workUnit<3,0,1,1,float,1>(), workUnit<3,0,2,0,float,1>(), workUnit<3,0,2,1,float,1>(), workUnit<3,0,2,2,float,1>(), workUnit<3,0,3,0,float,1>()};
    static const int u_fwd32_2_06[7] = {hasFlippedShape<3,0,0,0,float>() ? workUnit<0,0,3,0,float,0>() : 0, hasFlippedShape<3,0,1,0,float>() ? workUnit<1,0,3,0,float,0>() : 0, hasFlippedShape<3,0,1,1,float>() ? workUnit<1,1,3,0,float,0>() : 0, hasFlippedShape<3,0,2,0,float>() ? workUnit<2,0,3,0,float,0>() : 0, hasFlippedShape<3,0,2,1,float>() ? workUnit<2,1,3,0,float,0>() : 0, hasFlippedShape<3,0,2,2,float>() ? workUnit<2,2,3,0,float,0>() : 0, hasFlippedShape<3,0,3,0,float>() ? workUnit<3,0,3,0,float,0>() : 0};
    static const LaunchFn k_fwd32_07[8] = {&launch_fwd32_07_00, &launch_fwd32_07_01, &launch_fwd32_07_02, &launch_fwd32_07_03, &launch_fwd32_07_04, &launch_fwd32_07_05, &launch_fwd32_07_06, &launch_fwd32_07_07};
    static const LaunchFn k_fwd32v_07[8] = {hasShapeVariant<3,1,0,0,float>() ? &launch_fwd32_07_00_v1 : nullptr, hasShapeVariant<3,1,1,0,float>() ? &launch_fwd32_07_01_v1 : nullptr, hasShapeVariant<3,1,1,1,float>() ? &launch_fwd32_07_02_v1 : nullptr, hasShapeVariant<3,1,2,0,float>() ? &launch_fwd32_07_03_v1 : nullptr, hasShapeVariant<3,1,2,1,float>() ? &launch_fwd32_07_04_v1 : nullptr, hasShapeVariant<3,1,2,2,float>() ? &launch_fwd32_07_05_v1 : nullptr, hasShapeVariant<3,1,3,0,float>() ? &launch_fwd32_07_06_v1 : nullptr, hasShapeVariant<3,1,3,1,float>() ? &launch_fwd32_07_07_v1 : nullptr};
    static const LaunchFn k_fwd32f_07[8] = {hasFlippedShape<3,1,0,0,float>() ? &launch_fwd32_07_00_f : nullptr, hasFlippedShape<3,1,1,0,float>() ? &launch_fwd32_07_01_f : nullptr, hasFlippedShape<3,1,1,1,float>() ? &launch_fwd32_07_02_f : nullptr, hasFlippedShape<3,1,2,0,float>() ? &launch_fwd32_07_03_f : nullptr, hasFlippedShape<3,1,2,1,float>() ? &launch_fwd32_07_04_f : nullptr, hasFlippedShape<3,1,2,2,float>() ? &launch_fwd32_07_05_f : nullptr, hasFlippedShape<3,1,3,0,float>() ? &launch_fwd32_07_06_f : nullptr, hasFlippedShape<3,1,3,1,float>() ? &launch_fwd32_07_07_f : nullptr};
    static const int u_fwd32_0_07[8] = {workUnit<3,1,0,0,float,0>(), workUnit<3,1,1,0,float,0>(), workUnit<3,1,1,1,float,0>(), workUnit<3,1,2,0,float,0>(), workUnit<3,1,2,1,float,0>(), workUnit<3,1,2,2,float,0>(), workUnit<3,1,3,0,float,0>(), workUnit<3,1,3,1,float,0>()};
    static const int u_fwd32_1_07[8] = {workUnit<3,1,0,0,float,1>(), workUnit<3,1,1,0,float,1>(), workUnit<3,1,1,1,float,1>(), workUnit<3,1,2,0,float,1>(), workUnit<3,1,2,1,float,1>(), workUnit<3,1,2,2,float,1>(), workUnit<3,1,3,0,float,1>(), workUnit<3,1,3,1,float,1>()};
    static const int u_fwd32_2_07[8] = {hasFlippedShape<3,1,0,0,float>() ? workUnit<0,0,3,1,float,0>() : 0, hasFlippedShape<3,1,1,0,float>() ? workUnit<1,0,3,1,float,0>() : 0, hasFlippedShape<3,1,1,1,float>() ? workUnit<1,1,3,1,float,0>() : 0, hasFlippedShape<3,1,2,0,float>() ? workUnit<2,0,3,1,float,0>() : 0, hasFlippedShape<3,1,2,1,float>() ? workUnit<2,1,3,1,float,0>() : 0, hasFlippedShape<3,1,2,2,float>() ? workUnit<2,2,3,1,float,0>() : 0, hasFlippedShape<3,1,3,0,float>() ? workUnit<3,0,3,1,float,0>() : 0, hasFlippedShape<3,1,3,1,float>() ? workUnit<3,1,3,1,float,0>() : 0};
    static const LaunchFn k_fwd32_08[9] = {&launch_fwd32_08_00, &launch_fwd32_08_01, &launch_fwd32_08_02, &launch_fwd32_08_03, &launch_fwd32_08_04, &launch_fwd32_08_05, &launch_fwd32_08_06, &launch_fwd32_08_07, &launch_fwd32_08_08};
    static const LaunchFn k_fwd32v_08[9] = {hasShapeVariant<3,2,0,0,float>() ? &launch_fwd32_08_00_v1 : nullptr, hasShapeVariant<3,2,1,0,float>() ? &launch_fwd32_08_01_v1 : nullptr, hasShapeVariant<3,2,1,1,float>() ? &launch_fwd32_08_02_v1 : nullptr, hasShapeVariant<3,2,2,0,float>() ? &launch_fwd32_08_03_v1 : nullptr, hasShapeVariant<3,2,2,1,float>() ? &launch_fwd32_08_04_v1 : nullptr, hasShapeVariant<3,2,2,2,float>() ? &launch_fwd32_08_05_v1 : nullptr, hasShapeVariant<3,2,3,0,float>() ? &launch_fwd32_08_06_v1 : nullptr, hasShapeVariant<3,2,3,1,float>() ? &launch_fwd32_08_07_v1 : nullptr, hasShapeVariant<3,2,3,2,float>() ? &launch_fwd32_08_08_v1 : nullptr};
    static const LaunchFn k_fwd32f_08[9] = {hasFlippedShape<3,2,0,0,float>() ? &launch_fwd32_08_00_f : nullptr, hasFlippedShape<3,2,1,0,float>() ? &launch_fwd32_08_01_f : nullptr, hasFlippedShape<3,2,1,1,float>() ? &launch_fwd32_08_02_f : nullptr, hasFlippedShape<3,2,2,0,float>() ? &launch_fwd32_08_03_f : nullptr, hasFlippedShape<3,2,2,1,float>() ? &launch_fwd32_08_04_f : nullptr, hasFlippedShape<3,2,2,2,float>() ? &launch_fwd32_08_05_f : nullptr, hasFlippedShape<3,2,3,0,float>() ? &launch_fwd32_08_06_f : nullptr, hasFlippedShape<3,2,3,1,float>() ? &launch_fwd32_08_07_f : nullptr, hasFlippedShape<3,2,3,2,float>() ? &launch_fwd32_08_08_f : nullptr};
    static const int u_fwd32_0_08[9] = {workUnit<3,2,0,0,float,0>(), workUnit<3,2,1,0,float,0>(), workUnit<3,2,1,1,float,0>(), workUnit<3,2,2,0,float,0>(), workUnit<3,2,2,1,float,0>(), workUnit<3,2,2,2,float,0>(), workUnit<3,2,3,0,float,0>(), workUnit<3,2,3,1,float,0>(), workUnit<3,2,3,2,float,0>()};
    static const int u_fwd32_1_08[9] = {workUnit<3,2,0,0,float,1>(), workUnit<3,2,1,0,float,1>(), workUnit<3,2,1,1,float,1>(), workUnit<3,2,2,0,float,1>(), workUnit<3,2,2,1,float,1>(), workUnit<3,2,2,2,float,1>(), workUnit<3,2,3,0,float,1>(), workUnit<3,2,3,1,float,1>(), workUnit<3,2,3,2,float,1>()};
    static const int u_fwd32_2_08[9] = {hasFlippedShape<3,2,0,0,float>() ? workUnit<0,0,3,2,float,0>() : 0, hasFlippedShape<3,2,1,0,float>() ? workUnit<1,0,3,2,float,0>() : 0, hasFlippedShape<3,2,1,1,float>() ? workUnit<1,1,3,2,float,0>() : 0, hasFlippedShape<3,2,2,0,float>() ? workUnit<2,0,3,2,float,0>() : 0, hasFlippedShape<3,2,2,1,float>() ? workUnit<2,1,3,2,float,0>() : 0, hasFlippedShape<3,2,2,2,float>() ? workUnit<2,2,3,2,float,0>() : 0, hasFlippedShape<3,2,3,0,float>() ? workUnit<3,0,3,2,float,0>() : 0, hasFlippedShape<3,2,3,1,float>() ? workUnit<3,1,3,2,float,0>() : 0, hasFlippedShape<3,2,3,2,float>() ? workUnit<3,2,3,2,float,0>() : 0};
    static const LaunchFn k_fwd32_09[10] = {&launch_fwd32_09_00, &launch_fwd32_09_01, &launch_fwd32_09_02, &launch_fwd32_09_03, &launch_fwd32_09_04, &launch_fwd32_09_05, &launch_fwd32_09_06, &launch_fwd32_09_07, &launch_fwd32_09_08, &launch_fwd32_09_09};
    static const LaunchFn k_fwd32v_09[10] = {hasShapeVariant<3,3,0,0,float>() ? &launch_fwd32_09_00_v1 : nullptr, hasShapeVariant<3,3,1,0,float>() ? &launch_fwd32_09_01_v1 : nullptr, hasShapeVariant<3,3,1,1,float>() ? &launch_fwd32_09_02_v1 : nullptr, hasShapeVariant<3,3,2,0,float>() ? &launch_fwd32_09_03_v1 : nullptr, hasShapeVariant<3,3,2,1,float>() ? &launch_fwd32_09_04_v1 : nullptr, hasShapeVariant<3,3,2,2,float>() ? &launch_fwd32_09_05_v1 : nullptr, hasShapeVariant<3,3,3,0,float>() ? &launch_fwd32_09_06_v1 : nullptr, hasShapeVariant<3,3,3,1,float>() ? &launch_fwd32_09_07_v1 : nullptr, hasShapeVariant<3,3,3,2,float>() ? &launch_fwd32_09_08_v1 : nullptr, hasShapeVariant<3,3,3,3,float>() ? &launch_fwd32_09_09_v1 : nullptr};
    static const LaunchFn k_fwd32f_09[10] = {hasFlippedShape<3,3,0,0,float>() ? &launch_fwd32_09_00_f : nullptr, hasFlippedShape<3,3,1,0,float>() ? &launch_fwd32_09_01_f : nullptr, hasFlippedShape<3,3,1,1,float>() ? &launch_fwd32_09_02_f : nullptr, hasFlippedShape<3,3,2,0,float>() ? &launch_fwd32_09_03_f : nullptr, hasFlippedShape<3,3,2,1,float>() ? &launch_fwd32_09_04_f : nullptr, hasFlippedShape<3,3,2,2,float>() ? &launch_fwd32_09_05_f : nullptr, hasFlippedShape<3,3,3,0,float>() ? &launch_fwd32_09_06_f : nullptr, hasFlippedShape<3,3,3,1,float>() ? &launch_fwd32_09_07_f : nullptr, hasFlippedShape<3,3,3,2,float>() ? &launch_fwd32_09_08_f : nullptr, hasFlippedShape<3,3,3,3,float>() ? &launch_fwd32_09_09_f : nullptr};
    static const int u_fwd32_0_09[10] = {workUnit<3,3,0,0,float,0>(), workUnit<3,3,1,0,float,0>(), workUnit<3,3,1,1,float,0>(), workUnit<3,3,2,0,float,0>(), workUnit<3,3,2,1,float,0>(), workUnit<3,3,2,2,float,0>(), workUnit<3,3,3,0,float,0>(), workUnit<3,3,3,1,float,0>(), workUnit<3,3,3,2,float,0>(), workUnit<3,3,3,3,float,0>()};
    static const int u_fwd32_1_09[10] = {workUnit<3,3,0,0,float,1>(), workUnit<3,3,1,0,float,1>(), workUnit<3,3,1,1,float,1>(), workUnit<3,3,2,0,float,1>(), workUnit<3,3,2,1,float,1>(), workUnit<3,3,2,2,float,1>(), workUnit<3,3,3,0,float,1>(), workUnit<3,3,3,1,float,1>(), workUnit<3,3,3,2,float,1>(), workUnit<3,3,3,3,float,1>()};
    static const int u_fwd32_2_09[10] = {hasFlippedShape<3,3,0,0,float>() ? workUnit<0,0,3,3,float,0>() : 0, hasFlippedShape<3,3,1,0,float>() ? workUnit<1,0,3,3,float,0>() : 0, hasFlippedShape<3,3,1,1,float>() ? workUnit<1,1,3,3,float,0>() : 0, hasFlippedShape<3,3,2,0,float>() ? workUnit<2,0,3,3,float,0>() : 0, hasFlippedShape<3,3,2,1,float>() ? workUnit<2,1,3,3,float,0>() : 0, hasFlippedShape<3,3,2,2,float>() ? workUnit<2,2,3,3,float,0>() : 0, hasFlippedShape<3,3,3,0,float>() ? workUnit<3,0,3,3,float,0>() : 0, hasFlippedShape<3,3,3,1,float>() ? workUnit<3,1,3,3,float,0>() : 0, hasFlippedShape<3,3,3,2,float>() ? workUnit<3,2,3,3,float,0>() : 0, hasFlippedShape<3,3,3,3,float>() ? workUnit<3,3,3,3,float,0>() : 0};
    static const int *const u_fwd32_0[10] = {u_fwd32_0_00, u_fwd32_0_01, u_fwd32_0_02, u_fwd32_0_03, u_fwd32_0_04, u_fwd32_0_05, u_fwd32_0_06, u_fwd32_0_07, u_fwd32_0_08, u_fwd32_0_09};
    static const int *const u_fwd32_1[10] = {u_fwd32_1_00, u_fwd32_1_01, u_fwd32_1_02, u_fwd32_1_03, u_fwd32_1_04, u_fwd32_1_05, u_fwd32_1_06, u_fwd32_1_07, u_fwd32_1_08, u_fwd32_1_09};
    static const int *const u_fwd32_2[10] = {u_fwd32_2_00, u_fwd32_2_01, u_fwd32_2_02, u_fwd32_2_03, u_fwd32_2_04, u_fwd32_2_05, u_fwd32_2_06, u_fwd32_2_07, u_fwd32_2_08, u_fwd32_2_09};
    static const LaunchFn *const k_fwd32v[10] = {k_fwd32v_00, k_fwd32v_01, k_fwd32v_02, k_fwd32v_03, k_fwd32v_04, k_fwd32v_05, k_fwd32v_06, k_fwd32v_07, k_fwd32v_08, k_fwd32v_09};
    static const LaunchFn *const k_fwd32f[10] = {k_fwd32f_00, k_fwd32f_01, k_fwd32f_02, k_fwd32f_03, k_fwd32f_04, k_fwd32f_05, k_fwd32f_06, k_fwd32f_07, k_fwd32f_08, k_fwd32f_09};
    static const LaunchFn *const k_fwd32[10] = {k_fwd32_00, k_fwd32_01, k_fwd32_02, k_fwd32_03, k_fwd32_04, k_fwd32_05, k_fwd32_06, k_fwd32_07, k_fwd32_08, k_fwd32_09};
    cudaError_t launch_d1_00_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_01_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_01_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_02_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_02_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_02_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_03_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_03_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_03_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_03_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_04_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_04_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_04_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_04_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_04_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_05_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_05_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_05_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_05_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_05_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_05_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_06_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_07_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_08_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_09_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_10_10(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_05(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_07(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_08(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_09(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_10(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_d1_11_11(const QuartetArgs &, cudaStream_t, int);
    static const LaunchFn k_d1_00[1] = {&launch_d1_00_00};
    static const LaunchFn k_d1_01[2] = {&launch_d1_01_00, &launch_d1_01_01};
    static const LaunchFn k_d1_02[3] = {&launch_d1_02_00, &launch_d1_02_01, &launch_d1_02_02};
    static const LaunchFn k_d1_03[4] = {&launch_d1_03_00, &launch_d1_03_01, &launch_d1_03_02, &launch_d1_03_03};
    static const LaunchFn k_d1_04[5] = {&launch_d1_04_00, &launch_d1_04_01, &launch_d1_04_02, &launch_d1_04_03, &launch_d1_04_04};
    static const LaunchFn k_d1_05[6] = {&launch_d1_05_00, &launch_d1_05_01, &launch_d1_05_02, &launch_d1_05_03, &launch_d1_05_04, &launch_d1_05_05};
    static const LaunchFn k_d1_06[7] = {&launch_d1_06_00, &launch_d1_06_01, &launch_d1_06_02, &launch_d1_06_03, &launch_d1_06_04, &launch_d1_06_05, &launch_d1_06_06};
    static const LaunchFn k_d1_07[8] = {&launch_d1_07_00, &launch_d1_07_01, &launch_d1_07_02, &launch_d1_07_03, &launch_d1_07_04, &launch_d1_07_05, &launch_d1_07_06, &launch_d1_07_07};
    static const LaunchFn k_d1_08[9] = {&launch_d1_08_00, &launch_d1_08_01, &launch_d1_08_02, &launch_d1_08_03, &launch_d1_08_04, &launch_d1_08_05, &launch_d1_08_06, &launch_d1_08_07, &launch_d1_08_08};
    static const LaunchFn k_d1_09[10] = {&launch_d1_09_00, &launch_d1_09_01, &launch_d1_09_02, &launch_d1_09_03, &launch_d1_09_04, &launch_d1_09_05, &launch_d1_09_06, &launch_d1_09_07, &launch_d1_09_08, &launch_d1_09_09};
    static const LaunchFn k_d1_10[11] = {&launch_d1_10_00, &launch_d1_10_01, &launch_d1_10_02, &launch_d1_10_03, &launch_d1_10_04, &launch_d1_10_05, &launch_d1_10_06, &launch_d1_10_07, &launch_d1_10_08, &launch_d1_10_09, &launch_d1_10_10};
    static const LaunchFn k_d1_11[12] = {&launch_d1_11_00, &launch_d1_11_01, &launch_d1_11_02, &launch_d1_11_03, &launch_d1_11_04, &launch_d1_11_05, &launch_d1_11_06, &launch_d1_11_07, &launch_d1_11_08, &launch_d1_11_09, &launch_d1_11_10, &launch_d1_11_11};
    static const LaunchFn *const k_d1[12] = {k_d1_00, k_d1_01, k_d1_02, k_d1_03, k_d1_04, k_d1_05, k_d1_06, k_d1_07, k_d1_08, k_d1_09, k_d1_10, k_d1_11};
    cudaError_t launch_split64_00_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_01_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_01_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_02_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_02_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_02_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_03_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_03_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_03_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_03_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_04_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_04_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_04_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_04_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_04_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_05_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_05_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_05_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_05_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_06_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_06_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_06_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_06_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_06_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_06_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_07_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_07_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_07_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_07_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_08_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_08_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split64_09_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_00_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_01_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_01_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_02_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_02_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_02_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_03_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_03_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_03_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_03_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_04_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_04_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_04_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_04_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_04_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_05_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_05_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_05_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_05_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_06_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_06_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_06_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_06_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_06_04(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_06_06(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_07_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_07_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_07_02(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_07_03(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_08_00(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_08_01(const QuartetArgs &, cudaStream_t, int);
    cudaError_t launch_split32_09_00(const QuartetArgs &, cudaStream_t, int);
    LaunchFn lookupSplit(int bt, int kt, bool fp32)
    {
        switch (100 * bt + kt)
        {
        case 0:
            if (fp32)
                return hasSplitForm<0,0,0,0,float>() || hasSplitForm<0,0,0,0,float>() ? &launch_split32_00_00 : nullptr;
            else
                return hasSplitForm<0,0,0,0,double>() || hasSplitForm<0,0,0,0,double>() ? &launch_split64_00_00 : nullptr;
        case 100:
            if (fp32)
                return hasSplitForm<1,0,0,0,float>() || hasSplitForm<0,0,1,0,float>() ? &launch_split32_01_00 : nullptr;
            else
                return hasSplitForm<1,0,0,0,double>() || hasSplitForm<0,0,1,0,double>() ? &launch_split64_01_00 : nullptr;
        case 101:
            if (fp32)
                return hasSplitForm<1,0,1,0,float>() || hasSplitForm<1,0,1,0,float>() ? &launch_split32_01_01 : nullptr;
            else
                return hasSplitForm<1,0,1,0,double>() || hasSplitForm<1,0,1,0,double>() ? &launch_split64_01_01 : nullptr;
        case 200:
            if (fp32)
                return hasSplitForm<1,1,0,0,float>() || hasSplitForm<0,0,1,1,float>() ? &launch_split32_02_00 : nullptr;
            else
                return hasSplitForm<1,1,0,0,double>() || hasSplitForm<0,0,1,1,double>() ? &launch_split64_02_00 : nullptr;
        case 201:
            if (fp32)
                return hasSplitForm<1,1,1,0,float>() || hasSplitForm<1,0,1,1,float>() ? &launch_split32_02_01 : nullptr;
            else
                return hasSplitForm<1,1,1,0,double>() || hasSplitForm<1,0,1,1,double>() ? &launch_split64_02_01 : nullptr;
        case 202:
            if (fp32)
                return hasSplitForm<1,1,1,1,float>() || hasSplitForm<1,1,1,1,float>() ? &launch_split32_02_02 : nullptr;
            else
                return hasSplitForm<1,1,1,1,double>() || hasSplitForm<1,1,1,1,double>() ? &launch_split64_02_02 : nullptr;
        case 300:
            if (fp32)
                return hasSplitForm<2,0,0,0,float>() || hasSplitForm<0,0,2,0,float>() ? &launch_split32_03_00 : nullptr;
            else
                return hasSplitForm<2,0,0,0,double>() || hasSplitForm<0,0,2,0,double>() ? &launch_split64_03_00 : nullptr;
        case 301:
            if (fp32)
                return hasSplitForm<2,0,1,0,float>() || hasSplitForm<1,0,2,0,float>() ? &launch_split32_03_01 : nullptr;
            else
                return hasSplitForm<2,0,1,0,double>() || hasSplitForm<1,0,2,0,double>() ? &launch_split64_03_01 : nullptr;
        case 302:
            if (fp32)
                return hasSplitForm<2,0,1,1,float>() || hasSplitForm<1,1,2,0,float>() ? &launch_split32_03_02 : nullptr;
            else
                return hasSplitForm<2,0,1,1,double>() || hasSplitForm<1,1,2,0,double>() ? &launch_split64_03_02 : nullptr;
        case 303:
            if (fp32)
                return hasSplitForm<2,0,2,0,float>() || hasSplitForm<2,0,2,0,float>() ? &launch_split32_03_03 : nullptr;
            else
                return hasSplitForm<2,0,2,0,double>() || hasSplitForm<2,0,2,0,double>() ? &launch_split64_03_03 : nullptr;
        case 400:
            if (fp32)
                return hasSplitForm<2,1,0,0,float>() || hasSplitForm<0,0,2,1,float>() ? &launch_split32_04_00 : nullptr;
            else
                return hasSplitForm<2,1,0,0,double>() || hasSplitForm<0,0,2,1,double>() ? &launch_split64_04_00 : nullptr;
        case 401:
            if (fp32)
                return hasSplitForm<2,1,1,0,float>() || hasSplitForm<1,0,2,1,float>() ? &launch_split32_04_01 : nullptr;
            else
                return hasSplitForm<2,1,1,0,double>() || hasSplitForm<1,0,2,1,double>() ? &launch_split64_04_01 : nullptr;
        case 402:
            if (fp32)
                return hasSplitForm<2,1,1,1,float>() || hasSplitForm<1,1,2,1,float>() ? &launch_split32_04_02 : nullptr;
            else
                return hasSplitForm<2,1,1,1,double>() || hasSplitForm<1,1,2,1,double>() ? &launch_split64_04_02 : nullptr;
        case 403:
            if (fp32)
                return hasSplitForm<2,1,2,0,float>() || hasSplitForm<2,0,2,1,float>() ? &launch_split32_04_03 : nullptr;
            else
                return hasSplitForm<2,1,2,0,double>() || hasSplitForm<2,0,2,1,double>() ? &launch_split64_04_03 : nullptr;
        case 404:
            if (fp32)
                return hasSplitForm<2,1,2,1,float>() || hasSplitForm<2,1,2,1,float>() ? &launch_split32_04_04 : nullptr;
            else
                return hasSplitForm<2,1,2,1,double>() || hasSplitForm<2,1,2,1,double>() ? &launch_split64_04_04 : nullptr;
        case 500:
            if (fp32)
                return hasSplitForm<2,2,0,0,float>() || hasSplitForm<0,0,2,2,float>() ? &launch_split32_05_00 : nullptr;
            else
                return hasSplitForm<2,2,0,0,double>() || hasSplitForm<0,0,2,2,double>() ? &launch_split64_05_00 : nullptr;
        case 501:
            if (fp32)
                return hasSplitForm<2,2,1,0,float>() || hasSplitForm<1,0,2,2,float>() ? &launch_split32_05_01 : nullptr;
            else
                return hasSplitForm<2,2,1,0,double>() || hasSplitForm<1,0,2,2,double>() ? &launch_split64_05_01 : nullptr;
        case 502:
            if (fp32)
                return hasSplitForm<2,2,1,1,float>() || hasSplitForm<1,1,2,2,float>() ? &launch_split32_05_02 : nullptr;
            else
                return hasSplitForm<2,2,1,1,double>() || hasSplitForm<1,1,2,2,double>() ? &launch_split64_05_02 : nullptr;
        case 503:
            if (fp32)
                return hasSplitForm<2,2,2,0,float>() || hasSplitForm<2,0,2,2,float>() ? &launch_split32_05_03 : nullptr;
            else
                return hasSplitForm<2,2,2,0,double>() || hasSplitForm<2,0,2,2,double>() ? &launch_split64_05_03 : nullptr;
        case 600:
            if (fp32)
                return hasSplitForm<3,0,0,0,float>() || hasSplitForm<0,0,3,0,float>() ? &launch_split32_06_00 : nullptr;
            else
                return hasSplitForm<3,0,0,0,double>() || hasSplitForm<0,0,3,0,double>() ? &launch_split64_06_00 : nullptr;
        case 601:
            if (fp32)
                return hasSplitForm<3,0,1,0,float>() || hasSplitForm<1,0,3,0,float>() ? &launch_split32_06_01 : nullptr;
            else
                return hasSplitForm<3,0,1,0,double>() || hasSplitForm<1,0,3,0,double>() ? &launch_split64_06_01 : nullptr;
        case 602:
            if (fp32)
                return hasSplitForm<3,0,1,1,float>() || hasSplitForm<1,1,3,0,float>() ? &launch_split32_06_02 : nullptr;
            else
                return hasSplitForm<3,0,1,1,double>() || hasSplitForm<1,1,3,0,double>() ? &launch_split64_06_02 : nullptr;
        case 603:
            if (fp32)
                return hasSplitForm<3,0,2,0,float>() || hasSplitForm<2,0,3,0,float>() ? &launch_split32_06_03 : nullptr;
            else
                return hasSplitForm<3,0,2,0,double>() || hasSplitForm<2,0,3,0,double>() ? &launch_split64_06_03 : nullptr;
        case 604:
            if (fp32)
                return hasSplitForm<3,0,2,1,float>() || hasSplitForm<2,1,3,0,float>() ? &launch_split32_06_04 : nullptr;
            else
                return hasSplitForm<3,0,2,1,double>() || hasSplitForm<2,1,3,0,double>() ? &launch_split64_06_04 : nullptr;
        case 606:
            if (fp32)
                return hasSplitForm<3,0,3,0,float>() || hasSplitForm<3,0,3,0,float>() ? &launch_split32_06_06 : nullptr;
            else
                return hasSplitForm<3,0,3,0,double>() || hasSplitForm<3,0,3,0,double>() ? &launch_split64_06_06 : nullptr;
        case 700:
            if (fp32)
                return hasSplitForm<3,1,0,0,float>() || hasSplitForm<0,0,3,1,float>() ? &launch_split32_07_00 : nullptr;
            else
                return hasSplitForm<3,1,0,0,double>() || hasSplitForm<0,0,3,1,double>() ? &launch_split64_07_00 : nullptr;
        case 701:
            if (fp32)
                return hasSplitForm<3,1,1,0,float>() || hasSplitForm<1,0,3,1,float>() ? &launch_split32_07_01 : nullptr;
            else
                return hasSplitForm<3,1,1,0,double>() || hasSplitForm<1,0,3,1,double>() ? &launch_split64_07_01 : nullptr;
        case 702:
            if (fp32)
                return hasSplitForm<3,1,1,1,float>() || hasSplitForm<1,1,3,1,float>() ? &launch_split32_07_02 : nullptr;
            else
                return hasSplitForm<3,1,1,1,double>() || hasSplitForm<1,1,3,1,double>() ? &launch_split64_07_02 : nullptr;
        case 703:
            if (fp32)
                return hasSplitForm<3,1,2,0,float>() || hasSplitForm<2,0,3,1,float>() ? &launch_split32_07_03 : nullptr;
            else
                return hasSplitForm<3,1,2,0,double>() || hasSplitForm<2,0,3,1,double>() ? &launch_split64_07_03 : nullptr;
        case 800:
            if (fp32)
                return hasSplitForm<3,2,0,0,float>() || hasSplitForm<0,0,3,2,float>() ? &launch_split32_08_00 : nullptr;
            else
                return hasSplitForm<3,2,0,0,double>() || hasSplitForm<0,0,3,2,double>() ? &launch_split64_08_00 : nullptr;
        case 801:
            if (fp32)
                return hasSplitForm<3,2,1,0,float>() || hasSplitForm<1,0,3,2,float>() ? &launch_split32_08_01 : nullptr;
            else
                return hasSplitForm<3,2,1,0,double>() || hasSplitForm<1,0,3,2,double>() ? &launch_split64_08_01 : nullptr;
        case 900:
            if (fp32)
                return hasSplitForm<3,3,0,0,float>() || hasSplitForm<0,0,3,3,float>() ? &launch_split32_09_00 : nullptr;
            else
                return hasSplitForm<3,3,0,0,double>() || hasSplitForm<0,0,3,3,double>() ? &launch_split64_09_00 : nullptr;
        default:
            return nullptr;
        }
    }
    bool splitFlipped(int bt, int kt, bool fp32)
    {
        switch (100 * bt + kt)
        {
        case 0:
            if (fp32)
                return !hasSplitForm<0,0,0,0,float>();
            else
                return !hasSplitForm<0,0,0,0,double>();
        case 100:
            if (fp32)
                return !hasSplitForm<1,0,0,0,float>();
            else
                return !hasSplitForm<1,0,0,0,double>();
        case 101:
            if (fp32)
                return !hasSplitForm<1,0,1,0,float>();
            else
                return !hasSplitForm<1,0,1,0,double>();
        case 200:
            if (fp32)
                return !hasSplitForm<1,1,0,0,float>();
            else
                return !hasSplitForm<1,1,0,0,double>();
        case 201:
            if (fp32)
                return !hasSplitForm<1,1,1,0,float>();
            else
                return !hasSplitForm<1,1,1,0,double>();
        case 202:
            if (fp32)
                return !hasSplitForm<1,1,1,1,float>();
            else
                return !hasSplitForm<1,1,1,1,double>();
        case 300:
            if (fp32)
                return !hasSplitForm<2,0,0,0,float>();
            else
                return !hasSplitForm<2,0,0,0,double>();
        case 301:
            if (fp32)
                return !hasSplitForm<2,0,1,0,float>();
            else
                return !hasSplitForm<2,0,1,0,double>();
        case 302:
            if (fp32)
                return !hasSplitForm<2,0,1,1,float>();
            else
                return !hasSplitForm<2,0,1,1,double>();
        case 303:
            if (fp32)
                return !hasSplitForm<2,0,2,0,float>();
            else
                return !hasSplitForm<2,0,2,0,double>();
        case 400:
            if (fp32)
                return !hasSplitForm<2,1,0,0,float>();
            else
                return !hasSplitForm<2,1,0,0,double>();
        case 401:
            if (fp32)
                return !hasSplitForm<2,1,1,0,float>();
            else
                return !hasSplitForm<2,1,1,0,double>();
        case 402:
            if (fp32)
                return !hasSplitForm<2,1,1,1,float>();
            else
                return !hasSplitForm<2,1,1,1,double>();
        case 403:
            if (fp32)
                return !hasSplitForm<2,1,2,0,float>();
            else
                return !hasSplitForm<2,1,2,0,double>();
        case 404:
            if (fp32)
                return !hasSplitForm<2,1,2,1,float>();
            else
                return !hasSplitForm<2,1,2,1,double>();
        case 500:
            if (fp32)
                return !hasSplitForm<2,2,0,0,float>();
            else
                return !hasSplitForm<2,2,0,0,double>();
        case 501:
            if (fp32)
                return !hasSplitForm<2,2,1,0,float>();
            else
                return !hasSplitForm<2,2,1,0,double>();
        case 502:
            if (fp32)
                return !hasSplitForm<2,2,1,1,float>();
            else
                return !hasSplitForm<2,2,1,1,double>();
        case 503:
            if (fp32)
                return !hasSplitForm<2,2,2,0,float>();
            else
                return !hasSplitForm<2,2,2,0,double>();
        case 600:
            if (fp32)
                return !hasSplitForm<3,0,0,0,float>();
            else
                return !hasSplitForm<3,0,0,0,double>();
        case 601:
            if (fp32)
                return !hasSplitForm<3,0,1,0,float>();
            else
                return !hasSplitForm<3,0,1,0,double>();
        case 602:
            if (fp32)
                return !hasSplitForm<3,0,1,1,float>();
            else
                return !hasSplitForm<3,0,1,1,double>();
        case 603:
            if (fp32)
                return !hasSplitForm<3,0,2,0,float>();
            else
                return !hasSplitForm<3,0,2,0,double>();
        case 604:
            if (fp32)
                return !hasSplitForm<3,0,2,1,float>();
            else
                return !hasSplitForm<3,0,2,1,double>();
        case 606:
            if (fp32)
                return !hasSplitForm<3,0,3,0,float>();
            else
                return !hasSplitForm<3,0,3,0,double>();
        case 700:
            if (fp32)
                return !hasSplitForm<3,1,0,0,float>();
            else
                return !hasSplitForm<3,1,0,0,double>();
        case 701:
            if (fp32)
                return !hasSplitForm<3,1,1,0,float>();
            else
                return !hasSplitForm<3,1,1,0,double>();
        case 702:
            if (fp32)
                return !hasSplitForm<3,1,1,1,float>();
            else
                return !hasSplitForm<3,1,1,1,double>();
        case 703:
            if (fp32)
                return !hasSplitForm<3,1,2,0,float>();
            else
                return !hasSplitForm<3,1,2,0,double>();
        case 800:
            if (fp32)
                return !hasSplitForm<3,2,0,0,float>();
            else
                return !hasSplitForm<3,2,0,0,double>();
        case 801:
            if (fp32)
                return !hasSplitForm<3,2,1,0,float>();
            else
                return !hasSplitForm<3,2,1,0,double>();
        case 900:
            if (fp32)
                return !hasSplitForm<3,3,0,0,float>();
            else
                return !hasSplitForm<3,3,0,0,double>();
        default:
            return false;
        }
    }
    LaunchFn lookupFwd64(int bt, int kt, int shape)
    {
        if (bt < 0 || bt >= 12 || kt < 0 || kt > bt)
            return nullptr;
        return shape == 2 ? k_fwd64f[bt][kt] : shape ? k_fwd64v[bt][kt] : k_fwd64[bt][kt];
    }
    LaunchFn lookupFwd32(int bt, int kt, int shape)
    {
        if (bt < 0 || bt >= 10 || kt < 0 || kt > bt)
            return nullptr;
        return shape == 2 ? k_fwd32f[bt][kt] : shape ? k_fwd32v[bt][kt] : k_fwd32[bt][kt];
    }
    LaunchFn lookupD1(int bt, int kt)
    {
        if (bt < 0 || bt >= 12 || kt < 0 || kt > bt)
            return nullptr;
        return k_d1[bt][kt];
    }
    int unitFwd(int bt, int kt, bool fp32, int shape)
    {
        if (bt < 0 || kt < 0 || kt > bt || bt >= (fp32 ? 10 : 12))
            return 0;
        if (shape == 2)
            return fp32 ? u_fwd32_2[bt][kt] : u_fwd64_2[bt][kt];
        if (shape)
            return fp32 ? u_fwd32_1[bt][kt] : u_fwd64_1[bt][kt];
        return fp32 ? u_fwd32_0[bt][kt] : u_fwd64_0[bt][kt];
    }
    bool hasFwdVariant(int bt, int kt, bool fp32, int shape)
    {
        return (fp32 ? lookupFwd32(bt, kt, shape) : lookupFwd64(bt, kt, shape)) != nullptr;
    }
}
