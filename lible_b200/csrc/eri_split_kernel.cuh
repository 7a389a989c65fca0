// Split form of the register path for heavily contracted quartets: one warp per quartet, its thread
// groups sharing the quartet's primitive pairs.
//
// The register path evaluates a quartet's K_ab K_cd primitive pairs one after another in one thread
// group.  Two contracted core pairs have 64 x 64 of them, a serial chain of about 1.6 ms for (ss|ss)
// that no launch containing such a quartet can beat, however idle the device is.  Dealing the pairs
// out to the slots of a warp cuts the chain by up to 32; the price is one reduction and a digestion
// of a single quartet per warp, a few hundred instructions, which the plans accept for quartets
// that are heavy against the launch's even share (splitRuns in engine.cu).
// Bound by the latency of its longest quartet: (ss|ss) of (H2O)_16 cc-pVDZ takes 56 us, 128 primitive pairs a
// lane, with the FP64 pipe 16% active (2.64 -> 1.56 ms for the class with its ordinary launch).
#pragma once

#include "eri_kernel.cuh"

namespace lible_b200
{
    // Classes with a split form: register-path classes of total angular momentum up to 6 (above that no
    // basis in use has contractions long enough to matter).
    template <int LA, int LB, int LC, int LD, typename T>
    constexpr bool hasSplitForm()
    {
        return LA + LB + LC + LD <= 6 && Shape<LA, LB, LC, LD, T, 0>::GT > 0;
    }

    // Per-warp staging: a partial batch per slot, or (whole quartets per thread) the reduced batch.
    template <int LA, int LB, int LC, int LD, typename T>
    struct SplitShape
    {
        using C = Cls<LA, LB, LC, LD>;
        using S = Shape<LA, LB, LC, LD, T, 0>;
        static constexpr int GT = S::GT, QPW = S::QPW, slots = GT > 1 ? QPW : 1, blk = C::SAB * C::SCD;
        static constexpr int warps = 4;
        static constexpr size_t off_boys = (sizeof(double) * warps * slots * blk + 15) / 16 * 16;
        static constexpr size_t smem = off_boys + S::boys_bytes;
    };

    // J/K and (FP64) store epilogues as the class kernels; tasks from the chunk queue, or one per warp
    // without one.
    template <int LA, int LB, int LC, int LD, typename T>
    __global__ void __launch_bounds__(128) eriSplitKernel(QuartetArgs a)
    {
        using C = Cls<LA, LB, LC, LD>;
        using SS = SplitShape<LA, LB, LC, LD, T>;
        using S = typename SS::S;
        constexpr int GT = SS::GT, QPW = SS::QPW, CW = S::CW, blk = SS::blk;
        extern __shared__ __align__(16) unsigned char smem[];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot = lane / GT, member = lane % GT;
        double *vw = reinterpret_cast<double *>(smem) + (size_t)warp * SS::slots * blk;
        T *btab = reinterpret_cast<T *>(smem + SS::off_boys);
        if constexpr (sizeof(T) == 8)
            stageBoys(a.boys, C::L, reinterpret_cast<double *>(btab));
        else
            stageBoys(a.boys_f, C::L, reinterpret_cast<float *>(btab));
        __syncthreads();
        int cur = 0;
        auto run = [&](long long t) {
            uint32_t ib, ik, pos;
            decodeCursor(a, t, cur, ib, ik, pos);
            if (!inWindow(a, ib, ik, pos, true))
                return;
            T V[C::SAB * CW];
            // records of the pair itself: the lanes of a warp read different primitives of one pair
            quartetThread<LA, LB, LC, LD, T, 0, true>(a, ib, ik, member * CW, V, btab, make_uint4(0, 0, 0, 0), -1,
                                                      (uint32_t)slot, (uint32_t)QPW);
            // the parts summed in double into the warp's first staged batch
            if constexpr (GT == 1)
            {
#pragma unroll
                for (int e = 0; e < blk; e++)
                {
                    double v = (double)V[e];
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1)
                        v += __shfl_xor_sync(0xffffffffu, v, off);
                    if ((e & 31) == lane)
                        vw[e] = v;
                }
            }
            else
            {
                if (slot < QPW)
                {
#pragma unroll
                    for (int m = 0; m < C::SAB; m++)
#pragma unroll
                        for (int c = 0; c < CW; c++)
                            vw[slot * blk + m * C::SCD + member * CW + c] = (double)V[m * CW + c];
                }
                __syncwarp();
                for (int e = lane; e < blk; e += 32)
                {
                    double v = vw[e];
                    for (int k = 1; k < QPW; k++)
                        v += vw[k * blk + e];
                    vw[e] = v;
                }
            }
            __syncwarp();
            const int32_t *bi = a.bra.info + 8 * ib;
            const int32_t *ki = a.ket.info + 8 * ik;
            auto val = [&](int e) { return vw[e]; };
            bool store = false;
            if constexpr (sizeof(T) == 8)
                store = a.mode == kStore;
            if (store)
                for (int e = lane; e < blk; e += 32)
                {
                    const int m = e / C::SCD, kt = e % C::SCD;
                    a.out[(size_t)t * blk + storeIndex<C::SA, C::SB, C::SC, C::SD>(a.flags, m / C::SB, m % C::SB,
                                                                                   kt / C::SD, kt % C::SD)] = vw[e];
                }
            else
                digestJK<C::SA, C::SB, C::SC, C::SD, false>(a, quartetWeight(a, ib, ik), braFields(bi), ki, val, lane, 32);
            __syncwarp();
        };
        if (a.chunks)
        {
            for (;;)
            {
                unsigned long long c = 0;
                if (lane == 0)
                    c = atomicAdd(a.counter, 1ULL);
                c = __shfl_sync(0xffffffffu, c, 0);
                if (c >= (unsigned long long)a.n_chunks)
                    break;
                const long long t1 = (long long)__ldg(a.chunks + c + 1);
                for (long long t = (long long)__ldg(a.chunks + c); t < t1; t++)
                    run(t);
            }
        }
        else
            for (long long t = (long long)blockIdx.x * SS::warps + warp; t < a.n_tasks; t += (long long)gridDim.x * SS::warps)
                run(t);
    }

    // Launches the split form; with a work queue a persistent grid, else one warp per task.
    template <int LA, int LB, int LC, int LD, typename T>
    cudaError_t launchSplit(const QuartetArgs &a, cudaStream_t s, int num_sms)
    {
        if constexpr (!hasSplitForm<LA, LB, LC, LD, T>())
            return cudaErrorNotSupported;
        else
        {
            using SS = SplitShape<LA, LB, LC, LD, T>;
            const long long units = a.chunks ? a.n_chunks : a.n_tasks;
            if (units <= 0)
                return cudaSuccess;
            auto kern = eriSplitKernel<LA, LB, LC, LD, T>;
            if (SS::smem > 48 * 1024)
            {
                const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS::smem);
                if (e != cudaSuccess)
                    return e;
            }
            const long long grid = std::min<long long>((units + SS::warps - 1) / SS::warps, (long long)num_sms * 8);
            kern<<<(unsigned)grid, 32 * SS::warps, SS::smem, s>>>(a);
            return cudaGetLastError();
        }
    }
}
