// Warp form of the FP64 class kernels: one warp per quartet, its lanes owning the bra Hermite functions h in
// the first contraction and the bra functions m in the second.  It serves the classes with a large bra
// and a thin ket (warpClass).  The block form has too little work per quartet for its barriers there and
// pads its 8 x 8 tensor tiles, and the register form rebuilds R in each of its S_cd threads.
//
//   RE[h][c] = sum_{h'} s(h') R[h + h'] E_cd[h'][c]       lane h, R built by the warp (warpHermiteR)
//   V[m][c] += sum_h E_ab[m][h] RE[h][c]                  lane m, RE through the warp's shared memory
//
// E_ab is read transposed, so that consecutive lanes read consecutive m; the ket tile and RE are
// broadcast from shared memory.  Nothing synchronises more than one warp.
// Bound by L1/TEX wavefronts (R and its index table from shared memory, rows of E_ab): 74-77% of the unit on
// (dd|ps) and (fd|ps) of (H2O)_4 cc-pVTZ, at 15 warps an SM of 120-126 registers, the FP64 pipe 21% active.
#pragma once

#include "eri_kernel.cuh"

namespace lible_b200
{
    // Bras of at least 35 Hermite functions (dd, fp, fd, ff; aux g, h shells), kets of 3 to 9 functions, and
    // of one function with at least 84.  Measured on the (H2O)_8 cc-pVTZ J/K build against the register or
    // block kernel that served the class: (fd|ps) 7.24 -> 2.10 ms, (dd|pp) 4.83 -> 1.67, (fd|ds) 4.35 -> 1.37,
    // (dd|ps) 5.04 -> 3.26, (dd|ds) 4.13 -> 2.18, (fp|pp) 3.46 -> 1.67, (ff|ss) 1.73 -> 0.30; one function
    // is too thin for the smaller bras ((dd|ss) 1.40 -> 2.10 ms, (fp|ss) 2.18 -> 2.14).  Of the classes with
    // an auxiliary shell, the RI contractions of (H2O)_12 cc-pVTZ with def2-qzvp-rifit: (hs|ps) 1.64 -> 0.49 ms,
    // (hs|ds) 0.87 -> 0.34, (hs|pp) 0.84 -> 0.26, (gs|fs) 1.34 -> 0.46, (fd|fs) 1.12 -> 0.37, (ff|ss) 0.36 -> 0.11,
    // (gs|pp) 0.95 -> 0.89; (gs|ps) and (gs|ds) only while short (warpWhileShort).
    constexpr bool warpClass(int la, int lb, int lc, int ld)
    {
        const int scd = nsph(lc) * nsph(ld);
        return nherm(la + lb) >= (scd == 1 ? 84 : 35) && scd <= 9;
    }

    template <int LA, int LB, int LC, int LD>
    struct ShapeW
    {
        using C = Cls<LA, LB, LC, LD>;
        static constexpr int WARPS = 4;
        static constexpr int ROWS = (C::HAB + 31) / 32, MROWS = (C::SAB + 31) / 32;
        static constexpr int PC = (C::SCD + 1) / 2 * 2;  // row pitch of the ket tile and of RE (16-byte reads)
        static constexpr size_t a16(size_t x) { return (x + 15) / 16 * 16; }
        static constexpr size_t off_boys = 0;
        static constexpr size_t off_ix = a16(8 * kBoysTerms * kBoysPitch);                 // HCD x HAB R indices
        static constexpr size_t off_rule = a16(off_ix + 2 * (size_t)C::HCD * C::HAB);      // R rules, NR
        static constexpr size_t off_coef = a16(off_rule + 4 * (size_t)C::NR);
        static constexpr size_t off_w = a16(off_coef + 8 * (size_t)C::NR);
        // per warp: the ket tile [h'][PC], RE [h][PC] (later the batch [m][c]), 2 x NR, X Y Z
        static constexpr size_t warp_doubles = ((C::HCD + C::HAB) * PC + 2 * C::NR + 3 + 1) / 2 * 2;
        static constexpr size_t smem = off_w + 8 * WARPS * warp_doubles;
        static_assert(C::SAB * C::SCD <= C::HAB * PC, "the batch fits RE's space");
    };

    template <int LA, int LB, int LC, int LD>
    __global__ void __launch_bounds__(128, 4) eriWarpKernel(QuartetArgs a)
    {
        using C = Cls<LA, LB, LC, LD>;
        using S = ShapeW<LA, LB, LC, LD>;
        constexpr int ROWS = S::ROWS, MROWS = S::MROWS, PC = S::PC, SCD = C::SCD, SAB = C::SAB, blk = SAB * SCD;
        extern __shared__ __align__(16) unsigned char smem[];
        double *btab = reinterpret_cast<double *>(smem + S::off_boys);
        uint16_t *ixt = reinterpret_cast<uint16_t *>(smem + S::off_ix);
        uint32_t *rule = reinterpret_cast<uint32_t *>(smem + S::off_rule);
        double *coef = reinterpret_cast<double *>(smem + S::off_coef);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        double *ket = reinterpret_cast<double *>(smem + S::off_w) + warp * S::warp_doubles;
        double *re = ket + C::HCD * PC, *rbuf = re + C::HAB * PC, *xyz = rbuf + 2 * C::NR;
        stageBoys(a.boys, C::L, btab);
        buildWarpRules(C::NR, rule, coef);
        for (int e = threadIdx.x; e < C::HCD * C::HAB; e += 128)
        {
            int t, u, v, tp, up, vp;
            hermTuv(e % C::HAB, t, u, v);
            hermTuv(e / C::HAB, tp, up, vp);
            ixt[e] = (uint16_t)hermIndex(t + tp, u + up, v + vp);
        }
        __syncthreads();
        int cur = 0;
        auto run = [&](long long task) {
            uint32_t ib, ik, pos;
            decodeCursor(a, task, cur, ib, ik, pos);
            if (!inWindow(a, ib, ik, pos, true))
                return;
            double v[MROWS][SCD];
#pragma unroll
            for (int r = 0; r < MROWS; r++)
#pragma unroll
                for (int c = 0; c < SCD; c++)
                    v[r][c] = 0.0;
            const uint32_t p0 = a.bra.pofs[ib], p1 = a.bra.pofs[ib + 1];
            const uint32_t q0 = a.ket.pofs[ik], q1 = a.ket.pofs[ik + 1];
            for (uint32_t p = p0; p < p1; p++)
            {
                const PQ4 P = loadPQ(a.bra.pP, p);
                double rx[ROWS][SCD];
#pragma unroll
                for (int r = 0; r < ROWS; r++)
#pragma unroll
                    for (int c = 0; c < SCD; c++)
                        rx[r][c] = 0.0;
                for (uint32_t q = q0; q < q1; q++)
                {
                    __syncwarp();  // the last tile has been read
                    const double *ecd = a.ket.Et + (size_t)q * C::HCD * SCD;
                    for (int e = lane; e < C::HCD * SCD; e += 32)
                        cpAsync8(ket + e / SCD * PC + e % SCD, ecd + e);
                    const PQ4 Q = loadPQ(a.ket.pP, q);
                    const double rs = rsqrt(P.x + Q.x);
                    const double alpha = P.x * Q.x * (rs * rs);
                    const double X = P.y - Q.y, Y = P.z - Q.z, Z = P.w - Q.w;
                    const double fac = 34.986836655249725 * rs * P.ip * Q.ip;
                    double F[C::L + 1];
                    boysF<C::L, true>(alpha * (X * X + Y * Y + Z * Z), btab, F);
                    const double *R = warpHermiteR<C::L>(F, fac, -2.0 * alpha, X, Y, Z, rbuf, xyz, rule, coef, lane);
                    cpAsyncWaitAll();
                    __syncwarp();
#pragma unroll
                    for (int np = 0; np <= C::LCD; np++)
                    {
#pragma unroll 2
                        for (int hp = nherm(np - 1); hp < nherm(np); hp++)
                        {
                            double e0[PC];
#pragma unroll
                            for (int c = 0; c < PC; c += 2)
                            {
                                const double2 k2 = *reinterpret_cast<const double2 *>(ket + hp * PC + c);
                                e0[c] = k2.x;
                                e0[c + 1] = k2.y;
                            }
#pragma unroll
                            for (int r = 0; r < ROWS; r++)
                            {
                                const int h = lane + 32 * r < C::HAB ? lane + 32 * r : 0;
                                const double r0 = (np & 1) ? -R[ixt[hp * C::HAB + h]] : R[ixt[hp * C::HAB + h]];
#pragma unroll
                                for (int c = 0; c < SCD; c++)
                                    rx[r][c] += r0 * e0[c];
                            }
                        }
                    }
                }
                // (RE's last readers, the previous primitive's second contraction or the previous quartet's
                // digestion, are behind the barriers of the R build)
#pragma unroll
                for (int r = 0; r < ROWS; r++)
                    if (lane + 32 * r < C::HAB)
                    {
#pragma unroll
                        for (int c = 0; c < SCD; c++)
                            re[(lane + 32 * r) * PC + c] = rx[r][c];
                    }
                __syncwarp();
                const double *et = a.bra.Et + (size_t)p * C::HAB * SAB;
#pragma unroll 5
                for (int h = 0; h < C::HAB; h++)
                {
                    double e0[PC];
#pragma unroll
                    for (int c = 0; c < PC; c += 2)
                    {
                        const double2 k2 = *reinterpret_cast<const double2 *>(re + h * PC + c);
                        e0[c] = k2.x;
                        e0[c + 1] = k2.y;
                    }
#pragma unroll
                    for (int r = 0; r < MROWS; r++)
                    {
                        const double e = __ldg(et + h * SAB + (lane + 32 * r < SAB ? lane + 32 * r : 0));
#pragma unroll
                        for (int c = 0; c < SCD; c++)
                            v[r][c] += e * e0[c];
                    }
                }
            }
            const int32_t *bi = a.bra.info + 8 * ib;
            const int32_t *ki = a.ket.info + 8 * ik;
            if (a.mode == kStore)
            {
#pragma unroll
                for (int r = 0; r < MROWS; r++)
                {
                    const int m = lane + 32 * r;
                    if (m < SAB)
                    {
#pragma unroll
                        for (int c = 0; c < SCD; c++)
                            a.out[(size_t)task * blk + storeIndex<C::SA, C::SB, C::SC, C::SD>(
                                                           a.flags, m / C::SB, m % C::SB, c / C::SD, c % C::SD)] = v[r][c];
                    }
                }
                return;
            }
            // the batch [m][c] over RE (every lane is done with the last second contraction)
            __syncwarp();
#pragma unroll
            for (int r = 0; r < MROWS; r++)
                if (lane + 32 * r < SAB)
                {
#pragma unroll
                    for (int c = 0; c < SCD; c++)
                        re[(lane + 32 * r) * SCD + c] = v[r][c];
                }
            __syncwarp();
            auto val = [&](int e) { return re[e]; };
            if (a.mode == kJK)
            {
                const double f = quartetWeight(a, ib, ik);
                const BraFields bf = braFields(bi);
                // J from the registers: J_ab[m] in lane m, J_cd[c] by a sum over the warp
                const size_t n = (size_t)bf.n;
                const double *D = a.D + bf.base;
                double *Jm = a.J + bf.base;
                double jc[SCD], dcd[SCD];
#pragma unroll
                for (int c = 0; c < SCD; c++)
                {
                    jc[c] = 0.0;
                    dcd[c] = __ldg(D + (size_t)(ki[0] + c / C::SD) * n + ki[1] + c % C::SD);
                }
#pragma unroll
                for (int r = 0; r < MROWS; r++)
                {
                    const int m = lane + 32 * r;
                    if (m < SAB)
                    {
                        const size_t at = (size_t)(bf.oa + m / C::SB) * n + bf.ob + m % C::SB;
                        const double dab = __ldg(D + at);
                        double s = 0.0;
#pragma unroll
                        for (int c = 0; c < SCD; c++)
                        {
                            s += v[r][c] * dcd[c];
                            jc[c] += v[r][c] * dab;
                        }
                        atomicAdd(Jm + at, 2.0 * f * s);
                    }
                }
                double mine = 0.0;
#pragma unroll
                for (int c = 0; c < SCD; c++)
                {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
                        jc[c] += __shfl_xor_sync(0xffffffffu, jc[c], o);
                    if (lane == c)
                        mine = jc[c];
                }
                if (lane < SCD)
                    atomicAdd(Jm + (size_t)(ki[0] + lane / C::SD) * n + ki[1] + lane % C::SD, 2.0 * f * mine);
                // K: the outputs past J_ab and J_cd
                digestJK<C::SA, C::SB, C::SC, C::SD, false>(a, f, bf, ki, val, SAB + SCD + lane, 32);
            }
            else
                digestRI<C::SA, C::SB, C::SC, C::SD, false>(a, bi, ki, val, lane, 32);
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
            for (long long t = (long long)blockIdx.x * S::WARPS + warp; t < a.n_tasks; t += (long long)gridDim.x * S::WARPS)
                run(t);
    }

    // Launches the warp form: a persistent grid over the work queue, or one warp per listed task.
    template <int LA, int LB, int LC, int LD>
    cudaError_t launchWarp(const QuartetArgs &a, cudaStream_t s, int num_sms)
    {
        using S = ShapeW<LA, LB, LC, LD>;
        auto kern = eriWarpKernel<LA, LB, LC, LD>;
        if (S::smem > 48 * 1024)
        {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem);
            if (e != cudaSuccess)
                return e;
        }
        int occ = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * S::WARPS, S::smem);
        if (e != cudaSuccess)
            return e;
        const long long units = a.chunks ? a.n_chunks : a.n_tasks;
        const int per_sm = a.chunks ? std::max(occ / std::max(a.grid_div, 1), 1) : 8 * std::max(occ, 1);
        const long long grid =
            std::max<long long>(1, std::min<long long>((units + S::WARPS - 1) / S::WARPS, (long long)num_sms * per_sm));
        kern<<<(unsigned)grid, 32 * S::WARPS, S::smem, s>>>(a);
        return cudaGetLastError();
    }
}
