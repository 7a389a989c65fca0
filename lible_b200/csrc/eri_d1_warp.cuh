// Warp form of the J/K and RI-J gradient contraction (kD1Grad, kD1GradRI): one warp per quartet, its
// lanes owning the bra Hermite functions h.  It serves the classes with a large bra and a thin ket
// (d1WarpClass), whose work per quartet is too small for a block with its barriers and too wide for the
// registers of single threads.
//
// With Gamma the density block of the quartet, per bra primitive a lane forms its rows of
//     GE = Gamma^T E_ab,   GE1_x = Gamma^T E1_ab,x        ([H_ab] x [S_cd], K = S_ab)
// from coalesced loads of E (consecutive lanes read consecutive h), and per primitive quartet, for its h
// and every h' of the ket,
//     w0 = GE E_cd^T,  w1_x = GE1_x E_cd^T,  w2_x = GE E1_cd,x^T     (K = S_cd, in registers)
//     t1_x += w0 s R[h + h' + e_x],  t13_x += w1_x s R[h + h'],  tc_x += w2_x s R[h + h'] - (c/q) w0 s R[h + h' + e_x]
// with s = (-1)^{|h'|}, as the register and tensor-pipe forms do.  R (to order L + 1) is built by the
// warp in its own shared memory (warpHermiteR), so nothing synchronises more than one warp, the ket's E
// and E1 are staged there with the four values of an element side by side, and the nine sums are
// reduced once per quartet.
// Bound by L1/TEX wavefronts (four R values and an index per Hermite pair, the ket tile): 71% of the unit on
// (dp|ps) and (fd|ps) of (H2O)_4 cc-pVTZ, at 12 warps an SM of 164-168 registers, the FP64 pipe 32% active.
#pragma once

#include "eri_d1_kernel.cuh"

namespace lible_b200
{
    template <int LA, int LB, int LC, int LD>
    struct ShapeD1W
    {
        using C = Cls<LA, LB, LC, LD>;
        static constexpr int ROWS = (C::HAB + 31) / 32, WARPS = 4;
        static constexpr size_t a16(size_t x) { return (x + 15) / 16 * 16; }
        static constexpr size_t off_boys = 0;
        static constexpr size_t off_ix = a16(8 * kBoysTerms * kBoysPitch);                  // HCD x HAB packed R indices
        static constexpr size_t off_rule = a16(off_ix + 4 * (size_t)C::HCD * C::HAB);       // R rules, NR1
        static constexpr size_t off_coef = a16(off_rule + 4 * (size_t)C::NR1);
        static constexpr size_t off_w = a16(off_coef + 8 * (size_t)C::NR1);
        // per warp: the ket tile [h'][c][4], Gamma, 2 x NR1, X Y Z (an even number of doubles)
        static constexpr size_t warp_doubles = (4 * C::HCD * C::SCD + C::SAB * C::SCD + 2 * C::NR1 + 3 + 1) / 2 * 2;
        static constexpr size_t off_sg = off_w + 8 * WARPS * warp_doubles;                  // the block's gradient
        static constexpr size_t smem = off_sg;
    };
    constexpr int kD1WarpSharedAtoms = 512;  // the block's gradient is summed in shared memory up to this many atoms

    template <int LA, int LB, int LC, int LD>
    __global__ void __launch_bounds__(128) eriD1WarpKernel(QuartetArgs a)
    {
        using C = Cls<LA, LB, LC, LD>;
        using S = ShapeD1W<LA, LB, LC, LD>;
        constexpr int L1 = C::L + 1, ROWS = S::ROWS;
        extern __shared__ __align__(16) unsigned char smem[];
        double *btab = reinterpret_cast<double *>(smem + S::off_boys);
        uint32_t *ixt = reinterpret_cast<uint32_t *>(smem + S::off_ix);
        uint32_t *rule = reinterpret_cast<uint32_t *>(smem + S::off_rule);
        double *coef = reinterpret_cast<double *>(smem + S::off_coef);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        double *ket = reinterpret_cast<double *>(smem + S::off_w) + warp * S::warp_doubles;
        double *G = ket + 4 * C::HCD * C::SCD, *rbuf = G + C::SAB * C::SCD, *xyz = rbuf + 2 * C::NR1;
        double *sg = reinterpret_cast<double *>(smem + S::off_sg);
        const bool shared_grad = a.n_atoms <= kD1WarpSharedAtoms;
        stageBoys(a.boys, L1, btab);
        buildWarpRules(C::NR1, rule, coef);
        // R indices of h + h' (bits 0-9), h + h' + e_x (10-19) and h + h' + e_y (20-29; e_z is the next one)
        for (int e = threadIdx.x; e < C::HCD * C::HAB; e += 128)
        {
            int t, u, v, tp, up, vp;
            hermTuv(e % C::HAB, t, u, v);
            hermTuv(e / C::HAB, tp, up, vp);
            t += tp;
            u += up;
            v += vp;
            ixt[e] = (uint32_t)hermIndex(t, u, v) | (uint32_t)hermIndex(t + 1, u, v) << 10 |
                     (uint32_t)hermIndex(t, u + 1, v) << 20;
        }
        if (shared_grad)
            for (int e = threadIdx.x; e < 3 * a.n_atoms; e += 128)
                sg[e] = 0.0;
        __syncthreads();
        const size_t n = (size_t)a.nao;
        const double *D = a.D;
        double *const grad = shared_grad ? sg : a.grad;
        int cur = 0;
        auto run = [&](long long task) {
            uint32_t ib, ik;
            decodeCursor(a, task, cur, ib, ik);
            if (!inWindow(a, ib, ik, 0, false))
                return;
            const int32_t *bi = a.bra.info + 8 * ib;
            const int32_t *ki = a.ket.info + 8 * ik;
            __syncwarp();  // every lane is done with the previous quartet's Gamma
            if (a.mode == kD1GradRI)
            {
                const int32_t *mi = a.aux_side == 0 ? bi : ki;
                const double w = a.aux_side == 2 ? -((a.same_class && ib == ik) ? 0.5 : 1.0) : (mi[4] == mi[5] ? 1.0 : 2.0);
                for (int e = lane; e < C::SAB * C::SCD; e += 32)
                {
                    const int m = e / C::SCD, c = e % C::SCD;
                    double v;
                    if (a.aux_side == 2)
                        v = __ldg(a.dcoef + bi[0] + m) * __ldg(a.dcoef + ki[0] + c);
                    else if (a.aux_side == 0)
                        v = __ldg(D + (size_t)(bi[0] + m / C::SB) * n + bi[1] + m % C::SB) * __ldg(a.dcoef + ki[0] + c);
                    else
                        v = __ldg(D + (size_t)(ki[0] + c / C::SD) * n + ki[1] + c % C::SD) * __ldg(a.dcoef + bi[0] + m);
                    G[e] = w * v;
                }
            }
            else
            {
                const double f = quartetWeight(a, ib, ik);
                for (int e = lane; e < C::SAB * C::SCD; e += 32)
                {
                    const int m = e / C::SCD, c = e % C::SCD;
                    const size_t mu = bi[0] + m / C::SB, nu = bi[1] + m % C::SB;
                    const size_t ka = ki[0] + c / C::SD, ta = ki[1] + c % C::SD;
                    G[e] = f * (4.0 * __ldg(D + mu * n + nu) * __ldg(D + ka * n + ta) -
                                __ldg(D + mu * n + ka) * __ldg(D + nu * n + ta) -
                                __ldg(D + mu * n + ta) * __ldg(D + nu * n + ka));
                }
            }
            __syncwarp();
            double g[9];
#pragma unroll
            for (int x = 0; x < 9; x++)
                g[x] = 0.0;
            const uint32_t p0 = a.bra.pofs[ib], p1 = a.bra.pofs[ib + 1];
            const uint32_t q0 = a.ket.pofs[ik], q1 = a.ket.pofs[ik + 1];
            for (uint32_t p = p0; p < p1; p++)
            {
                const PQ4 P = loadPQ(a.bra.pP, p);
                const double2 AB = __ldg(reinterpret_cast<const double2 *>(a.bra.ab) + p);
                const double *eab = a.bra.E + (size_t)p * C::SAB * C::HAB;
                const double *e1ab = a.bra.E1 + (size_t)p * 3 * C::SAB * C::HAB;
                // this lane's rows of GE (x = 0) and GE1 (x = 1..3); rows past H_ab stay zero
                double ge[ROWS][4][C::SCD];
#pragma unroll
                for (int r = 0; r < ROWS; r++)
                {
#pragma unroll
                    for (int x = 0; x < 4; x++)
#pragma unroll
                        for (int c = 0; c < C::SCD; c++)
                            ge[r][x][c] = 0.0;
                    const int h = lane + 32 * r;
                    if (h < C::HAB)
                    {
#pragma unroll 5
                        for (int m = 0; m < C::SAB; m++)
                        {
                            const double e0 = __ldg(eab + m * C::HAB + h);
                            const double e1 = __ldg(e1ab + (0 * C::SAB + m) * C::HAB + h);
                            const double e2 = __ldg(e1ab + (1 * C::SAB + m) * C::HAB + h);
                            const double e3 = __ldg(e1ab + (2 * C::SAB + m) * C::HAB + h);
#pragma unroll
                            for (int c = 0; c < C::SCD; c++)
                            {
                                const double gm = G[m * C::SCD + c];
                                ge[r][0][c] += gm * e0;
                                ge[r][1][c] += gm * e1;
                                ge[r][2][c] += gm * e2;
                                ge[r][3][c] += gm * e3;
                            }
                        }
                    }
                }
                double t1[3] = {0, 0, 0}, t13[3] = {0, 0, 0}, tc[3] = {0, 0, 0};
                for (uint32_t q = q0; q < q1; q++)
                {
                    const PQ4 Q = loadPQ(a.ket.pP, q);
                    const double cq = __ldg(a.ket.ab + 2 * q) * Q.ip;
                    const double rs = rsqrt(P.x + Q.x);
                    const double alpha = P.x * Q.x * (rs * rs);
                    const double X = P.y - Q.y, Y = P.z - Q.z, Z = P.w - Q.w;
                    const double fac = 34.986836655249725 * rs * P.ip * Q.ip;
                    double F[L1 + 1];
                    boysF<L1, true>(alpha * (X * X + Y * Y + Z * Z), btab, F);
                    // the ket tile, by the R build's barriers (its first one ends the reads of the last tile)
                    const double *ecd = a.ket.Et + (size_t)q * C::HCD * C::SCD;
                    const double *e1cd = a.ket.E1t + (size_t)q * 3 * C::HCD * C::SCD;
                    __syncwarp();
                    for (int e = lane; e < C::HCD * C::SCD; e += 32)
                    {
                        cpAsync8(ket + 4 * e, ecd + e);
                        cpAsync8(ket + 4 * e + 1, e1cd + e);
                        cpAsync8(ket + 4 * e + 2, e1cd + C::HCD * C::SCD + e);
                        cpAsync8(ket + 4 * e + 3, e1cd + 2 * C::HCD * C::SCD + e);
                    }
                    const double *R = warpHermiteR<L1>(F, fac, -2.0 * alpha, X, Y, Z, rbuf, xyz, rule, coef, lane);
                    cpAsyncWaitAll();
                    __syncwarp();
                    // ux, uy, uz: sums of w0 s R[h + h' + e]; t13 and the E1 part of tc directly
                    double ux = 0.0, uy = 0.0, uz = 0.0;
                    // Hermite functions of the ket in order of |h'|, so the sign is known per order
#pragma unroll
                    for (int np = 0; np <= C::LCD; np++)
                    {
                        const double sgn = (np & 1) ? -1.0 : 1.0;
#pragma unroll 1
                        for (int hp = nherm(np - 1); hp < nherm(np); hp++)
                        {
                            double e0[C::SCD], ex[C::SCD], ey[C::SCD], ez[C::SCD];
#pragma unroll
                            for (int c = 0; c < C::SCD; c++)
                            {
                                const double2 *k2 = reinterpret_cast<const double2 *>(ket + 4 * (hp * C::SCD + c));
                                const double2 ka = k2[0], kb = k2[1];
                                e0[c] = ka.x;
                                ex[c] = ka.y;
                                ey[c] = kb.x;
                                ez[c] = kb.y;
                            }
#pragma unroll
                            for (int r = 0; r < ROWS; r++)
                            {
                                const int h = lane + 32 * r < C::HAB ? lane + 32 * r : 0;
                                const uint32_t ix = ixt[hp * C::HAB + h];
                                const double r0 = sgn * R[ix & 1023], rx = sgn * R[(ix >> 10) & 1023];
                                const double ry = sgn * R[ix >> 20], rz = sgn * R[(ix >> 20) + 1];
                                double w0 = 0, w1x = 0, w1y = 0, w1z = 0, w2x = 0, w2y = 0, w2z = 0;
#pragma unroll
                                for (int c = 0; c < C::SCD; c++)
                                {
                                    w0 += ge[r][0][c] * e0[c];
                                    w1x += ge[r][1][c] * e0[c];
                                    w1y += ge[r][2][c] * e0[c];
                                    w1z += ge[r][3][c] * e0[c];
                                    w2x += ge[r][0][c] * ex[c];
                                    w2y += ge[r][0][c] * ey[c];
                                    w2z += ge[r][0][c] * ez[c];
                                }
                                ux += w0 * rx;
                                uy += w0 * ry;
                                uz += w0 * rz;
                                t13[0] += w1x * r0;
                                t13[1] += w1y * r0;
                                t13[2] += w1z * r0;
                                tc[0] += w2x * r0;
                                tc[1] += w2y * r0;
                                tc[2] += w2z * r0;
                            }
                        }
                    }
                    t1[0] += ux;
                    t1[1] += uy;
                    t1[2] += uz;
                    tc[0] -= cq * ux;
                    tc[1] -= cq * uy;
                    tc[2] -= cq * uz;
                }
                const double ap = AB.x * P.ip, bp = AB.y * P.ip;
#pragma unroll
                for (int x = 0; x < 3; x++)
                {
                    g[x] += ap * t1[x] + t13[x];
                    g[3 + x] += bp * t1[x] - t13[x];
                    g[6 + x] += tc[x];
                }
            }
            // the warp's sums; lane 3 k + x adds component x of centre k (D by translational invariance)
            double mine = 0.0;
#pragma unroll
            for (int x = 0; x < 9; x++)
            {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    g[x] += __shfl_xor_sync(0xffffffffu, g[x], o);
                if (lane == x)
                    mine = g[x];
            }
#pragma unroll
            for (int x = 0; x < 3; x++)
                if (lane == 9 + x)
                    mine = -(g[x] + g[3 + x] + g[6 + x]);
            if (lane < 12)
            {
                const int k = lane / 3;
                const int atom = k == 0 ? bi[2] : k == 1 ? bi[3] : k == 2 ? ki[2] : ki[3];
                atomicAdd(grad + 3 * atom + lane % 3, mine);
            }
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
        if (shared_grad)
        {
            __syncthreads();
            for (int e = threadIdx.x; e < 3 * a.n_atoms; e += 128)
                if (sg[e] != 0.0)
                    atomicAdd(a.grad + e, sg[e]);
        }
    }

    template <int LA, int LB, int LC, int LD>
    cudaError_t launchD1Warp(const QuartetArgs &a, cudaStream_t s, int num_sms)
    {
        using S = ShapeD1W<LA, LB, LC, LD>;
        auto kern = eriD1WarpKernel<LA, LB, LC, LD>;
        const size_t smem = S::smem + (a.n_atoms <= kD1WarpSharedAtoms ? sizeof(double) * 3 * (size_t)a.n_atoms : 0);
        if (smem > 48 * 1024)
        {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess)
                return e;
        }
        int occ = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 128, smem);
        if (e != cudaSuccess)
            return e;
        const long long units = a.chunks ? a.n_chunks : a.n_tasks;
        const long long grid = std::max<long long>(
            1, std::min<long long>((units + S::WARPS - 1) / S::WARPS, (long long)num_sms * std::max(occ, 1)));
        kern<<<(unsigned)grid, 128, smem, s>>>(a);
        return cudaGetLastError();
    }
}
