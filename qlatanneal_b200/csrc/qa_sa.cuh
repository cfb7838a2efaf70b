// qa_sa.cuh -- SA Metropolis of dense models (annealer.cpp:50-67: spins in fixed
// order, running energy, best copied on every new minimum), one CTA of up to
// four warps per read.
//
// Same run as sa_kernel<K_DENSE>, bit for bit.  A read is one
// chain, and a warp alone on its SM issues an instruction about every four
// cycles, so the time is what the chain's warp has to do:
//  * up to three warps draw the next sweep's uniforms and turn them into limits
//    on s(h + g) while the first sweeps (sa_form; with many reads the first draws
//    them itself): rejecting a block of 32 spins is a few loads, a handful of
//    operations and one vote;
//  * a block with flips is resolved on registers against the limits (exact test
//    in between).  +-1 couplings (PM1): the block's flips change the fields of
//    all spins at once, from bits in shared memory.  Others: a flip's float32
//    row is asked for in pieces that are all in flight together with the one
//    coupling that the next decision needs (before, 32 loads one after another:
//    13 ms of a 15 ms call at an acceptance of 0.9%);
//  * the best state is stored once a block (its last improvement's flips).
// Whole call: +-1, n = 256, 64 reads, 1000 sweeps: 3.44 -> 2.83 ms; real, n = 1000,
// 128 reads, 200 sweeps: 13.8 -> 2.7 ms; real, n = 1500, 300 reads, 40 sweeps:
// 21.7 -> 3.9 ms.  Not kept: four blocks ahead (instructions count, not the votes'
// latency: 2.83 -> 3.31 ms), all rows prefetched into L1 and added per block
// (2.7 -> 4.4 ms).
#pragma once
#include <algorithm>
#include <type_traits>

#include "qa_ptc.cuh"

namespace qa {

constexpr int kSaWarps = 4;
// The sweeping warp and one for each 128 uniforms of a sweep, up to three.
static inline int sa_warps(int n) { return 1 + std::min(kSaWarps - 1, (n + 127) / 128); }

// How nr reads run: warps a read, 0 for sa_kernel.  many / one: reads resident on
// the GPU at once with sa_warps(n) warps and with one (which draws its own limits).
// Drawing ahead shortens a lone chain by up to 15% and costs residency (real
// couplings, n = 256: 592 reads against 1776), so it stops where the reads no longer
// fit, with two warps at half of that, where the SMs are busy without it (+-1,
// n = 64, 600 reads: 0.46 ms either way, 1000 reads 0.52 -> 0.48).  Real, n = 1000,
// 1000 reads 13.2 -> 5.0 ms; n = 256, 4000 reads 11.5 -> 5.6; +-1, n = 64, 8000 reads
// 2.72 -> 1.60.  +-1 from n = 400 on is bounded by shared memory either way (2%
// slower with one warp).  Reads beyond that of small real models go to sa_kernel,
// whose 64 registers hold 32 reads an SM against 12 here (n = 64, 4000 reads: one
// warp 2.00, sa_kernel 1.62 ms; n = 128, 4700 reads: 3.93 and 4.42), and the smallest
// ones at once (n = 9, 829 reads 0.64 / 0.55; n = 17, 1445 reads 1.12 / 1.04; n = 19, 923
// reads 0.119 / 0.125).
static inline int sa_form(bool pm1, int n, long long nr, long long many, long long one) {
    if (nr <= (sa_warps(n) > 2 ? many : many / 2)) return sa_warps(n);
    if (!pm1 && (n < 18 || (n < 96 && nr > one))) return 0;
    return one > many ? 1 : sa_warps(n);
}

template <bool PM1>
__host__ __device__ inline size_t sa_dense_smem_bytes(int n) {
    const int nw = (n + 31) / 32, np = pm1_npad(n);
    return (PM1 ? (size_t)nw * np * 4 : 0) + (size_t)np * 16 + (size_t)((nw + 3) & ~3) * 4;
}

// g += cf row over 128 NC columns from base on (cf = +-2: the product is exact).
template <int NC>
__device__ __forceinline__ void sa_add_row(const float *row, float *g, int ld, int base, float cf, int lane) {
    const int col = base + 4 * lane;
    const unsigned long long c2 = pack2(cf);
    ulonglong2 v[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (col + 128 * c < ld) v[c] = __ldg(reinterpret_cast<const ulonglong2 *>(row + col + 128 * c));
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (col + 128 * c < ld) {
            ulonglong2 x = *reinterpret_cast<ulonglong2 *>(g + col + 128 * c);
            fma2(x.x, v[c].x, c2);
            fma2(x.y, v[c].y, c2);
            *reinterpret_cast<ulonglong2 *>(g + col + 128 * c) = x;
        }
}

// ONE: one warp a read, which draws its own limits (a form of its own, so that the
// other carries none of it: real, n = 414, 3 reads, 650 sweeps 2.24 -> 2.19 ms).
template <bool PM1, bool ONE>
__global__ void __launch_bounds__(32 * kSaWarps) sa_dense_kernel(SAParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const RingDev R = p.rings[blockIdx.x];
    const ProbDev Pd = p.probs[R.prob];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = Pd.n, nw = Pd.nw, npad = pm1_npad(n);
    const int ld = dense_ld(n);
    using GT = typename std::conditional<PM1, int, float>::type;
    uint32_t *Jw = reinterpret_cast<uint32_t *>(smem);
    GT *G = reinterpret_cast<GT *>(Jw + (PM1 ? (size_t)nw * npad : 0));
    float *h = reinterpret_cast<float *>(G + npad);
    float *cb = h + npad;  // two sweeps' limits, by spin
    uint32_t *S = reinterpret_cast<uint32_t *>(cb + 2 * npad);
    if (PM1)
        for (int idx = threadIdx.x * 4; idx < nw * npad; idx += blockDim.x * 4)
            *reinterpret_cast<uint4 *>(Jw + idx) = __ldg(reinterpret_cast<const uint4 *>(Pd.Jw + idx));
    for (int q = threadIdx.x; q < nw; q += blockDim.x) S[q] = p.spins[R.spin_off + q];
    for (int i = threadIdx.x; i < npad; i += blockDim.x) h[i] = i < n ? Pd.h32[i] : 0.0f;
    __syncthreads();
    for (int m = threadIdx.x; m < npad; m += blockDim.x) {
        if (PM1) {
            int g = 0;
            if (m < n)
                for (int q = 0; q < nw; ++q) {
                    const int rem = n - 32 * q;
                    uint32_t vm = rem >= 32 ? FULL : ((1u << rem) - 1u);
                    if (q == (m >> 5)) vm &= ~(1u << (m & 31));
                    g += 2 * __popc(~(Jw[q * npad + m] ^ S[q]) & vm) - __popc(vm);
                }
            G[m] = (GT)g;
        } else {
            G[m] = m < n ? (GT)p.fields[R.field_off + m] : (GT)0;
        }
    }
    // limits of sweep x (0 .. steps * spb - 1) into buffer x & 1: c = ln(u) / 2 beta
    const long long sweeps = (long long)p.steps * p.spb;
    auto draw = [&](long long x, int w0, int ws) {
        const float rB = 1.0f / p.B[x / p.spb];
        float *c = cb + (x & 1) * npad;
        for (int b = w0; b < (nw + 3) >> 2; b += ws) {
            const U4 r = philox((uint32_t)(b * 32 + lane), 0u, (uint32_t)x, DOM_SA, R.key);
            c[128 * b + lane] = accept_limit(u24(r.x)) * rB;
            c[128 * b + 32 + lane] = accept_limit(u24(r.y)) * rB;
            c[128 * b + 64 + lane] = accept_limit(u24(r.z)) * rB;
            c[128 * b + 96 + lane] = accept_limit(u24(r.w)) * rB;
        }
    };
    draw(0, warp, (int)blockDim.x >> 5);
    __syncthreads();

    double E = 0.0, best;
    uint32_t *bb = p.best_bits + (long long)blockIdx.x * p.nw_max;
    int bstep = -1;
    unsigned long long acc = 0;
    if (warp == 0) {
        // E = c + (sum s h + (sum s g) / 2), sums in warp order (cell_energy)
        double ph = 0.0, pg = 0.0;
        for (int i = lane; i < n; i += 32) {
            const bool up = (S[i >> 5] >> (i & 31)) & 1u;
            ph = __dadd_rn(ph, up ? (double)h[i] : -(double)h[i]);
            pg = __dadd_rn(pg, up ? (double)G[i] : -(double)G[i]);
        }
        E = __dadd_rn(Pd.c, __dadd_rn(warp_sum_d(ph), __dmul_rn(0.5, warp_sum_d(pg))));
        for (int q = lane; q < nw; q += 32) bb[q] = S[q];
    }
    best = E;
    const float eps = accept_margin(0.0f);
    long long x = 0;
    for (int step = 0; step < p.steps; ++step) {
        const float B = p.B[step], eB = eps / B;
        // else every lane takes the exact test: no s g is below -inf or reaches a NaN
        // (an upper limit of +inf would accept an infinite field at B = 0)
        const bool plain = B > 1e-30f && B < 1e30f;
        for (int sw = 0; sw < p.spb; ++sw, ++x) {
            if (!ONE && warp != 0) {
                if (x + 1 < sweeps) draw(x + 1, warp - 1, ((int)blockDim.x >> 5) - 1);
            } else {
                if (ONE && x > 0) {  // nobody drew ahead
                    draw(x, 0, 1);
                    __syncwarp();
                }
                const float *c = cb + (x & 1) * npad;
#pragma unroll 1
                for (int q = 0; q < nw; ++q) {
                    const int i = (q << 5) | lane;
                    const uint32_t sword = S[q], sbit = (sword >> lane) & 1u;
                    const float hi = h[i], gf = (float)G[i], sh = sbit ? hi : -hi;
                    float sg = sbit ? gf : -gf;
                    const float th = c[i] - sh, e = __fmaf_rn(1e-6f, fabsf(c[i]) + fabsf(sh), eB);
                    const float lo = plain ? th - e : -f_inf(), up = plain ? th + e : __int_as_float(0x7fffffff);
                    uint32_t pend = n - (q << 5) >= 32 ? FULL : (1u << (n - (q << 5))) - 1u;
                    uint32_t m = __ballot_sync(FULL, sg >= lo) & pend;
                    if (!m) continue;
                    uint32_t F = 0, Fbest = 0;
                    const uint32_t jd = PM1 ? sword ^ Jw[q * npad + i] : 0u, jx = sbit ? jd : ~jd;
                    for (;;) {
                        if (m & ~__ballot_sync(FULL, sg >= up)) {
                            // between the limits: the exact test, its uniform drawn again
                            const float u = u24(pick(philox((uint32_t)(((q >> 2) << 5) | lane), 0u, (uint32_t)x, DOM_SA,
                                                            R.key), q & 3));
                            m = __ballot_sync(FULL, metropolis_nb24(__fmul_rn(__fadd_rn(sh, sg), B), u)) & pend;
                        }
                        if (!m) break;
                        const int j = __ffs(m) - 1;
                        F |= 1u << j;
                        pend &= ~((2u << j) - 1u);
                        // the energy falls by 2 s (h + g) of spin j, in float64
                        const double xj = __dadd_rn((double)__shfl_sync(FULL, sh, j), (double)__shfl_sync(FULL, sg, j));
                        if (PM1) {
                            sg = __fadd_rn(sg, ((jx >> j) & 1u) ? 2.0f : -2.0f);
                        } else {
                            // this lane's coupling and the row's pieces in flight
                            // together (zero diagonal: spin j's own field stays)
                            const float *row = Pd.J32 + (size_t)((q << 5) | j) * ld;
                            const float v = i < n ? __ldg(row + i) : 0.0f;
                            const float cf = (sword >> j) & 1u ? -2.0f : 2.0f;
                            if (ld <= 512) {
                                sa_add_row<4>(row, reinterpret_cast<float *>(G), ld, 0, cf, lane);
                            } else {
                                for (int base = 0; base < ld; base += 1024)
                                    sa_add_row<8>(row, reinterpret_cast<float *>(G), ld, base, cf, lane);
                            }
                            sg = __fmaf_rn(sbit ? cf : -cf, v, sg);
                        }
                        E = __dadd_rn(E, __dmul_rn(-2.0, xj));
                        if (E < best) {
                            best = E;
                            bstep = step;
                            Fbest = F;
                        }
                        m = __ballot_sync(FULL, sg >= lo) & pend;
                    }
                    if (!F) continue;
                    acc += (unsigned long long)__popc(F);
                    if (Fbest) {
                        for (int w = lane; w < nw; w += 32) bb[w] = w == q ? sword ^ Fbest : S[w];
                        __syncwarp();
                    }
                    if (lane == 0) S[q] = sword ^ F;
                    if constexpr (PM1) pm1_block_update(G, Jw, npad, n, q, F, sword, lane);
                    __syncwarp();
                }
            }
            __syncthreads();
        }
        if (warp == 0) {
            if (lane == 0) p.trace[(long long)blockIdx.x * p.steps + step] = E;
            if (p.mag_trace) sa_record_mag(p, S, n, nw, step, lane);
        }
    }
    for (int q = threadIdx.x; q < nw; q += blockDim.x) p.spins[R.spin_off + q] = S[q];
    if (!PM1)
        for (int i = threadIdx.x; i < n; i += blockDim.x) p.fields[R.field_off + i] = (float)G[i];
    if (threadIdx.x == 0) {
        p.best_E[blockIdx.x] = best;
        if (p.best_step) p.best_step[blockIdx.x] = bstep;
        atomicAdd(p.counters + 0, (unsigned long long)n * (unsigned long long)sweeps);
        atomicAdd(p.counters + 1, acc);
    }
}

}  // namespace qa
