// qa_ptc.cuh -- classical parallel tempering of dense +-1 models in one launch
// (parallel_tempering.cpp:36-122: Metropolis sweeps of one chain per beta,
// cascading neighbour swaps, the traces).
//
// One CTA per read, one warp per rung's chain, the couplings' bits shared by the
// chains.  The general path launches the rings once per swap interval and the
// swaps after it (pt_segment_kernel): at the sizes of this method the launches,
// the reload of each chain's state and the one-thread swap cascade are most of
// the time.  Here the chains stay in shared memory for the whole run and a
// barrier takes a launch's place; lane r of warp 0 holds slot r's energy in the
// cascade.  n = 128, 24 rungs, 32 reads, 100 steps of 5 sweeps, swaps after each:
// 9.8 -> 4.9 ms; n = 30 .. 400, 1 to 32 reads: 1.5 to 7 times faster.  One SM for a
// read's rungs costs less than the launches even where a launch per swap interval has
// an SM for each rung and swaps are rare: 1 read, 32 rungs, swaps every 1000 steps,
// n = 600 28 -> 25 ms, n = 8 3.7 -> 3.2 (1920 shapes, n = 8 .. 900, 2 to 32 rungs, 1 to
// 200 reads, intervals of 1 to 1000 steps: none slower).  What is left
// is the hottest chain of a read, whose blocks are chains of accepted flips
// (limits on s g instead of the exponential after each: 5.7 -> 4.9 ms).
#pragma once
#include "qa_dense.cuh"
#include "qa_pt.cuh"

namespace qa {

struct PTChainParams {
    const ProbDev *probs;
    const RingDev *rings;         // ring r of read q: q * R + r (slot r at the start)
    const uint32_t *spins;        // the starting states
    const float *B;               // [slot] 2 beta
    const double *bp;             // [slot] beta
    int R, steps, spb, swap_interval, nw_max;
    double *best_E;               // [ring], as the ring kernels record them:
    int *best_step, *best_slot;   //   step -1 is the starting state
    uint32_t *best_bits, *final_bits;  // [ring][nw_max]
    double *last_E;               // [ring * rec_stride] energy after the last step
    int rec_stride;
    int *ring_in;                 // [read][slot] ring in each slot at the end
    double *avg_trace, *swap_trace;    // [read][steps]
    unsigned long long *counters;
};

// The acceptance as limits on s g (the signed field without h): rejected below
// lo, accepted from up on, the exact test in between.  y = s(h + g) B - tro is
// increasing in s g for B > 0, so y >= limit is s g >= (limit + tro) / B - s h;
// the distance covers the limit's margin and the roundings of y and of this
// expression (rB = 1 / B; other B: every lane is in between).
__device__ __forceinline__ void field_limits(float u24v, float tro, float sh, float B, float rB, float eps, float *lo,
                                             float *up) {
    const float c = (accept_limit(u24v) + tro) * rB, th = c - sh;
    const float e = __fmaf_rn(1e-6f, fabsf(c) + fabsf(sh), eps * rB);
    const bool plain = B > 1e-30f && B < 1e30f;
    *lo = plain ? th - e : -__int_as_float(0x7f800000);
    *up = plain ? th + e : __int_as_float(0x7f800000);
}

// A block of 32 spins resolved in lane order, decisions on s g against limits
// (field_limits): the lanes flipped.  jx: bit j tells whether a flip of lane j
// raises this lane's s g by 2 or lowers it by 2 (the flipped lane's own is not
// used again); exact(sg) decides between the limits.  The loop is one chain of
// votes: add, compare, vote, lowest bit.
template <class Exact>
__device__ __forceinline__ uint32_t chain_resolve(float sg, float lo, float up, uint32_t jx, uint32_t pend,
                                                Exact exact) {
    uint32_t F = 0;
    while (pend) {
        uint32_t m = __ballot_sync(FULL, sg >= lo) & pend;
        if (m & ~__ballot_sync(FULL, sg >= up)) m = __ballot_sync(FULL, exact(sg)) & pend;
        if (!m) break;
        const uint32_t bit = m & (0u - m);
        F |= bit;
        pend &= ~(bit | (bit - 1u));
        sg = __fadd_rn(sg, (jx & bit) ? 2.0f : -2.0f);
    }
    return F;
}

__host__ __device__ inline size_t ptc_smem_bytes(int R, int n) {
    const int nw = (n + 31) / 32, np = pm1_npad(n);
    return (size_t)nw * np * 4 + (size_t)np * 4 + (size_t)R * np * 4 + align_up((size_t)R * nw * 4, 16) +
           (size_t)R * 8 + (size_t)R * 4 + 16;
}

__global__ void __launch_bounds__(1024, 1) pt_chains_kernel(PTChainParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int R = p.R, lane = threadIdx.x & 31, r = threadIdx.x >> 5, ring = blockIdx.x * R + r;
    const RingDev D = p.rings[ring];
    const ProbDev *Pd = p.probs + D.prob;
    const int n = Pd->n, nw = Pd->nw, npad = pm1_npad(n);
    const double c0 = Pd->c;
    unsigned char *ptr = smem;
    double *Es = reinterpret_cast<double *>(ptr); ptr += align_up((size_t)R * 8, 16);  // [ring]
    uint32_t *Jw = reinterpret_cast<uint32_t *>(ptr); ptr += (size_t)nw * npad * 4;
    float *h = reinterpret_cast<float *>(ptr); ptr += (size_t)npad * 4;
    int *G = reinterpret_cast<int *>(ptr) + (size_t)r * npad; ptr += (size_t)R * npad * 4;
    uint32_t *S = reinterpret_cast<uint32_t *>(ptr) + (size_t)r * nw; ptr += align_up((size_t)R * nw * 4, 16);
    int *slot_of = reinterpret_cast<int *>(ptr);  // [ring]
    for (int idx = threadIdx.x; idx < nw * npad; idx += blockDim.x) Jw[idx] = Pd->Jw[idx];
    for (int i = threadIdx.x; i < npad; i += blockDim.x) h[i] = i < n ? Pd->h32[i] : 0.0f;
    for (int q = lane; q < nw; q += 32) S[q] = p.spins[D.spin_off + q];
    if (lane == 0) slot_of[r] = r;
    __syncthreads();
    for (int m = lane; m < npad; m += 32) {
        int g = 0;
        if (m < n)
            for (int q = 0; q < nw; ++q) {
                const int rem = n - 32 * q;
                uint32_t vm = rem >= 32 ? FULL : ((1u << rem) - 1u);
                if (q == (m >> 5)) vm &= ~(1u << (m & 31));
                g += 2 * __popc(~(Jw[q * npad + m] ^ S[q]) & vm) - __popc(vm);
            }
        G[m] = g;
    }
    __syncwarp();

    int slot = r, my_ring = lane, bestStep = -1, bestSlot = r;  // warp 0: my_ring = the ring in slot `lane`
    double bestE = __longlong_as_double(0x7ff0000000000000LL);
    unsigned long long acc = 0;
    const float eps = accept_margin(0.0f);
    // E = c + (sum s h + (sum s g)/2), sums in warp order; best state
    auto score = [&](int step) {
        double ph = 0.0;
        int pg = 0;
        for (int i = lane; i < n; i += 32) {
            const uint32_t up = (S[i >> 5] >> (i & 31)) & 1u;
            ph = __dadd_rn(ph, (double)signed_by_bit(h[i], up));
            pg += up ? G[i] : -G[i];
        }
        const double E = __dadd_rn(c0, __dadd_rn(warp_sum_d(ph), __dmul_rn(0.5, (double)__reduce_add_sync(FULL, pg))));
        if (E < bestE) {
            bestE = E;
            bestStep = step;
            bestSlot = slot;
            for (int q = lane; q < nw; q += 32) p.best_bits[(long long)ring * p.nw_max + q] = S[q];
        }
        return E;
    };
    score(-1);
    for (int step = 0; step < p.steps; ++step) {
        const float B = p.B[slot], rB = 1.0f / B;
        for (int sw = 0; sw < p.spb; ++sw) {
            const uint32_t sigma = (uint32_t)(step * p.spb + sw);
            U4 rnd{0, 0, 0, 0};
#pragma unroll 1
            for (int q = 0; q < nw; ++q) {
                if ((q & 3) == 0) rnd = philox((uint32_t)(((q >> 2) << 5) | lane), (uint32_t)slot, sigma, DOM_SLICE | D.tag_extra, D.key);
                const int i = (q << 5) | lane;
                const uint32_t sw0 = S[q], sbit = (sw0 >> lane) & 1u;
                const float u = u24(pick(rnd, q & 3)), hi = h[i], Bs = sbit ? B : -B;
                const float gk = __int2float_rn(G[i]);
                if (!__any_sync(FULL, (i < n) & metropolis_maybe24(__fmul_rn(__fadd_rn(hi, gk), Bs), u))) continue;
                // resolve the block in spin order on registers (see pm1_block)
                float lo, up;
                field_limits(u, 0.0f, sbit ? hi : -hi, B, rB, eps, &lo, &up);
                const uint32_t F = chain_resolve(
                    sbit ? gk : -gk, lo, up, sbit ? sw0 ^ Jw[q * npad + i] : ~(sw0 ^ Jw[q * npad + i]),
                    __ballot_sync(FULL, i < n), [&](float sg) {
                        return metropolis_nb24(__fmul_rn(__fadd_rn(hi, sbit ? sg : -sg), Bs), u);
                    });
                if (!F) continue;
                acc += (unsigned long long)__popc(F);
                if (lane == 0) S[q] = sw0 ^ F;
                pm1_block_update(G, Jw, npad, n, q, F, sw0, lane);
                __syncwarp();
            }
        }
        const double E = score(step);
        if (lane == 0) Es[r] = E;
        __syncthreads();
        if (r == 0) {
            // slot `lane` holds ring my_ring; swaps of neighbouring slots in
            // order, each on the pair the ones before it left (pt_segment_kernel
            // with J_perp = 0), then the mean energy in slot order
            double e = lane < R ? Es[my_ring] : 0.0;
            const bool swap = (step + 1) % p.swap_interval == 0;
            int taken = 0;
            if (swap) {
                const double bl = lane < R ? p.bp[lane] : 0.0;
                const float ul = u01(philox((uint32_t)lane, 0u, (uint32_t)((step + 1) / p.swap_interval - 1), DOM_SWAP, D.key).x);
                for (int k = 0; k + 1 < R; ++k) {
                    const double ea = __shfl_sync(FULL, e, k), eb = __shfl_sync(FULL, e, k + 1);
                    const double ba = __shfl_sync(FULL, bl, k), bb = __shfl_sync(FULL, bl, k + 1);
                    const int xa = __shfl_sync(FULL, my_ring, k), xb = __shfl_sync(FULL, my_ring, k + 1);
                    const double delta = __dsub_rn(__dadd_rn(__dmul_rn(ba, eb), __dmul_rn(bb, ea)),
                                                   __dadd_rn(__dmul_rn(ba, ea), __dmul_rn(bb, eb)));
                    if (metropolis(__double2float_rn(-delta), __shfl_sync(FULL, ul, k))) {
                        if (lane == k) { e = eb; my_ring = xb; }
                        if (lane == k + 1) { e = ea; my_ring = xa; }
                        ++taken;
                    }
                }
                if (lane < R) slot_of[my_ring] = lane;
            }
            double avg = 0.0;
            for (int k = 0; k < R; ++k) avg = __dadd_rn(avg, __shfl_sync(FULL, e, k));
            if (lane == 0) {
                const long long o = (long long)blockIdx.x * p.steps + step;
                p.avg_trace[o] = __ddiv_rn(avg, (double)R);
                p.swap_trace[o] = swap ? __ddiv_rn((double)taken, (double)(R - 1)) : 0.0;
            }
        }
        __syncthreads();
        slot = slot_of[r];
        if (step == p.steps - 1) {
            for (int q = lane; q < nw; q += 32) p.final_bits[(long long)ring * p.nw_max + q] = S[q];
            if (lane == 0) p.last_E[(long long)ring * p.rec_stride] = E;
        }
    }
    if (r == 0 && lane < R) p.ring_in[(long long)blockIdx.x * R + lane] = my_ring;
    if (lane == 0) {
        p.best_E[ring] = bestE;
        p.best_step[ring] = bestStep;
        p.best_slot[ring] = bestSlot;
        atomicAdd(p.counters + 0, (unsigned long long)n * p.spb * p.steps);
        atomicAdd(p.counters + 1, acc);
    }
}

}  // namespace qa
