// qa_slab.cuh -- Trotter-ring sweep kernel for sparse models whose rows fit the
// 16-byte neighbour records (integer couplings in [-127, 127], at most four
// neighbours a spin).
//
// Same replay semantics as ring_kernel<K_SPARSE>; the loops are the other way
// round.  A move of spin i in slice t depends on its own slice's neighbours and
// on spin i in slices t - 1 and t + 1, so a sweep may take the spins outside and
// the slices inside, as long as (t, i) follows (t - 1, i) and (t, j) for the
// neighbours j before i in the visiting order:
//  * a warp takes 128 visiting positions (four blocks of 32, lane = position)
//    through all slices: records, fields h, own worldlines and the draws'
//    counters are loaded once for P slices, one Philox call serves the four
//    blocks of a slice, and slice t - 1's bit is in a register;
//  * warp after warp follows one slice step behind (a progress counter per 128
//    positions), which puts earlier neighbours' bits in place;
//  * within a block every lane decides at once; a lane with an earlier neighbour
//    in its block (known from the inverse order) is decided again while the
//    flips before it change.  Each is final once the flips of the lanes before
//    it are, so this ends in the sequential sweep's decisions, and most blocks
//    have no such lane that matters;
//  * decisions compare with a limit formed from log2 u (accept_limit), exact test
//    near it; the neighbours' bits of a slice are four rotated words and one
//    four-way byte dot product.
// Worldline moves take the same blocks in turn, one warp after the other.
//
// Bound by instruction issue: 122 warp instructions for 32 sites (585 before),
// 2.3 issued a cycle and SM.  SQA-PT, n = 2048, P = 16, 1024 rings, device time of
// 200 slice + 50 worldline sweeps: ring_sparse_kernel 144 -> 40.6 ms (58 -> 207 G
// site attempts/s).  80 registers, three CTAs of 8 warps an SM, about 200 bytes
// spilled in slab_sweep: 128 registers 54.1 against 52.1 ms for the call, 64 (more
// spilled) 64.1; 4 warps a ring the same.
// Not kept: four slices at a time on one reading of the neighbours' words (a
// ring's warps then follow four steps behind each other: 55 to 83 ms), sleeping
// in the waits (no change).
#pragma once
#include <algorithm>
#include <cmath>

#include "qa_dense.cuh"
#include "qa_sparse.cuh"

namespace qa {

// Shared memory of one ring: byte offsets (W, the worldline words, at 0).
struct SlabLay {
    uint32_t inv, ord0, ord1, prog, abortf, cellE, part, flag, total;
};
__host__ __device__ inline SlabLay slab_layout(int P, int n, int wbytes, bool ref_order) {
    const int nw = (n + 31) / 32, n32 = nw * 32, nsb = (n + 127) / 128;
    SlabLay L{};
    uint32_t o = (uint32_t)align_up((size_t)n32 * wbytes, 16);
    auto take = [&](size_t bytes) {
        const uint32_t at = o;
        o += (uint32_t)align_up(bytes, 16);
        return at;
    };
    L.prog = take((size_t)nsb * 4);   // steps done by each 128 positions
    L.abortf = take(4);
    L.cellE = take((size_t)P * 8);
    L.part = take((size_t)(32 + P) * 4);  // partial sums by warp; sums of s g by slice
    L.flag = take(16);                // [0]: best slice, [3]: lowest slice
    if (ref_order) {
        L.inv = take((size_t)n32 * 2);  // position of each spin
        L.ord0 = take(ord_row_bytes(n32));
        L.ord1 = take(ord_row_bytes(n32));
    }
    L.total = o;
    return L;
}
__host__ __device__ inline size_t slab_smem_bytes(int P, int n, bool ref_order) {
    return slab_layout(P, n, P <= 32 ? 4 : 8, ref_order).total;
}

// Whether a call's rings run here or on ring_sparse_kernel.  A sweep is P slices one
// after another for each 128 spins, so in the checkerboard order, where
// ring_sparse_kernel sweeps the slices of a phase side by side (two phases; three for
// an odd P, one for P = 1), few spins and many slices are faster there.  In units of a
// sixteenth of a slice here a sweep costs 16 (P + 2.5); there n + 24 a phase, times what
// the rings share an SM's 32 such warps.  One ring or a few, there / here: P = 32, 50
// slice sweeps: n = 40 0.64 / 1.74 ms, n = 128 1.34 / 2.02, n = 256 2.27 / 1.92; 40
// steps: P = 16, n = 104 0.89 / 1.17; P = 8, n = 52 1.60 / 1.90; P = 4, n = 12 0.27 /
// 0.38; P = 5, n = 40 2.01 / 1.25; P = 1, n = 14 0.114 / 0.162; many: P = 64, n = 40,
// 148 rings 0.90 / 3.86, 600 rings 4.7 / 4.1.  In qanneal's order both take one slice
// after another, and up to 13 spins are faster there (P = 20, n = 8, 14 rings 0.75 /
// 1.07 ms; P = 16, n = 10, 2 rings 0.66 / 0.87; n = 16 from 0.91 to 1.2 times as fast
// here).  2075 shapes, n = 8 .. 2000, 1 to 1500 rings, timed against
// ring_sparse_kernel: with the lines here 13 below 0.96 of its speed, down to 0.81.
inline bool slab_pays(int P, int n, int rings, int sms, bool ref_order) {
    const int w = (P + 1) / 2, per_sm = std::max(1, 32 / w), phases = P == 1 ? 1 : 2 + (P & 1);
    const double share = std::max(1.0 + 1.5 * std::max(0.0, (double)rings / sms - 1.0) * w / 32.0,
                                  std::ceil((double)rings / ((double)per_sm * sms)));
    if (ref_order && P > 1) return n * share > 13.0;
    return phases * (n + 24) * share > 16.0 * (P + 2.5);
}

__device__ __forceinline__ int popc_of(uint32_t w) { return __popc(w); }
__device__ __forceinline__ int popc_of(unsigned long long w) { return __popcll(w); }
// Bit t of w at bit k.
__device__ __forceinline__ uint32_t bit_at(uint32_t w, int t, int k) { return __funnelshift_r(w, w, t - k) & (1u << k); }
__device__ __forceinline__ uint32_t bit_at(unsigned long long w, int t, int k) {
    return bit_at(t < 32 ? (uint32_t)w : (uint32_t)(w >> 32), t & 31, k);
}

// Whole warp: until the 128 positions sb have done `need` steps.  Polls like
// spin_wait.
__device__ __forceinline__ void slab_wait(const int *prog, int need, int *abortf, unsigned long long *err, int lane) {
    unsigned long long t0 = 0;
    for (int k = 1; ld_acquire_cta(prog) < need; ++k) {
        if ((k & 63) == 0) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            bool out = *(volatile int *)abortf != 0;
            if (now - t0 > QA_WAIT_NS) {
                out = true;
                if (lane == 0) {
                    *(volatile int *)abortf = 1;
                    atomicExch(err, QA_DEV_ERR_TIMEOUT);
                }
            }
            if (__any_sync(FULL, out)) return;
            __nanosleep(40);
        }
    }
}

// A lane's spin in one block of 32 positions: its record, and for each
// neighbour the earlier lane of the block that holds it (0x80: none).
struct SlabSpin {
    uint32_t ca, cb, v;  // columns 0 | 1 << 16, 2 | 3 << 16; the four int8 couplings
    uint32_t near;       // four bytes
    uint32_t lanes;      // those lanes as a mask
    int i;
};
__device__ __forceinline__ int slab_col(const SlabSpin &s, int e) {
    return (int)(((e < 2 ? s.ca : s.cb) >> (16 * (e & 1))) & 0xFFFFu);
}

template <bool ORD>
__device__ __forceinline__ SlabSpin slab_load(const uint4 *slab, const OrdT *ord, const OrdT *inv, int n, int pos) {
    SlabSpin s;
    s.i = pos < n ? (ORD ? (int)ord[pos] : pos) : 0;
    const uint4 r = __ldg(slab + s.i);
    s.ca = r.x;
    s.cb = r.y;
    s.v = r.z;
    s.near = s.lanes = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int c = slab_col(s, e), p = ORD ? (int)inv[c] : c;
        const bool hit = ((s.v >> (8 * e)) & 0xFFu) != 0u && pos < n && (p >> 5) == (pos >> 5) && p < pos;
        s.near |= (hit ? (uint32_t)(p & 31) : 0x80u) << (8 * e);
        s.lanes |= hit ? 1u << (p & 31) : 0u;
    }
    return s;
}

// Mask with a 1 in byte e when neighbour e sits in an earlier lane of F.
__device__ __forceinline__ uint32_t slab_flipped(uint32_t near, uint32_t F) {
    uint32_t m = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const uint32_t b = near >> (8 * e);
        m |= ((b & 0x80u) ? 0u : ((F >> (b & 31u)) & 1u)) << (8 * e);
    }
    return m;
}

// One slice sweep (all slices), one warp's share; the number of flips.
template <class WT, bool ORD>
__device__ __noinline__ int slab_sweep(const uint4 *slab, const float *h32, uint32_t ordo, unsigned long long *err,
                                       int n, int NP, int W, float B, float T4, uint64_t key, uint32_t cell,
                                       uint32_t sigma, uint32_t tag) {
    const int lane = threadIdx.x & 31;
    const SlabLay L = slab_layout(NP, n, (int)sizeof(WT), ORD);
    WT *Wc = dsm<WT>(0);
    int *prog = dsm<int>(L.prog), *abortf = dsm<int>(L.abortf);
    const OrdT *ord = dsm<OrdT>(ordo), *inv = dsm<OrdT>(L.inv);
    const int nsb = (n + 127) >> 7;
    const float eps = accept_margin(T4), hT = 0.5f * T4;
    const int even = (NP & 1) ? (NP - 1) / 2 : NP / 2;  // checkerboard: slices 0, 2, .., then 1, 3, .., then an odd last
    int flips = 0;
    for (int sb = threadIdx.x >> 5; sb < nsb; sb += W) {
        SlabSpin s[4];
        float h[4];
        WT w[4];
        uint32_t near_any = 0;  // bit k: block k has lanes with earlier neighbours in it
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int pos = (sb << 7) + 32 * k + lane;
            s[k] = slab_load<ORD>(slab, ord, inv, n, pos);
            h[k] = __ldg(h32 + s[k].i);
            w[k] = Wc[s[k].i];
            near_any |= __any_sync(FULL, s[k].lanes != 0u) ? 1u << k : 0u;
        }
#pragma unroll 1
        for (int st = 0; st < NP; ++st) {
            const int t = ORD ? st : (st < even ? 2 * st : (st < even + NP / 2 ? 2 * (st - even) + 1 : NP - 1));
            const int tp = t == 0 ? NP - 1 : t - 1, tn = t + 1 == NP ? 0 : t + 1;
            const U4 r = philox((uint32_t)(sb * 32 + lane), cell + (uint32_t)t, sigma, tag, key);
            if (sb > 0) slab_wait(prog + sb - 1, st + 1, abortf, err, lane);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float u = u24(k == 0 ? r.x : (k == 1 ? r.y : (k == 2 ? r.z : r.w)));
                const bool valid = (sb << 7) + 32 * k + lane < n;
                // the neighbours' bits as bytes 0 / 2: 2 sum v b, less sum v, is the field
                uint32_t nb = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) nb |= bit_at(Wc[slab_col(s[k], e)], t, 8 * e + 1);
                const int base = 0x4B400000 - __dp4a((int)s[k].v, 0x01010101, 0);
                const uint32_t up = bit_at(w[k], t, 31);
                // s(s_p + s_n) T4 / 2, exact: each half T4 with the sign of s s_x
                const float tro = __int_as_float((int)((up ^ bit_at(w[k], tp, 31)) ^ __float_as_uint(hT))) +
                                  __int_as_float((int)((up ^ bit_at(w[k], tn, 31)) ^ __float_as_uint(hT)));
                const float Bs = __uint_as_float(__float_as_uint(B) ^ up ^ 0x80000000u);  // s B
                const float lim = accept_limit(u) + tro;
                auto decide = [&](uint32_t bits) {
                    // the small integer g as a float: 1.5 * 2^23 + g in the low bits
                    const float g = __int_as_float(base + __dp4a((int)s[k].v, (int)bits, 0)) - 12582912.0f;
                    const float xs = __fmul_rn(__fadd_rn(h[k], g), Bs);
                    bool ok = xs >= lim;
                    if (__any_sync(FULL, !(fabsf(xs - lim) > eps))) ok = metropolis_nb24(__fsub_rn(xs, tro), u);
                    return valid & ok;
                };
                bool ok = decide(nb);
                uint32_t F = __ballot_sync(FULL, ok);
                if ((near_any >> k) & 1u) {
                    uint32_t before = 0;  // the flips the lanes were last decided on
                    while (__any_sync(FULL, (s[k].lanes & (F ^ before)) != 0u)) {
                        before = F;
                        ok = decide(nb ^ (slab_flipped(s[k].near, before) << 1));
                        F = __ballot_sync(FULL, ok);
                    }
                }
                if (ok) {
                    w[k] ^= (WT)1 << t;
                    Wc[s[k].i] = w[k];
                    ++flips;
                }
                __syncwarp();
            }
            __threadfence_block();
            __syncwarp();
            if (lane == 0) st_release_cta(prog + sb, st + 1);
        }
    }
    return __reduce_add_sync(FULL, flips);
}

// One worldline sweep, one warp's share (prog reset by the caller); the number
// of moves.
template <class WT, bool ORD>
__device__ __noinline__ int slab_worldlines(const uint4 *slab, const float *h32, uint32_t ordo, unsigned long long *err,
                                            int n, int NP, int W, float B, uint64_t key, uint32_t slot,
                                            uint32_t sigma) {
    const int lane = threadIdx.x & 31;
    const SlabLay L = slab_layout(NP, n, (int)sizeof(WT), ORD);
    WT *Wc = dsm<WT>(0);
    int *prog = dsm<int>(L.prog), *abortf = dsm<int>(L.abortf);
    const OrdT *ord = dsm<OrdT>(ordo), *inv = dsm<OrdT>(L.inv);
    const WT pmask = NP == 8 * (int)sizeof(WT) ? ~(WT)0 : (((WT)1 << NP) - 1);
    int moves = 0;
    for (int sb = threadIdx.x >> 5; sb < (n + 127) >> 7; sb += W) {
        const U4 r = philox((uint32_t)(sb * 32 + lane), slot, sigma, DOM_WORLD, key);
        SlabSpin s[4];
        float h[4];
        WT w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            s[k] = slab_load<ORD>(slab, ord, inv, n, (sb << 7) + 32 * k + lane);
            h[k] = __ldg(h32 + s[k].i);
            w[k] = Wc[s[k].i];
        }
        if (sb > 0) slab_wait(prog + sb - 1, 1, abortf, err, lane);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float u = u24(k == 0 ? r.x : (k == 1 ? r.y : (k == 2 ? r.z : r.w)));
            const bool valid = (sb << 7) + 32 * k + lane < n;
            const int sh = 2 * popc_of(w[k]) - NP;
            int d[4];  // slices in which the neighbour differs
#pragma unroll
            for (int e = 0; e < 4; ++e) d[e] = popc_of((WT)(w[k] ^ Wc[slab_col(s[k], e)]));
            auto decide = [&](uint32_t fl) {  // fl: byte e, neighbour e has moved
                int gs = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int a = NP - 2 * d[e];
                    gs += (int)(signed char)(s[k].v >> (8 * e)) * ((fl >> (8 * e)) & 1u ? -a : a);
                }
                const float x = __double2float_rn(__dadd_rn(__dmul_rn((double)h[k], (double)sh), (double)gs));
                return valid & metropolis_nb24(__fmul_rn(x, B), u);
            };
            bool ok = decide(0u);
            uint32_t F = __ballot_sync(FULL, ok), before = 0;
            while (__any_sync(FULL, (s[k].lanes & (F ^ before)) != 0u)) {
                before = F;
                ok = decide(slab_flipped(s[k].near, before));
                F = __ballot_sync(FULL, ok);
            }
            if (ok) {
                Wc[s[k].i] = w[k] ^ pmask;
                ++moves;
            }
            __syncwarp();
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0) st_release_cta(prog + sb, 1);
    }
    return __reduce_add_sync(FULL, moves);
}

// sum_i s_i g_i of every slice into sg[P] (zeroed by the caller), whole CTA: a
// lane's neighbours' words are read once for all slices.
template <class WT>
__device__ __noinline__ void slab_bond_energies(const uint4 *slab, int n, int NP, int *sg) {
    const int lane = threadIdx.x & 31;
    const WT *Wc = dsm<WT>(0);
    for (int t0 = 0; t0 < NP; t0 += 8) {  // eight slices at a time in registers
        int acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const uint4 r = __ldg(slab + i);
            const WT w = Wc[i];
            const SlabSpin s{r.x, r.y, r.z, 0u, 0u, i};
            WT x[4];  // bit t: the neighbour agrees with spin i in slice t
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = ~(w ^ Wc[slab_col(s, e)]);
            const int sv = __dp4a((int)r.z, 0x01010101, 0);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int t = (t0 + k) & (8 * (int)sizeof(WT) - 1);  // (behind the last slice: not read)
                uint32_t b = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) b |= bit_at(x[e], t, 8 * e + 1);
                acc[k] += __dp4a((int)r.z, (int)b, 0) - sv;
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int v = __reduce_add_sync(FULL, acc[k]);
            if (lane == 0 && t0 + k < NP) atomicAdd(sg + t0 + k, v);
        }
    }
}

template <class WT, bool ORD>
__global__ void __launch_bounds__(256, 3) ring_slab_kernel(RingParams p) {
    const RingDev R = p.rings[blockIdx.x];
    const ProbDev *Pd = p.probs + R.prob;
    const int NP = p.P, W = p.W, n = Pd->n, nw = Pd->nw, nsb = (n + 127) >> 7;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 *slab = Pd->spslab;
    const float *h32 = Pd->h32;
    const SlabLay L = slab_layout(NP, n, (int)sizeof(WT), ORD);
    WT *Wc = dsm<WT>(0);
    double *cellE = dsm<double>(L.cellE);
    int *wpart = dsm<int>(L.part), *sg = wpart + 32, *flag = dsm<int>(L.flag), *prog = dsm<int>(L.prog);
    if (threadIdx.x == 0) *dsm<int>(L.abortf) = 0;
    for (int q = warp; q < nw; q += W) {
        WT wc = 0;
        const int i = (q << 5) | lane;
        for (int t = 0; t < NP; ++t) wc |= (WT)((p.spins[R.spin_off + t * nw + q] >> lane) & 1u) << t;
        Wc[i] = i < n ? wc : (WT)0;
    }
    __syncthreads();

    const WT pmask = NP == 8 * (int)sizeof(WT) ? ~(WT)0 : (((WT)1 << NP) - 1);
    const int slot = p.slot ? p.slot[blockIdx.x] : R.k;
    OrderFeed feed = feed_open(ORD ? dsm<OrdT>(L.ord0) : nullptr, ORD ? dsm<OrdT>(L.ord1) : nullptr,
                               ORD ? p.ordg + blockIdx.x * p.ord_ring : nullptr, p.ord_stride, n,
                               ORD ? (p.step1 - p.step0) * p.ord_per_step : 0);
    unsigned long long att_s = 0, acc_s = 0, att_w = 0, acc_w = 0;
    double bestE = p.best_E[blockIdx.x];
    int bestStep = p.best_step[blockIdx.x];
    // sum over the CTA's spins of f(worldline word); valid on thread 0
    auto spin_total = [&](auto f) {
        int s = 0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) s += f(Wc[i]);
        s = __reduce_add_sync(FULL, s);
        if (lane == 0) wpart[warp] = s;
        __syncthreads();
        long long tot = 0;
        if (threadIdx.x == 0)
            for (int w = 0; w < W; ++w) tot += wpart[w];
        return tot;
    };
    // imaginary-time bonds of one worldline: P - 2 (slices that differ from the next)
    auto bonds = [&](WT w) { return NP - 2 * popc_of((WT)((w ^ ((w >> 1) | ((w & 1) << (NP - 1)))) & pmask)); };
    // a sweep's order, its inverse and a clean progress row; whole CTA
    auto begin_sweep = [&]() {
        uint32_t ord = 0;
        for (int b = threadIdx.x; b < nsb; b += blockDim.x) prog[b] = 0;
        if (ORD) {
            const OrdT *o = feed_take(feed);
            OrdT *inv = dsm<OrdT>(L.inv);
            for (int x = threadIdx.x; x < n; x += blockDim.x) inv[o[x]] = (OrdT)x;
            ord = (uint32_t)(reinterpret_cast<const unsigned char *>(o) - dense_sm);
        }
        __syncthreads();
        return ord;
    };

    for (int step = p.step0 - (p.init_scan ? 1 : 0); step < p.step1; ++step) {
        // step -1 (init_scan) only scores the starting state
        const int spb = step >= 0 ? p.spb : 0, wls = step >= 0 ? p.wls : 0;
        const int si_tab = R.sched + (p.per_slot_sched ? slot + max(step, 0) * p.slot_step : max(step, 0));
        const float B = p.B[si_tab], T4 = p.T4[si_tab];
        for (int sw = 0; sw < spb; ++sw) {
            const uint32_t sigma = (uint32_t)(step * p.spb + sw);
            const uint32_t ord = begin_sweep();
            const int f = slab_sweep<WT, ORD>(slab, h32, ord, p.counters + 4, n, NP, W, B, T4, R.key,
                                              (uint32_t)(slot * NP), sigma, p.slice_tag | R.tag_extra);
            acc_s += (unsigned long long)f;
            if (threadIdx.x == 0) att_s += (unsigned long long)NP * (unsigned long long)n;
            __syncthreads();
            if (p.mag) {
                const long long up = spin_total([&](WT w) { return popc_of(w); });
                if (threadIdx.x == 0)
                    p.mag[(long long)blockIdx.x * (p.steps_total * p.spb) + sigma] = (int)(2 * up - (long long)NP * n);
                __syncthreads();
            }
            if (p.bsamp) {
                const long long b = spin_total(bonds);
                if (threadIdx.x == 0)
                    p.bsamp[(long long)blockIdx.x * p.bstride + (long long)(step - p.step0) * p.spb + sw] = b;
                __syncthreads();
            }
        }
        for (int sw = 0; sw < wls; ++sw) {
            const uint32_t sigma = (uint32_t)(step * p.wls + sw);
            const uint32_t ord = begin_sweep();
            const int f =
                slab_worldlines<WT, ORD>(slab, h32, ord, p.counters + 4, n, NP, W, B, R.key, (uint32_t)slot, sigma);
            if (lane == 0) acc_w += (unsigned long long)f;
            if (threadIdx.x == 0) att_w += (unsigned long long)n;
            __syncthreads();
        }
        // ---- step end: slice energies E = c + (sum s h + (sum s g)/2), ring sum, best
        for (int t = threadIdx.x; t < NP; t += blockDim.x) sg[t] = 0;
        __syncthreads();
        slab_bond_energies<WT>(slab, n, NP, sg);
        for (int t = warp; t < NP; t += W) {
            double ph = 0.0;
            for (int i = lane; i < n; i += 32) {
                const double hv = (double)__ldg(h32 + i);
                ph = __dadd_rn(ph, (Wc[i] >> t) & 1 ? hv : -hv);
            }
            ph = warp_sum_d(ph);
            if (lane == 0) cellE[t] = ph;
        }
        const long long bsum = p.ring_bond ? spin_total(bonds) : 0;
        __syncthreads();
        for (int t = threadIdx.x; t < NP; t += blockDim.x)
            cellE[t] = __dadd_rn(Pd->c, __dadd_rn(cellE[t], __dmul_rn(0.5, (double)sg[t])));
        __syncthreads();
        if (threadIdx.x == 0) {
            double sum = 0.0, emin = __longlong_as_double(0x7ff0000000000000LL);
            int tmin = 0;
            for (int t = 0; t < NP; ++t) {
                const double E = cellE[t];
                sum = __dadd_rn(sum, E);
                if (E < emin) { emin = E; tmin = t; }
            }
            const long long ro = (long long)blockIdx.x * p.rec_stride + p.rec_base + step;
            if (p.ring_sum) p.ring_sum[ro] = sum;
            if (p.ring_min) p.ring_min[ro] = emin;
            if (p.ring_bond) p.ring_bond[ro] = bsum;
            flag[0] = emin < bestE ? tmin : -1;
            flag[3] = tmin;
        }
        __syncthreads();
        const int tb = flag[0], tl = flag[3];
        if (tb >= 0) {
            bestE = cellE[tb];
            bestStep = step;
            if (threadIdx.x == 0 && p.best_slot) p.best_slot[blockIdx.x] = slot;
        }
        const bool fin = p.final_bits && step == p.steps_total - 1;
        if (tb >= 0 || fin)
            for (int q = warp; q < nw; q += W) {
                const WT w = Wc[(q << 5) | lane];
                const uint32_t bb = __ballot_sync(FULL, tb >= 0 && ((w >> (tb & 63)) & 1));
                const uint32_t bf = __ballot_sync(FULL, ((w >> tl) & 1) != 0);
                if (lane == 0) {
                    if (tb >= 0) p.best_bits[(long long)blockIdx.x * p.nw_max + q] = bb;
                    if (fin) p.final_bits[(long long)blockIdx.x * p.nw_max + q] = bf;
                }
            }
        __syncthreads();
    }
    for (int q = warp; q < nw; q += W) {
        const WT w = Wc[(q << 5) | lane];
        for (int t = 0; t < NP; ++t) {
            const uint32_t b = __ballot_sync(FULL, ((w >> t) & 1) != 0);
            if (lane == 0) p.spins[R.spin_off + t * nw + q] = b;
        }
    }
    if (lane == 0) {
        atomicAdd(p.counters + 1, acc_s);
        atomicAdd(p.counters + 3, acc_w);
    }
    if (threadIdx.x == 0) {
        atomicAdd(p.counters + 0, att_s);
        atomicAdd(p.counters + 2, att_w);
        p.best_E[blockIdx.x] = bestE;
        p.best_step[blockIdx.x] = bestStep;
    }
}

}  // namespace qa
