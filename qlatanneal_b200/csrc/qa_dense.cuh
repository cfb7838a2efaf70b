// qa_dense.cuh -- Trotter-ring sweep kernel for dense models with real
// couplings (QUBO matrices first of all).
//
// Same replay semantics as ring_kernel<K_DENSE> (qa_kernels.cuh); different
// data path.  What bounds this path is the chain of decisions of a sweep and,
// for each accepted flip, one coupling row added to the slice's n fields.
//  * A block of 32 spins is decided on registers alone: each lane carries its
//    spin's field, takes a flip of the block from one coupling, and compares
//    s(h+g)B with a limit formed once per block (ln u plus the Trotter term)
//    instead of evaluating e^y after every flip.  The limit is good to about
//    2e-5; a lane nearer to it than 1e-4 evaluates the exact test.
//  * The fields of the whole slice take all flips of the block at once, in
//    flip order: one load and store of each field, and one packed fused
//    multiply-add per coupling pair (the product with +-2 is exact, so the
//    sum is the one the flip-by-flip update rounds).
//  * qanneal's order: the slices are handed on spin by spin, not block by
//    block.  While it decides a block a slice publishes how far it has got and
//    its new bits in one 64-bit word; the next slice stops only at a spin that
//    its predecessor has not decided and that could flip under either value
//    of the predecessor's bit.
//  * Worldline moves: each warp evaluates one block of 32 positions on the
//    current worldlines; the first block with a move is resolved by its own
//    warp on a copy of the block's fields, its flips go to every slice at once,
//    and the evaluation resumes behind it.
// Spins live as worldline words (bit t of W[i]: slice t), P <= 64.
//
// Measured (solve() on a real QUBO, the whole call; before: ring_kernel):
//   n = 24,  P = 32, 1 read,    50 steps of 20 + 5 sweeps   31.5 -> 10.9 ms
//   n = 200, P = 32, 32 reads,  50 steps of 20 + 5 sweeps   85.3 -> 28.8 ms
//   n = 200, P = 32, 600 reads, 20 steps of 20 + 5 sweeps  151.9 -> 67.5 ms
//   n = 900, P = 16, 100 reads, 40 steps of 2 + 1 sweeps    76.6 -> 14.7 ms
// What is left is the chain of votes: at n = 24 each further slice adds 0.26 us
// (500 cycles) to a sweep.  Not kept: the couplings of a block in a shared-memory
// tile (its gather cost what it saved), J in shared memory (48.7 against
// 43.8 ms at n = 200, in an earlier form), 32 warps at 64 registers (30 -> 48 ms),
// a shorter loop for blocks whose predecessor is done (the
// chain, not the instruction count, is the time).
#pragma once
#include <algorithm>
#include <cmath>

#include "qa_pm1.cuh"

namespace qa {

// Row stride of J32 and of a slice's fields in shared memory: 16-byte rows.
__host__ __device__ inline int dense_ld(int n) { return (n + 3) & ~3; }

// Shared memory of one ring: byte offsets.  The sweeps are functions of their
// own (a slice sweep and the rest of the kernel together would not fit the 128
// registers of a 512-thread CTA) and take offsets, so that their accesses
// stay shared-memory ones.
struct DenseLay {
    uint32_t G, W, h, uw, cellE, gb, wold, wsp, mask, part, flag, ord0, ord1, prog, pbits, abortf, total;
};
__host__ __device__ inline DenseLay dense_layout(int P, int n, bool ref_order) {
    const int nw = (n + 31) / 32, n32 = nw * 32, ld = dense_ld(n);
    DenseLay L{};
    uint32_t o = 0;
    auto take = [&](size_t bytes) {
        const uint32_t at = o;
        o += (uint32_t)align_up(bytes, 16);
        return at;
    };
    L.G = take((size_t)P * ld * 4);      // fields [P][ld]
    L.W = take((size_t)n32 * 8);         // worldline bits
    L.h = take((size_t)n32 * 4);
    L.uw = take((size_t)n32 * 4);        // worldline uniforms
    L.cellE = take((size_t)P * 8);
    L.gb = take((size_t)P * 32 * 4);     // [P][32] a worldline block's fields
    L.wold = take(32 * 8);               // a worldline block's old words,
    L.wsp = take(32 * 4);                //   its spins
    L.mask = take(2 * 32 * 4);           // move masks of a worldline round, two rounds
    L.part = take(32 * 4);
    L.flag = take(16);                   // [0]: best slice, [1]: worldline flips F, [3]: lowest slice
    if (ref_order) {
        L.ord0 = take(ord_row_bytes(n32));
        L.ord1 = take(ord_row_bytes(n32));
        L.prog = take((size_t)P * 8);
        L.pbits = take((size_t)P * nw * 4);
        L.abortf = take(4);
    }
    L.total = o;
    return L;
}
__host__ __device__ inline size_t dense_smem_bytes(int P, int n, bool ref_order) {
    return dense_layout(P, n, ref_order).total;
}

// Warps of a ring, 0 for ring_kernel.  One per slice up to 16 (128 registers a
// thread); 8 where the rings are at least two waves and blocks are few (n <= 256):
// two rings on an SM then beat one with twice the warps (P = 32, 600 rings: n = 24
// 23.3 -> 17.7 ms, n = 64 36.8 -> 28.3, n = 200 69.9 -> 66.4; 300 rings of n = 900
// 25.1 -> 28.2, so not there).  In the checkerboard order half the slices rest: with
// more rings than SMs no more warps than slices of a phase, and of those the number
// with the least waves of rings times rounds of a phase's slices (0.4: the rest of a
// sweep in rounds; 350 shapes of n = 66 .. 400, P = 3 .. 48, 160 to 1200 rings: 1% from
// the best number on average, 10% with 8 or a phase's slices for all; n = 84, P = 20,
// 371 rings, 60 slice sweeps 1.61 -> 1.03 ms, ring_kernel 1.23).  With at most two
// blocks nothing is left of the shorter chain where a phase's slices no longer fit on
// the SMs, 16 warps each: ring_kernel has 64 registers (n = 24: P = 8, 3000 rings 0.56
// here with 4 warps / 0.46 there; P = 24, 300 rings 0.35 / 0.29).  smem: a ring's shared
// memory, cap: an SM's.
inline int dense_warps(int P, int n, int rings, int sms, bool ref_order, size_t smem, size_t cap) {
    const int w = std::min(P, rings >= 2 * sms && n <= 256 ? 8 : 16);
    if (ref_order && P > 1) return w;
    const int phase = (P + 1) / 2;
    if (n <= 64 && rings > sms * (16 / phase)) return 0;
    if (rings <= sms) return w;
    const int fit = std::max(1, (int)(cap / smem));
    int best = 1;
    double cost = 0.0;
    for (int v = 1; v <= std::min(phase, 16); ++v) {
        const double waves = std::ceil((double)rings / ((double)std::min(16 / v, fit) * sms));
        const double c = waves * ((phase + v - 1) / v + 0.4);
        if (v == 1 || c <= cost) {
            best = v;
            cost = c;
        }
    }
    return best;
}

extern __shared__ __align__(16) unsigned char dense_sm[];
template <class T>
__device__ __forceinline__ T *dsm(uint32_t off) {
    return reinterpret_cast<T *>(dense_sm + off);
}

__device__ __forceinline__ unsigned long long ld_acquire_cta64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.cta.shared.b64 %0, [%1];"
                 : "=l"(v)
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.cta.shared.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "l"(v)
                 : "memory");
}
// Enough for a slice's progress: the word itself carries the new bits of the block in
// work, pbits of a finished block precede a fence and a store for the next block, and
// nothing else is handed on: no slice reads another's flips in the worldline words,
// nor its fields, before the next CTA barrier.  Nor can the store pass the reads of the
// next slice's old bits, which that slice may flip once it sees the word: the votes
// that the word's count rests on have consumed them.
__device__ __forceinline__ void st_relaxed_cta64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.cta.shared.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "l"(v)
                 : "memory");
}

// The slices' hand-off in qanneal's order.  prog[t]: low word, the visiting
// positions slice t has decided in this sweep; high word, its new bits by
// position for the block it is deciding.  pbits[t * nw + q]: its bits of a
// finished block.
struct SpinPipe {
    unsigned long long *prog;  // [P]
    uint32_t *pbits;           // [P][nw]
    int *abortf;
    unsigned long long *err;
};

// Whole warp: until slice t has decided `need` positions; returns its word.
// The wait is on the sweep's critical path: it polls without a back-off and
// looks at the clock and the abort flag (bounded like pipe_wait) only every
// 64 polls.
__device__ __forceinline__ unsigned long long spin_wait(const SpinPipe &pp, int t, int need, int lane) {
    unsigned long long t0 = 0;
    for (int k = 1;; ++k) {
        const unsigned long long v = ld_acquire_cta64(pp.prog + t);
        if ((int)(uint32_t)v >= need) return v;
        if ((k & 63) == 0) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            bool out = *(volatile int *)pp.abortf != 0;
            if (now - t0 > QA_WAIT_NS) {
                out = true;
                if (lane == 0) {
                    *(volatile int *)pp.abortf = 1;
                    atomicExch(pp.err, QA_DEV_ERR_TIMEOUT);
                }
            }
            if (__any_sync(FULL, out)) return 0x7fffffffull;
            __nanosleep(40);
        }
    }
}

// ln(u) of the scaled uniform u24 = u 2^24 as a limit on y: accept iff
// y >= limit, up to 2e-5 (the approximate log2 is good to 4e-6, e^y's own
// polynomial and the roundings to about 1e-5).  u = 0 accepts iff y > -17.
__device__ __forceinline__ float accept_limit(float u24v) {
    float l;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(u24v));  // u24 is 0 or at least 1
    return fmaxf(__fmaf_rn(l, 0.693147181f, -16.6355323f), -17.0f);
}
// Distance from the limit below which the exact test decides: five times the
// limit's error, and the rounding of limit + Trotter term where T4 is large.
__device__ __forceinline__ float accept_margin(float T4) { return __fmaf_rn(fabsf(T4), 5e-7f, 1e-4f); }

__device__ __forceinline__ void fma2(unsigned long long &g, unsigned long long j, unsigned long long c) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(g) : "l"(j), "l"(c));
}
__device__ __forceinline__ unsigned long long pack2(float c) {
    const unsigned long long b = (unsigned)__float_as_int(c);
    return b | (b << 32);
}

// Fields of one slice after the spins of lanes F flipped (lane's spin i, old
// bits ups by lane): NC groups of 128 fields from column base on, a flip's
// pieces of its row in flight at once.
template <int NC>
__device__ __forceinline__ void dense_update_cols(const float *J, int ld, float *gt, uint32_t F, int i, uint32_t ups,
                                                  int base, int lane) {
    const int col = base + 4 * lane;
    ulonglong2 g[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (col + 128 * c < ld) g[c] = *reinterpret_cast<const ulonglong2 *>(gt + col + 128 * c);
#pragma unroll 1
    for (uint32_t f = F; f; f &= f - 1) {
        const int j = __ffs(f) - 1;
        const unsigned long long cf = pack2((ups >> j) & 1u ? -2.0f : 2.0f);
        const float *r = J + (size_t)__shfl_sync(FULL, i, j) * ld + col;
        ulonglong2 v[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (col + 128 * c < ld) v[c] = __ldg(reinterpret_cast<const ulonglong2 *>(r + 128 * c));
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (col + 128 * c < ld) {
                fma2(g[c].x, v[c].x, cf);
                fma2(g[c].y, v[c].y, cf);
            }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (col + 128 * c < ld) *reinterpret_cast<ulonglong2 *>(gt + col + 128 * c) = g[c];
}

// More than 256 fields (WIDE): four groups at a time, so that 512 columns of a
// row are in flight at once, in a function of its own (its registers would
// push the block's state out).  Two groups at a time against this:
//   n = 900,  P = 16, 100 reads, 40 steps of 2 + 1 sweeps  16.3 -> 14.7 ms
//   n = 400,  P = 32, 40 reads,  20 steps of 20 + 5        29.1 -> 27.7 ms
//   n = 280,  the same                                      20.8 -> 20.7 ms
//   n = 1500, P = 16, 20 reads,  5 steps of 20 + 5          40.8 -> 33.0 ms
// At most 256 fields keep the loop in line: the call costs there (n = 24
// 10.9 -> 11.5 ms, n = 200 28.9 -> 31.5 ms).  Eight groups at a time: n = 900
// 27.0 ms.  At 128 registers the kernels spill 16 to 56 bytes, the WIDE ones 164
// to 264 around the calls and at most 12 inside a sweep.
__device__ __noinline__ void dense_update_wide(const float *J, int ld, float *gt, uint32_t F, int i, uint32_t ups,
                                               int lane) {
    int base = 0;
#pragma unroll 1
    for (; base + 256 < ld; base += 512) dense_update_cols<4>(J, ld, gt, F, i, ups, base, lane);
#pragma unroll 1
    for (; base + 128 < ld; base += 256) dense_update_cols<2>(J, ld, gt, F, i, ups, base, lane);
    if (base < ld) dense_update_cols<1>(J, ld, gt, F, i, ups, base, lane);
}

template <bool WIDE>
__device__ __forceinline__ void dense_update(const float *J, int ld, float *gt, uint32_t F, int i, uint32_t ups,
                                             int lane) {
    __syncwarp();
    if (WIDE) {
        dense_update_wide(J, ld, gt, F, i, ups, lane);
    } else {
        int base = 0;
#pragma unroll 1
        for (; base + 128 < ld; base += 256) dense_update_cols<2>(J, ld, gt, F, i, ups, base, lane);
        if (base < ld) dense_update_cols<1>(J, ld, gt, F, i, ups, base, lane);
    }
    __syncwarp();
}

// One block of 32 positions of slice t (ORD: qanneal's order, spins ord[...];
// else the checkerboard, spins ascending).
template <bool ORD, bool WIDE>
__device__ __forceinline__ int dense_block(const float *J, int ld, float *gt, unsigned long long *Wc, const float *h,
                                           const OrdT *ord, int n, int nw, int q, int t, int tp, int tn, uint32_t rw,
                                           float B, float T4, int lane, const SpinPipe &pp) {
    const int pos = (q << 5) | lane, first = q << 5;
    const bool valid = pos < n;
    const int i = !valid ? 0 : (ORD ? (int)ord[pos] : pos);
    const float u = u24(rw), lim = accept_limit(u), eps = accept_margin(T4), hi = h[i];
    float gk = gt[i];
    // In qanneal's order the worldline words of the block's spins show the state
    // before this sweep in the bits of slices t and tn (slice tn flips a spin
    // only after slice t has decided it), except slice 0's for the last slice.
    const unsigned long long w0 = Wc[i];
    const uint32_t sb = (uint32_t)(w0 >> t) & 1u;
    const uint32_t ups = __ballot_sync(FULL, sb != 0u);
    uint32_t nb = __ballot_sync(FULL, ((w0 >> tn) & 1ull) != 0ull);
    auto bits_of = [&](int x, unsigned long long v, int d) {  // slice x's new bits of the block, d of them decided
        return d > 32 ? pp.pbits[x * nw + q] : (uint32_t)(v >> 32);
    };
    if (ORD && t > 0 && tn == 0) {
        const unsigned long long v = spin_wait(pp, 0, first + 32, lane);
        nb = bits_of(0, v, (int)(uint32_t)v - first);
    }
    const int dn = (int)(((nb >> lane) & 1u) ^ sb);
    // Trotter term and limit with slice tp's bit equal to s / differing from it
    const float troE = __fmul_rn(__int2float_rn(1 - dn), T4), troN = __fmul_rn(__int2float_rn(-dn), T4);
    const float limE = __fadd_rn(lim, troE), limN = __fadd_rn(lim, troN);
    uint32_t pend = n - first >= 32 ? FULL : (1u << (n - first)) - 1u;
    // lanes whose bit in slice tp is known, and whether it differs from s
    uint32_t known = FULL, diff = 0u;
    auto learn = [&](unsigned long long v) {
        const int d = (int)(uint32_t)v - first;
        known = d >= 32 ? FULL : (d > 0 ? (1u << d) - 1u : 0u);
        diff = bits_of(tp, v, d) ^ ups;
    };
    if (ORD && t > 0)
        learn(ld_acquire_cta64(pp.prog + tp));
    else
        diff = __ballot_sync(FULL, ((w0 >> tp) & 1ull) != 0ull) ^ ups;
    auto publish = [&](int count, uint32_t F) {
        return (unsigned long long)(uint32_t)(first + count) | ((unsigned long long)(ups ^ F) << 32);
    };
    auto coupling = [&](int j) {
        // zero diagonal: lane j's own field stays
        return __ldg(J + (size_t)__shfl_sync(FULL, i, j) * ld + i);
    };
    uint32_t F = 0;
    int jn = -1;  // the likely next flip, its couplings loaded ahead
    float jvn = 0.0f;
    for (bool more = true; more;) {
        const float xs = __fmul_rn(signed_by_bit(__fadd_rn(hi, gk), sb), B);
        uint32_t mE = __ballot_sync(FULL, xs >= limE), mN = __ballot_sync(FULL, xs >= limN);
        if (__ballot_sync(FULL, !(fminf(fabsf(xs - limE), fabsf(xs - limN)) > eps)) & pend) {
            mE = __ballot_sync(FULL, metropolis_nb24(__fsub_rn(xs, troE), u));
            mN = __ballot_sync(FULL, metropolis_nb24(__fsub_rn(xs, troN), u));
        }
        for (;;) {
            const uint32_t m = ((mE & ~(known & diff)) | (mN & (~known | diff))) & pend;
            more = m != 0u;
            if (!more) break;
            const int j = __ffs(m) - 1;
            if (ORD && !((known >> j) & 1u)) {
                // lane j may flip, depending on a bit slice tp has yet to decide;
                // the lanes before it are rejected
                pend &= ~0u << j;
                if (j > 0) st_relaxed_cta64(pp.prog + t, publish(j, F));  // (j = 0: nothing new)
                learn(spin_wait(pp, tp, first + j + 1, lane));
                continue;
            }
            F |= 1u << j;
            pend = j == 31 ? 0u : pend & (~0u << (j + 1));
            const float jv = j == jn ? jvn : coupling(j);
            if (ORD) st_relaxed_cta64(pp.prog + t, publish(j + 1, F));
            const uint32_t m2 = m & pend;
            jn = m2 ? __ffs(m2) - 1 : j;
            jvn = coupling(jn);
            gk = __fmaf_rn((ups >> j) & 1u ? -2.0f : 2.0f, jv, gk);
            break;
        }
    }
    if (ORD) {
        // the word carries the block's bits until one of the next block
        // replaces it; pbits is in place by then
        st_relaxed_cta64(pp.prog + t, publish(32, F));
        pp.pbits[t * nw + q] = ups ^ F;
        __threadfence_block();
    }
    if ((F >> lane) & 1u) atomicXor(reinterpret_cast<uint32_t *>(Wc + i) + (t >> 5), 1u << (t & 31));
    if (F) dense_update<WIDE>(J, ld, gt, F, i, ups, lane);
    return __popc(F);
}

// Slices t0, t0 + dt, ... < t1 of one slice sweep, one warp; the number of
// flips.  cell: the ring's first RNG cell.
template <bool ORD, bool WIDE>
__device__ __noinline__ int dense_sweep(const float *J, uint32_t ord, unsigned long long *err, int n, int NP,
                                        int t0, int t1, int dt, float B, float T4, uint64_t key, uint32_t cell,
                                        uint32_t sigma, uint32_t tag) {
    const int lane = threadIdx.x & 31, nw = (n + 31) >> 5, ld = dense_ld(n);
    const DenseLay L = dense_layout(NP, n, ORD);
    const SpinPipe pp{dsm<unsigned long long>(L.prog), dsm<uint32_t>(L.pbits), dsm<int>(L.abortf), err};
    int flips = 0;
    for (int t = t0; t < t1; t += dt) {
        const int tp = t == 0 ? NP - 1 : t - 1, tn = t + 1 == NP ? 0 : t + 1;
        U4 r{0, 0, 0, 0};
#pragma unroll 1
        for (int q = 0; q < nw; ++q) {
            if ((q & 3) == 0) r = philox((uint32_t)(((q >> 2) << 5) | lane), cell + (uint32_t)t, sigma, tag, key);
            flips += dense_block<ORD, WIDE>(J, ld, dsm<float>(L.G) + t * ld, dsm<unsigned long long>(L.W),
                                            dsm<float>(L.h), dsm<OrdT>(ord), n, nw, q, t, tp, tn, pick(r, q & 3), B,
                                            T4, lane, pp);
        }
    }
    return flips;
}

// One worldline sweep, whole CTA of W warps (ends with a barrier); the number
// of moves accepted.
template <bool ORD, bool WIDE>
__device__ __noinline__ int dense_worldlines(const float *J, uint32_t ordo, int n, int NP, float B,
                                             uint64_t key, uint32_t slot, uint32_t sigma) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int nw = (n + 31) >> 5, n32 = nw * 32, ld = dense_ld(n);
    const DenseLay L = dense_layout(NP, n, ORD);
    float *G = dsm<float>(L.G), *uw = dsm<float>(L.uw), *gb = dsm<float>(L.gb);
    unsigned long long *Wc = dsm<unsigned long long>(L.W);
    uint32_t *mask = dsm<uint32_t>(L.mask);
    const unsigned long long pmask = NP == 64 ? ~0ull : ((1ull << NP) - 1ull);
    for (int x = threadIdx.x; x < n32; x += blockDim.x)
        if (((x >> 5) & 3) == 0) {  // positions q*32 + lane .. + 96: one Philox call
            const U4 r = philox((uint32_t)(((x >> 7) << 5) | lane), slot, sigma, DOM_WORLD, key);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (x + 32 * k < n32) uw[x + 32 * k] = u24(pick(r, k));
        }
    __syncthreads();
    int moves = 0, look = W;  // blocks of a round: two after one with moves, else all warps'
    uint32_t *mk = mask;
    for (int q0 = 0; q0 < nw;) {
        // this round: warp w evaluates block q0 + w on the current state
        const int q = warp < look ? q0 + warp : nw, pos = (q << 5) | lane;
        const bool valid = q < nw && pos < n;
        const int i = !valid ? 0 : (ORD ? (int)dsm<OrdT>(ordo)[pos] : pos);
        const unsigned long long wi = Wc[i];
        const float hi = dsm<float>(L.h)[i], u = valid ? uw[pos] : 0.0f;
        auto accept = [&](double Gt) {
            const int sh = 2 * __popcll(wi) - NP;
            const float x = __double2float_rn(__dadd_rn(__dmul_rn((double)hi, (double)sh), Gt));
            return valid & metropolis_nb24(__fmul_rn(x, B), u);
        };
        uint32_t m = 0;
        if (q < nw) {
            double Gt = 0.0;
#pragma unroll 8
            for (int t = 0; t < NP; ++t)
                Gt = __dadd_rn(Gt, (double)signed_by_bit(G[t * ld + i], (uint32_t)(wi >> t) & 1u));
            m = __ballot_sync(FULL, accept(Gt));
        }
        if (lane == 0) mk[warp] = m;
        __syncthreads();
        const uint32_t with = __ballot_sync(FULL, lane < W && mk[lane] != 0u);
        mk = mk == mask ? mask + 32 : mask;
        if (!with) {
            q0 += look;
            look = W;
            continue;
        }
        look = min(2, W);
        const int ws = __ffs(with) - 1;
        if (warp == ws) {
            // resolve the block in position order on a copy of its fields
#pragma unroll 8
            for (int t = 0; t < NP; ++t) gb[t * 32 + lane] = G[t * ld + i];
            uint32_t F = 0;
            do {
                const int j = __ffs(m) - 1;
                F |= 1u << j;
                const int ij = __shfl_sync(FULL, i, j);
                const unsigned long long wj = __shfl_sync(FULL, wi, j);
                const float jv = J[(size_t)ij * ld + i];
                double Gt = 0.0;
#pragma unroll 8
                for (int t = 0; t < NP; ++t) {
                    const float g = __fmaf_rn((wj >> t) & 1ull ? -2.0f : 2.0f, jv, gb[t * 32 + lane]);
                    gb[t * 32 + lane] = g;
                    Gt = __dadd_rn(Gt, (double)signed_by_bit(g, (uint32_t)(wi >> t) & 1u));
                }
                const uint32_t later = j == 31 ? 0u : (FULL << (j + 1));
                m = __ballot_sync(FULL, accept(Gt)) & later;
            } while (m);
            dsm<unsigned long long>(L.wold)[lane] = wi;
            dsm<int>(L.wsp)[lane] = i;
            if (lane == 0) dsm<int>(L.flag)[1] = (int)F;
        }
        __syncthreads();
        // every slice: flip the block's flipped spins and update its fields
        const uint32_t F = (uint32_t)dsm<int>(L.flag)[1];
        const int isp = dsm<int>(L.wsp)[lane];
        const unsigned long long wo = dsm<unsigned long long>(L.wold)[lane];
        for (int t = warp; t < NP; t += W)
            dense_update<WIDE>(J, ld, G + t * ld, F, isp, __ballot_sync(FULL, ((wo >> t) & 1ull) != 0ull), lane);
        if (warp == 0 && ((F >> lane) & 1u)) Wc[isp] = wo ^ pmask;
        moves += __popc(F);
        __syncthreads();
        q0 += ws + 1;
    }
    return moves;
}


// ORD: qanneal's update order.
template <bool ORD, bool WIDE>
__global__ void __launch_bounds__(512, 1) ring_dense_kernel(RingParams p) {
    const RingDev R = p.rings[blockIdx.x];
    const ProbDev *Pd = p.probs + R.prob;
    const int NP = p.P, W = p.W, n = Pd->n, nw = Pd->nw, n32 = nw * 32, ld = dense_ld(n);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *J = Pd->J32;
    const DenseLay L = dense_layout(NP, n, ORD);
    float *G = dsm<float>(L.G), *h = dsm<float>(L.h);
    unsigned long long *Wc = dsm<unsigned long long>(L.W);
    double *cellE = dsm<double>(L.cellE);
    int *wpart = dsm<int>(L.part), *flag = dsm<int>(L.flag);
    if (ORD && threadIdx.x == 0) *dsm<int>(L.abortf) = 0;

    float *Gg = p.fields + R.field_off;
    for (int t = warp; t < NP; t += W)
        for (int m = lane; m < ld; m += 32) G[t * ld + m] = m < n ? Gg[(long long)t * n + m] : 0.0f;
    for (int i = threadIdx.x; i < n32; i += blockDim.x) {
        h[i] = i < n ? Pd->h32[i] : 0.0f;
        unsigned long long wc = 0;
        if (i < n)
#pragma unroll 1
            for (int t = 0; t < NP; ++t)
                wc |= (unsigned long long)((p.spins[R.spin_off + t * nw + (i >> 5)] >> (i & 31)) & 1u) << t;
        Wc[i] = wc;
    }
    __syncthreads();

    const unsigned long long pmask = NP == 64 ? ~0ull : ((1ull << NP) - 1ull);
    const int slot = p.slot ? p.slot[blockIdx.x] : R.k;
    OrderFeed feed = feed_open(ORD ? dsm<OrdT>(L.ord0) : nullptr, ORD ? dsm<OrdT>(L.ord1) : nullptr,
                               ORD ? p.ordg + blockIdx.x * p.ord_ring : nullptr, p.ord_stride, n,
                               ORD ? (p.step1 - p.step0) * p.ord_per_step : 0);
    unsigned long long att_s = 0, acc_s = 0, att_w = 0, acc_w = 0;
    double bestE = p.best_E[blockIdx.x];
    int bestStep = p.best_step[blockIdx.x];
    // sum over the CTA's spins of f(worldline word); valid on thread 0 after the barrier
    auto spin_total = [&](auto f) {
        int s = 0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) s += f(Wc[i]);
        s = warp_sum_i(s);
        if (lane == 0) wpart[warp] = s;
        __syncthreads();
        long long tot = 0;
        if (threadIdx.x == 0)
            for (int w = 0; w < W; ++w) tot += wpart[w];
        return tot;
    };
    // imaginary-time bonds of one worldline: P - 2 (slices that differ from the next)
    auto bonds = [&](unsigned long long w) {
        return NP - 2 * __popcll((w ^ ((w >> 1) | ((w & 1ull) << (NP - 1)))) & pmask);
    };

    for (int step = p.step0 - (p.init_scan ? 1 : 0); step < p.step1; ++step) {
        // step -1 (init_scan) only scores the starting state
        const int spb = step >= 0 ? p.spb : 0, wls = step >= 0 ? p.wls : 0;
        const int si_tab = R.sched + (p.per_slot_sched ? slot + max(step, 0) * p.slot_step : max(step, 0));
        const float B = p.B[si_tab], T4 = p.T4[si_tab];
        for (int sw = 0; sw < spb; ++sw) {
            const uint32_t sigma = (uint32_t)(step * p.spb + sw), tag = p.slice_tag | R.tag_extra;
            uint32_t ord = 0;
            if (ORD) {
                for (int t = threadIdx.x; t < NP; t += blockDim.x) dsm<unsigned long long>(L.prog)[t] = 0ull;
                ord = (uint32_t)(reinterpret_cast<const unsigned char *>(feed_take(feed)) - dense_sm);
            }
            if (ORD) {
                acc_s += (unsigned long long)dense_sweep<true, WIDE>(J, ord, p.counters + 4, n, NP, warp, NP, W, B, T4,
                                                                     R.key, (uint32_t)(slot * NP), sigma, tag);
                __syncthreads();
            } else {
                for (int ph = 0; ph < 3; ++ph) {
                    const int cnt = phase_count(NP, ph), b = phase_slice(NP, ph, 0);
                    acc_s += (unsigned long long)dense_sweep<false, WIDE>(J, 0, nullptr, n, NP, b + 2 * warp,
                                                                          b + 2 * cnt, 2 * W, B, T4, R.key,
                                                                          (uint32_t)(slot * NP), sigma, tag);
                    if (cnt) __syncthreads();
                }
            }
            if (threadIdx.x == 0) att_s += (unsigned long long)NP * (unsigned long long)n;
            if (p.mag) {
                const long long up = spin_total([&](unsigned long long w) { return __popcll(w); });
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
            const uint32_t ord =
                ORD ? (uint32_t)(reinterpret_cast<const unsigned char *>(feed_take(feed)) - dense_sm) : 0;
            const int mv = dense_worldlines<ORD, WIDE>(J, ord, n, NP, B, R.key, (uint32_t)slot, sigma);
            if (threadIdx.x == 0) {
                att_w += (unsigned long long)n;
                acc_w += (unsigned long long)mv;
            }
            __syncthreads();
        }
        // ---- step end: slice energies E = c + (sum s h + (sum s g)/2), ring sum, best
        for (int t = warp; t < NP; t += W) {
            double ph = 0.0, pg = 0.0;
#pragma unroll 1
            for (int i = lane; i < n; i += 32) {
                const uint32_t up = (uint32_t)(Wc[i] >> t) & 1u;
                ph = __dadd_rn(ph, (double)signed_by_bit(h[i], up));
                pg = __dadd_rn(pg, (double)signed_by_bit(G[t * ld + i], up));
            }
            ph = warp_sum_d(ph);
            pg = warp_sum_d(pg);
            if (lane == 0) cellE[t] = __dadd_rn(Pd->c, __dadd_rn(ph, __dmul_rn(0.5, pg)));
        }
        const long long bsum = p.ring_bond ? spin_total(bonds) : 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            double sum = 0.0, emin = __longlong_as_double(0x7ff0000000000000LL);
            int tmin = 0;
#pragma unroll 1
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
                const unsigned long long w = Wc[(q << 5) | lane];
                const uint32_t bb = __ballot_sync(FULL, tb >= 0 && ((w >> tb) & 1ull));
                const uint32_t bf = __ballot_sync(FULL, ((w >> tl) & 1ull) != 0ull);
                if (lane == 0) {
                    if (tb >= 0) p.best_bits[(long long)blockIdx.x * p.nw_max + q] = bb;
                    if (fin) p.final_bits[(long long)blockIdx.x * p.nw_max + q] = bf;
                }
            }
        __syncthreads();
    }
    for (int q = warp; q < nw; q += W) {
        const unsigned long long w = Wc[(q << 5) | lane];
#pragma unroll 1
        for (int t = 0; t < NP; ++t) {
            const uint32_t b = __ballot_sync(FULL, ((w >> t) & 1ull) != 0ull);
            if (lane == 0) p.spins[R.spin_off + t * nw + q] = b;
        }
    }
    for (int t = warp; t < NP; t += W)
        for (int m = lane; m < n; m += 32) Gg[(long long)t * n + m] = G[t * ld + m];
    if (lane == 0) {
        atomicAdd(p.counters + 0, att_s);
        atomicAdd(p.counters + 1, acc_s);
    }
    if (threadIdx.x == 0) {
        atomicAdd(p.counters + 2, att_w);
        atomicAdd(p.counters + 3, acc_w);
        p.best_E[blockIdx.x] = bestE;
        p.best_step[blockIdx.x] = bestStep;
    }
}

}  // namespace qa
