// qa_hubo.cuh -- Trotter-ring sweep kernel for higher-order models whose terms
// have at most four spins.
//
// Same replay semantics as ring_kernel<K_HUBO>.  What bounds this path is the
// chain of an accepted flip: its field updates, and the decisions after it.
//  * a flip's updates are chunks of up to 32 records (ProbDev::hub_rec), one
//    coalesced load for the warp, the first asked for while the flip before is
//    applied;
//  * after a flip only lanes whose field it changed decide again (the inverse
//    order tells which of the updated spins sit in the block);
//  * worldline moves: a warp evaluates a block of 32 positions, the moves before
//    the first lane that one of them changes are applied to all slices together,
//    and the evaluation resumes at that lane;
//  * the energy scan takes a term's sign in every slice from the xor of its
//    spins' worldline words.
// n = 1024, P = 16, 128 reads, 60 steps: slice sweeps alone 16.2 -> 8.8 ms, with
// one worldline sweep a step 33.8 -> 17.3 ms.  What is left is about 150
// instructions a flip at 1.6 a cycle, and in the worldline sweeps the barriers of
// a round per block.  Not kept: the chunks of all lanes that will flip prefetched
// ahead of the wait for the previous slice (8.8 -> 8.9 ms).
#pragma once
#include "qa_slab.cuh"

namespace qa {

struct HuboLay {
    uint32_t G, S, W, h, uw, inv, ord0, ord1, prog, abortf, cellE, part, mask, wsp, flag, total;
};
__host__ __device__ inline HuboLay hubo_layout(int P, int n, bool ref_order) {
    const int nw = (n + 31) / 32, n32 = nw * 32, ld = dense_ld(n);
    HuboLay L{};
    uint32_t o = 0;
    auto take = [&](size_t bytes) {
        const uint32_t at = o;
        o += (uint32_t)align_up(bytes, 16);
        return at;
    };
    L.G = take((size_t)P * ld * 4);
    L.S = take((size_t)P * nw * 4);
    L.W = take((size_t)n32 * 8);     // worldline words, built for the energy scan
    L.h = take((size_t)n32 * 4);
    L.uw = take((size_t)n32 * 4);    // worldline uniforms
    L.cellE = take((size_t)P * 8);
    L.part = take(32 * 4);
    L.mask = take(2 * 32 * 4);       // move masks of a worldline round, two rounds
    L.wsp = take(32 * 4);            // a worldline batch's spins
    L.flag = take(16);               // [0]: best slice, [1]: batch, [2]: first lane to decide again, [3]: lowest slice
    L.prog = take((size_t)P * 4);
    L.abortf = take(4);
    if (ref_order) {
        L.inv = take((size_t)n32 * 2);
        L.ord0 = take(ord_row_bytes(n32));
        L.ord1 = take(ord_row_bytes(n32));
    }
    L.total = o;
    return L;
}
__host__ __device__ inline size_t hubo_smem_bytes(int P, int n, bool ref_order) {
    return hubo_layout(P, n, ref_order).total;
}

// Warps of a ring (at most 16: up to 126 registers a thread), 0 for ring_kernel.  smem: a
// ring's shared memory, cap: an SM's.
// qanneal's order: w warps take P / w slices each, behind one another; more rings an SM
// against a longer share, by waves of rings times P / w + 2.6 (fits n = 24 .. 200, P = 1
// .. 64, 148 .. 3000 rings within 1% of the best w on average: P = 16, n = 64, 450 rings 4
// warps 1.9 times as fast as 16).
// Checkerboard: where the slices of a phase fit on the SMs, 16 warps each, a warp for
// each (1.2 to 1.5 times ring_kernel); where they do not, ring_kernel with its 64
// registers is faster at every n (n = 200: P = 16, 600 rings 0.90, P = 24, 200 rings
// 0.86, P = 64, 100 rings 0.93 of its speed here; but P = 16, 200 rings 1.35).
inline int hubo_warps(int P, int rings, int sms, bool ref_order, size_t smem, size_t cap) {
    const int most = std::min(P, 16), phase = (P + 1) / 2;
    if (!ref_order || P == 1) {
        if (rings > sms * (16 / phase)) return 0;
        return rings > sms ? std::min(most, phase) : most;
    }
    const int fit = std::max(1, (int)(cap / smem));
    int best = most;
    double cost = 0.0;
    for (int w = most; w >= 1; --w) {
        const int per_sm = std::min(16 / w, fit);
        const double c = std::ceil((double)rings / ((double)per_sm * sms)) * ((double)P / w + 2.6);
        if (w == most || c < cost) {
            best = w;
            cost = c;
        }
    }
    return best;
}

// The field updates of a flip (ProbDev::hub_spin, hub_size, hub_rec).
struct HubRows {
    const uint4 *spin;
    const uint32_t *size;
    const int4 *rec;
};

// Lane j's entry in all lanes, and this lane's record of its first chunk.
__device__ __forceinline__ uint4 hub_of(const uint4 &hs, int j) {
    return make_uint4(__shfl_sync(FULL, hs.x, j), __shfl_sync(FULL, hs.y, j), __shfl_sync(FULL, hs.z, j),
                      __shfl_sync(FULL, hs.w, j));
}
__device__ __forceinline__ int4 hub_first(const HubRows &hr, uint32_t at, uint32_t sizes, int lane) {
    return (uint32_t)lane < (sizes & 255u) ? __ldg(hr.rec + at + lane) : make_int4(-1, -1, -1, 0);
}

// The lanes of block q (positions) that hold record r's target.
template <bool ORD>
__device__ __forceinline__ uint32_t hubo_touch(const int4 &r, const OrdT *inv, int q) {
    if (r.x < 0) return 0u;
    const int p = ORD ? (int)inv[r.x] : r.x;
    return (p >> 5) == q ? 1u << (p & 31) : 0u;
}

// Slices t0, t0 + dt, .. < t1 of one slice sweep, one warp; the number of flips.
template <bool ORD>
__device__ __noinline__ int hubo_sweep(const HubRows hr, uint32_t ordo, unsigned long long *err, int n,
                                       int NP, int t0, int t1, int dt, float B, float T4, uint64_t key, uint32_t cell,
                                       uint32_t sigma, uint32_t tag) {
    const int lane = threadIdx.x & 31, nw = (n + 31) >> 5, ld = dense_ld(n);
    const HuboLay L = hubo_layout(NP, n, ORD);
    uint32_t *S = dsm<uint32_t>(L.S);
    const float *h = dsm<float>(L.h);
    const OrdT *ord = dsm<OrdT>(ordo), *inv = dsm<OrdT>(L.inv);
    int *prog = dsm<int>(L.prog), *abortf = dsm<int>(L.abortf);
    const float eps = accept_margin(T4);
    int flips = 0;
    for (int t = t0; t < t1; t += dt) {
        const int tp = t == 0 ? NP - 1 : t - 1, tn = t + 1 == NP ? 0 : t + 1;
        uint32_t *St = S + t * nw;
        const uint32_t *Sp = S + tp * nw, *Sn = S + tn * nw;
        float *gt = dsm<float>(L.G) + t * ld;
        U4 r{0, 0, 0, 0};
#pragma unroll 1
        for (int q = 0; q < nw; ++q) {
            if ((q & 3) == 0) r = philox((uint32_t)(((q >> 2) << 5) | lane), cell + (uint32_t)t, sigma, tag, key);
            const int pos = (q << 5) | lane;
            const bool valid = pos < n;
            const int i = valid ? (ORD ? (int)ord[pos] : pos) : 0;
            const uint4 hs = __ldg(hr.spin + i);  // the spin's chunks
            const float u = u24(pick(r, q & 3)), hi = h[i];
            const uint32_t sb = (St[i >> 5] >> (i & 31)) & 1u;
            const float Bs = sb ? B : -B, lim0 = accept_limit(u);
            float gi = gt[i];
            if (ORD && t > 0) {
                slab_wait(prog + t - 1, q + 1, abortf, err, lane);
                if (tn == 0) slab_wait(prog, q + 1, abortf, err, lane);
            }
            const int d = (int)(((Sp[i >> 5] >> (i & 31)) & 1u) ^ sb) + (int)(((Sn[i >> 5] >> (i & 31)) & 1u) ^ sb);
            const float tro = __fmul_rn(__int2float_rn(1 - d), T4), lim = lim0 + tro;
            auto decide = [&]() {
                const float xs = __fmul_rn(__fadd_rn(hi, gi), Bs);
                bool ok = xs >= lim;
                if (__any_sync(FULL, !(fabsf(xs - lim) > eps))) ok = metropolis_nb24(__fsub_rn(xs, tro), u);
                return __ballot_sync(FULL, valid & ok);
            };
            uint32_t m = decide();
            if (m) {
                uint32_t at, sizes, atn, sizesn;  // records and chunk sizes of spin j, of the next
                auto chunk = [&](int j, uint32_t &x, uint32_t &y) {
                    x = __shfl_sync(FULL, hs.x, j);
                    y = __shfl_sync(FULL, hs.y, j);
                    return hub_first(hr, x, y, lane);
                };
                int j = __ffs(m) - 1;
                int4 rec = chunk(j, at, sizes);
                while (true) {
                    const uint32_t pend = j == 31 ? 0u : ~((2u << j) - 1u);
                    const int jj = __shfl_sync(FULL, i, j);
                    const int sj = __shfl_sync(FULL, sb, j) ? -1 : 1;  // the new spin
                    if (lane == 0) St[jj >> 5] ^= 1u << (jj & 31);
                    ++flips;
                    const int jn = (m & pend) ? __ffs(m & pend) - 1 : j;  // the likely next flip
                    const int4 recn = chunk(jn, atn, sizesn);
                    __syncwarp();
                    hub_add(rec, gt, St, sj);
                    uint32_t touch = hubo_touch<ORD>(rec, inv, q);
                    auto further = [&](const int4 &x) {
                        hub_add(x, gt, St, sj);
                        touch |= hubo_touch<ORD>(x, inv, q);
                    };
                    // (chunks in order: a target's terms stay in order; one further
                    // chunk by itself: n = 226, P = 16, 50 rings, 81 sweeps 5.20 -> 4.88 ms)
                    if (sizes >= 65536u) {
                        hub_chunks(make_uint4(at, sizes, __shfl_sync(FULL, hs.z, j), __shfl_sync(FULL, hs.w, j)), hr.size,
                                   hr.rec, lane, further);
                    } else if (sizes >= 256u) {
                        const int4 x = hub_first(hr, at + (sizes & 255u), sizes >> 8, lane);
                        __syncwarp();
                        further(x);
                    }
                    touch = __reduce_or_sync(FULL, touch) & pend;
                    __syncwarp();
                    if (touch) {
                        if ((touch >> lane) & 1u) gi = gt[i];
                        m = (m & ~touch) | (decide() & touch);
                    }
                    if (!(m & pend)) break;
                    j = __ffs(m & pend) - 1;
                    if (j == jn) {
                        rec = recn;
                        at = atn;
                        sizes = sizesn;
                    } else {
                        rec = chunk(j, at, sizes);
                    }
                }
            }
            if (ORD) {
                __threadfence_block();
                __syncwarp();
                if (lane == 0) st_release_cta(prog + t, q + 1);
            }
        }
    }
    return flips;
}

// One worldline sweep, whole CTA (ends with a barrier); the number of moves.
template <bool ORD>
__device__ __noinline__ int hubo_worldlines(const HubRows hr, uint32_t ordo, int n, int NP, float B,
                                            uint64_t key, uint32_t slot, uint32_t sigma) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int nw = (n + 31) >> 5, n32 = nw * 32, ld = dense_ld(n);
    const HuboLay L = hubo_layout(NP, n, ORD);
    uint32_t *S = dsm<uint32_t>(L.S), *mask = dsm<uint32_t>(L.mask);
    float *G = dsm<float>(L.G), *uw = dsm<float>(L.uw);
    const OrdT *ord = dsm<OrdT>(ordo), *inv = dsm<OrdT>(L.inv);
    int *flag = dsm<int>(L.flag), *wsp = dsm<int>(L.wsp);
    for (int x = threadIdx.x; x < n32; x += blockDim.x)
        if (((x >> 5) & 3) == 0) {  // positions q*32 + lane .. + 96: one Philox call
            const U4 r = philox((uint32_t)(((x >> 7) << 5) | lane), slot, sigma, DOM_WORLD, key);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (x + 32 * k < n32) uw[x + 32 * k] = u24(pick(r, k));
        }
    __syncthreads();
    int moves = 0, first = 0;  // lanes of block q0 before `first` are done
    int look = W;              // blocks of a round: two after one with moves, else all warps'
    uint32_t *mk = mask;
    for (int q0 = 0; q0 < nw;) {
        // this round: warp w evaluates block q0 + w on the current state
        const int q = warp < look ? q0 + warp : nw, pos = (q << 5) | lane;
        const bool valid = q < nw && pos < n && (warp > 0 || lane >= first);
        const int i = valid ? (ORD ? (int)ord[pos] : pos) : 0;
        uint32_t m = 0;
        if (q < nw) {
            double Gt = 0.0;
            int sh = 0;
            const uint32_t *Sw = S + (i >> 5);
#pragma unroll 4
            for (int t = 0; t < NP; ++t) {
                const uint32_t up = (Sw[t * nw] >> (i & 31)) & 1u;
                sh += up ? 1 : -1;
                Gt = __dadd_rn(Gt, (double)signed_by_bit(G[t * ld + i], up));
            }
            const float x = __double2float_rn(__dadd_rn(__dmul_rn((double)dsm<float>(L.h)[i], (double)sh), Gt));
            m = __ballot_sync(FULL, valid & metropolis_nb24(__fmul_rn(x, B), valid ? uw[pos] : 0.0f));
        }
        if (lane == 0) mk[warp] = m;
        __syncthreads();
        const uint32_t with = __ballot_sync(FULL, lane < W && mk[lane] != 0u);
        mk = mk == mask ? mask + 32 : mask;
        if (!with) {
            q0 += look;
            look = W;
            first = 0;
            continue;
        }
        look = min(2, W);
        const int ws = __ffs(with) - 1;
        if (warp == ws) {
            // the moves before the first lane that one of them changes
            const uint4 hs = __ldg(hr.spin + i);
            uint32_t F = 0, T = 0;
            for (uint32_t mm = m; mm; mm &= mm - 1u) {
                const int j = __ffs(mm) - 1;
                if (T && __ffs(T) - 1 <= j) break;
                F |= 1u << j;
                const uint4 hj = hub_of(hs, j);
                uint32_t touch = hubo_touch<ORD>(hub_first(hr, hj.x, hj.y, lane), inv, q);
                hub_chunks(hj, hr.size, hr.rec, lane, [&](const int4 &x) { touch |= hubo_touch<ORD>(x, inv, q); });
                T |= __reduce_or_sync(FULL, touch) & (j == 31 ? 0u : ~((2u << j) - 1u));
            }
            wsp[lane] = i;
            if (lane == 0) {
                flag[1] = (int)F;
                flag[2] = T ? __ffs(T) - 1 : 32;
            }
        }
        __syncthreads();
        const uint32_t F = (uint32_t)flag[1];
        const int again = flag[2], isp = wsp[lane];
        const uint4 hs = __ldg(hr.spin + isp);
        for (int t = warp; t < NP; t += W) {
            uint32_t *St = S + t * nw;
            for (uint32_t f = F; f; f &= f - 1u) {
                const int j = __ffs(f) - 1, jj = __shfl_sync(FULL, isp, j);
                const uint4 hj = hub_of(hs, j);
                const int4 rec = hub_first(hr, hj.x, hj.y, lane);
                const int sj = -spin_of(St, jj);
                __syncwarp();
                if (lane == 0) St[jj >> 5] ^= 1u << (jj & 31);
                __syncwarp();
                hub_add(rec, G + t * ld, St, sj);
                hub_chunks(hj, hr.size, hr.rec, lane, [&](const int4 &x) { hub_add(x, G + t * ld, St, sj); });
                __syncwarp();
            }
        }
        moves += __popc(F);
        __syncthreads();
        q0 += ws;
        first = again;
        if (again == 32) {
            ++q0;
            first = 0;
        }
    }
    return moves;
}

// ORD: qanneal's update order.
template <bool ORD>
__global__ void __launch_bounds__(512, 1) ring_hubo_kernel(RingParams p) {
    const RingDev R = p.rings[blockIdx.x];
    const ProbDev *Pd = p.probs + R.prob;
    const int NP = p.P, W = p.W, n = Pd->n, nw = Pd->nw, n32 = nw * 32, ld = dense_ld(n), T = Pd->T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const HubRows hr{Pd->hub_spin, Pd->hub_size, Pd->hub_rec};
    const HuboLay L = hubo_layout(NP, n, ORD);
    float *G = dsm<float>(L.G), *h = dsm<float>(L.h);
    uint32_t *S = dsm<uint32_t>(L.S);
    unsigned long long *Wc = dsm<unsigned long long>(L.W);
    double *cellE = dsm<double>(L.cellE);
    int *wpart = dsm<int>(L.part), *flag = dsm<int>(L.flag);
    if (threadIdx.x == 0) *dsm<int>(L.abortf) = 0;
    float *Gg = p.fields + R.field_off;
    for (int t = warp; t < NP; t += W)
        for (int m = lane; m < n; m += 32) G[t * ld + m] = Gg[(long long)t * n + m];
    for (int idx = threadIdx.x; idx < NP * nw; idx += blockDim.x) S[idx] = p.spins[R.spin_off + idx];
    for (int i = threadIdx.x; i < n32; i += blockDim.x) h[i] = i < n ? Pd->h32[i] : 0.0f;
    __syncthreads();

    const int slot = p.slot ? p.slot[blockIdx.x] : R.k;
    OrderFeed feed = feed_open(ORD ? dsm<OrdT>(L.ord0) : nullptr, ORD ? dsm<OrdT>(L.ord1) : nullptr,
                               ORD ? p.ordg + blockIdx.x * p.ord_ring : nullptr, p.ord_stride, n,
                               ORD ? (p.step1 - p.step0) * p.ord_per_step : 0);
    unsigned long long att_s = 0, acc_s = 0, att_w = 0, acc_w = 0;
    double bestE = p.best_E[blockIdx.x];
    int bestStep = p.best_step[blockIdx.x];
    // a sweep's order and its inverse, clean progress; whole CTA
    auto begin_sweep = [&]() {
        uint32_t ord = 0;
        for (int t = threadIdx.x; t < NP; t += blockDim.x) dsm<int>(L.prog)[t] = 0;
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
            const uint32_t sigma = (uint32_t)(step * p.spb + sw), tag = p.slice_tag | R.tag_extra;
            const uint32_t ord = begin_sweep();
            if (ORD) {
                acc_s += (unsigned long long)hubo_sweep<true>(hr, ord, p.counters + 4, n, NP, warp, NP, W, B, T4,
                                                              R.key, (uint32_t)(slot * NP), sigma, tag);
                __syncthreads();
            } else {
                for (int ph = 0; ph < 3; ++ph) {
                    const int cnt = phase_count(NP, ph), b = phase_slice(NP, ph, 0);
                    acc_s += (unsigned long long)hubo_sweep<false>(hr, 0, nullptr, n, NP, b + 2 * warp,
                                                                   b + 2 * cnt, 2 * W, B, T4, R.key,
                                                                   (uint32_t)(slot * NP), sigma, tag);
                    if (cnt) __syncthreads();
                }
            }
            if (threadIdx.x == 0) att_s += (unsigned long long)NP * (unsigned long long)n;
            if (p.mag) {
                int ps = 0;
                for (int idx = threadIdx.x; idx < NP * nw; idx += blockDim.x) ps += __popc(S[idx]);
                ps = warp_sum_i(ps);
                if (lane == 0) wpart[warp] = ps;
                __syncthreads();
                if (threadIdx.x == 0) {
                    long long tot = 0;
                    for (int w = 0; w < W; ++w) tot += wpart[w];
                    p.mag[(long long)blockIdx.x * (p.steps_total * p.spb) + sigma] = (int)(2 * tot - (long long)NP * n);
                }
                __syncthreads();
            }
            if (p.bsamp) record_bond_sample(p, S, NP, nw, n, wpart, W, step, sw);
        }
        for (int sw = 0; sw < wls; ++sw) {
            const uint32_t sigma = (uint32_t)(step * p.wls + sw);
            const uint32_t ord = begin_sweep();
            const int mv = hubo_worldlines<ORD>(hr, ord, n, NP, B, R.key, (uint32_t)slot, sigma);
            if (threadIdx.x == 0) {
                att_w += (unsigned long long)n;
                acc_w += (unsigned long long)mv;
            }
            __syncthreads();
        }
        // ---- step end: slice energies E = c + (sum s h + sum_t J_t prod s), ring sum, best
        for (int i = threadIdx.x; i < n32; i += blockDim.x) {
            unsigned long long w = 0;
            for (int t = 0; t < NP; ++t) w |= (unsigned long long)((S[t * nw + (i >> 5)] >> (i & 31)) & 1u) << t;
            Wc[i] = ~w;  // down spins
        }
        __syncthreads();
        // slices t and t + 1 of a warp in one pass over the terms, each slice's
        // sums in cell_energy's order
        for (int t = 2 * warp; t < NP; t += 2 * W) {
            double ha = 0.0, hb = 0.0, ja = 0.0, jb = 0.0;
            for (int i = lane; i < n; i += 32) {
                const double hv = (double)h[i];
                const uint32_t w = (uint32_t)(Wc[i] >> t);
                ha = __dadd_rn(ha, neg_by_bit(hv, w, 0));
                hb = __dadd_rn(hb, neg_by_bit(hv, w, 1));
            }
            for (int k = lane; k < T; k += 32) {
                const int4 r = __ldg(Pd->trec + k);
                const double v = (double)__ldg(Pd->coef32 + k);
                unsigned long long w = Wc[r.x] ^ Wc[r.y];
                if (r.z >= 0) w ^= Wc[r.z];
                if (r.w >= 0) w ^= Wc[r.w];
                const uint32_t b = (uint32_t)(w >> t);
                ja = __dadd_rn(ja, neg_by_bit(v, b, 0));
                jb = __dadd_rn(jb, neg_by_bit(v, b, 1));
            }
            ha = warp_sum_d(ha);
            hb = warp_sum_d(hb);
            ja = warp_sum_d(ja);
            jb = warp_sum_d(jb);
            if (lane == 0) {
                cellE[t] = __dadd_rn(Pd->c, __dadd_rn(ha, ja));
                if (t + 1 < NP) cellE[t + 1] = __dadd_rn(Pd->c, __dadd_rn(hb, jb));
            }
        }
        const long long bsum = p.ring_bond ? ring_bond_total(S, NP, nw, n, wpart, W) : 0;
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
            for (int q = threadIdx.x; q < nw; q += blockDim.x)
                p.best_bits[(long long)blockIdx.x * p.nw_max + q] = S[tb * nw + q];
        }
        if (p.final_bits && step == p.steps_total - 1)
            for (int q = threadIdx.x; q < nw; q += blockDim.x)
                p.final_bits[(long long)blockIdx.x * p.nw_max + q] = S[tl * nw + q];
        __syncthreads();
    }
    for (int idx = threadIdx.x; idx < NP * nw; idx += blockDim.x) p.spins[R.spin_off + idx] = S[idx];
    for (int t = warp; t < NP; t += W)
        for (int m = lane; m < n; m += 32) Gg[(long long)t * n + m] = G[t * ld + m];
    if (lane == 0) atomicAdd(p.counters + 1, acc_s);
    if (threadIdx.x == 0) {
        atomicAdd(p.counters + 0, att_s);
        atomicAdd(p.counters + 2, att_w);
        atomicAdd(p.counters + 3, acc_w);
        p.best_E[blockIdx.x] = bestE;
        p.best_step[blockIdx.x] = bestStep;
    }
}

}  // namespace qa
