// The neighbour phase of LOGO_SEARCH_NEIGHBOUR(_OROPT) as one cooperative
// launch (sm_103a): the tour stays in global memory, one grid barrier closes
// each sweep and another each move.  Barrier waits are bounded (2 s of
// %globaltimer); a CTA that gives up sets kErrTimeout and leaves the loop, so
// the others give up too and the launch ends.
//
// A move costs the latency of its sweep, the gather of the tour and two barriers.
// A thread that walks a position's whole list leaves each SM with five warps and
// eight neighbours one after another; so the sweep drops the positions that cannot
// beat what is known (a bound from the last sweep's best candidates, evaluated
// anew where their cities are now) and gives every list entry of the others a
// thread of its own (from an NN tour with Or-opt, n = 25,000: 26 -> 16 us a move,
// n = 1,000: 25 -> 11; without, n = 25,000: 13 -> 10).
#include <algorithm>
#include <climits>

#include "grid_barrier.cuh"
#include "logo_device.cuh"
#include "logo_internal.h"
#include "neighbour_core.cuh"

namespace logo {

namespace {

constexpr unsigned long long kCoopWaitNs = 2000000000ull;
// Threads of the one CTA per SM: 512 (the Or-opt candidates' registers allow no
// more); for 2-opt candidates alone 1024 where 512 a CTA do not hold all positions
// (n = 100,000: 20 -> 16.5 us a move; n = 1,000: 7.9 us a move with 512, 8.7 with 1024).
constexpr int kCoopNT = 512, kCoopWideNT = 1024;
constexpr uint32_t kCoopLeast = 64;  // positions per CTA at least

// The five segments of which the city at a position is an end: (i, 1), (i, 2),
// (i, 3), (i-1, 2), (i-2, 3) as (first, length).
struct NbrBases {
    int b1, b2, b3, c2, c3;  // d(s-1, s+L) - e[s] - e[s+L], or INT_MAX
};

// The best candidate met and the positions (i, q) whose list entry it came from:
// lowest delta, ties to the 2-opt move (cls 0), then the lower Or-opt slot, then
// the lower positions.
struct NbrPick {
    uint32_t hi;  // biased delta, class; ~0: none
    uint64_t lo;
    uint32_t i, q;
    __device__ __forceinline__ void offer(uint64_t key, uint32_t cls, uint32_t at, uint32_t to) {
        if (key == kNoMove) return;
        const uint32_t h = (uint32_t)(key >> 42) << 3 | cls;
        const uint64_t l = key & ((1ull << 42) - 1);
        if (h < hi || (h == hi && l < lo)) {
            hi = h;
            lo = l;
            i = at;
            q = to;
        }
    }
    // the warp's best, in every lane
    __device__ __forceinline__ void reduce() {
        const uint32_t h = __reduce_min_sync(0xffffffffu, hi);
        const uint32_t a =
            __reduce_min_sync(0xffffffffu, hi == h ? (uint32_t)(lo >> 21) : 0xffffffffu);
        const bool tie = hi == h && (uint32_t)(lo >> 21) == a;
        const uint32_t b =
            __reduce_min_sync(0xffffffffu, tie ? (uint32_t)lo & 0x1FFFFFu : 0xffffffffu);
        const uint32_t who =
            __ffs(__ballot_sync(0xffffffffu, tie && ((uint32_t)lo & 0x1FFFFFu) == b)) - 1;
        hi = h;
        lo = __shfl_sync(0xffffffffu, lo, who);
        i = __shfl_sync(0xffffffffu, i, who);
        q = __shfl_sync(0xffffffffu, q, who);
    }
    __device__ __forceinline__ int bound() const {
        return hi == ~0u ? -1 : (int)(hi >> 3) - kKeyDeltaBias;
    }
};

// Position i's bases; returns what none of its candidates is below: a 2-opt pair
// is no better than -2 times either edge it removes, a segment's move no better
// than its base less the segment's own edges (triangle inequality; 8 covers the
// rounding).
template <bool OR>
__device__ __forceinline__ int nbr_bases(uint32_t i, const OrderedCity* Q, uint32_t n,
                                         NbrBases& s) {
    s.b1 = s.b2 = s.b3 = s.c2 = s.c3 = INT_MAX;
    const OrderedCity qi = ld_city(Q + i), qip = ld_city(Q + min(i + 1, n - 1));
    int low = -2 * max((int)qi.e, (int)qip.e);
    if (OR) {
        const OrderedCity qm3 = ld_city(Q + (i >= 3 ? i - 3 : 0));
        const OrderedCity qm2 = ld_city(Q + (i >= 2 ? i - 2 : 0));
        const OrderedCity qim = ld_city(Q + (i >= 1 ? i - 1 : 0));
        const OrderedCity qp2 = ld_city(Q + min(i + 2, n - 1));
        const OrderedCity qp3 = ld_city(Q + min(i + 3, n - 1));
        if (i >= 1 && i + 1 <= n - 1) {
            s.b1 = exact_dist(qim.x, qim.y, qip.x, qip.y) - (int)qi.e - (int)qip.e;
            low = min(low, s.b1);
        }
        if (i >= 1 && i + 2 <= n - 1) {
            s.b2 = exact_dist(qim.x, qim.y, qp2.x, qp2.y) - (int)qi.e - (int)qp2.e;
            low = min(low, s.b2 - (int)qip.e);
        }
        if (i >= 1 && i + 3 <= n - 1) {
            s.b3 = exact_dist(qim.x, qim.y, qp3.x, qp3.y) - (int)qi.e - (int)qp3.e;
            low = min(low, s.b3 - (int)qip.e - (int)qp2.e);
        }
        if (i >= 2 && i + 1 <= n - 1) {  // segment [i-1, i+1): s-1 = i-2, s+L = i+1
            s.c2 = exact_dist(qm2.x, qm2.y, qip.x, qip.y) - (int)qim.e - (int)qip.e;
            low = min(low, s.c2 - (int)qi.e);
        }
        if (i >= 3 && i + 1 <= n - 1) {  // segment [i-2, i+1): s-1 = i-3, s+L = i+1
            s.c3 = exact_dist(qm3.x, qm3.y, qip.x, qip.y) - (int)qm2.e - (int)qip.e;
            low = min(low, s.c3 - (int)qim.e - (int)qi.e);
        }
    }
    return low - 8;
}

// The candidates of one list entry, the city at position q in the list of the
// city at position i, as in nbr_position; Or-opt candidates above B are passed by.
template <bool OR>
__device__ __forceinline__ void nbr_entry(uint32_t i, uint32_t q, const OrderedCity* Q,
                                          uint32_t n, float M, int B, const NbrBases& s,
                                          NbrPick& pick) {
    uint64_t best = kNoMove;
    uint64_t bo[kOrSlots];
#pragma unroll
    for (int v = 0; v < kOrSlots; ++v) bo[v] = kNoMove;
    const OrderedCity qim = ld_city(Q + (i >= 1 ? i - 1 : 0)), qi = ld_city(Q + i),
                      qip = ld_city(Q + min(i + 1, n - 1));
    const OrderedCity pm = ld_city(Q + (q >= 1 ? q - 1 : 0)), p = ld_city(Q + q),
                      pp = ld_city(Q + min(q + 1, n - 1));
    nbr_pairs(i, q, n, qim, qi, qip, pm, p, pp, best);
    pick.offer(best, 0, i, q);
    if (!OR) return;
    const OrderedCity qm2 = ld_city(Q + (i >= 2 ? i - 2 : 0));
    const OrderedCity qp2 = ld_city(Q + min(i + 2, n - 1));
    const float m = M + (float)(B + 1);
    or_try<1, false>(i, q, n, qi, qi, s.b1, m, p, pp, bo);
    or_try<2, false>(i, q, n, qi, qip, s.b2, m, p, pp, bo);
    or_try<3, false>(i, q, n, qi, qp2, s.b3, m, p, pp, bo);
    if (q >= 1) {
        or_try<1, false>(i, q - 1, n, qi, qi, s.b1, m, pm, p, bo);
        or_try<2, true>(i, q - 1, n, qi, qip, s.b2, m, pm, p, bo);
        or_try<3, true>(i, q - 1, n, qi, qp2, s.b3, m, pm, p, bo);
    }
    if (i >= 2) {
        or_try<2, true>(i - 1, q, n, qim, qi, s.c2, m, p, pp, bo);
        if (q >= 1) or_try<2, false>(i - 1, q - 1, n, qim, qi, s.c2, m, pm, p, bo);
    }
    if (i >= 3) {
        or_try<3, true>(i - 2, q, n, qm2, qi, s.c3, m, p, pp, bo);
        if (q >= 1) or_try<3, false>(i - 2, q - 1, n, qm2, qi, s.c3, m, pm, p, bo);
    }
#pragma unroll
    for (int v = 0; v < kOrSlots; ++v) pick.offer(bo[v], 1 + v, i, q);
}

// Per move, the CTAs leave the best candidates of their positions, one grid
// barrier, every CTA picks the same move (the rule of apply_nbr_move_kernel) and
// gathers its share of the moved tour (Q, route, pos; buffers cur and cur ^ 1 as
// for the multi-kernel path), a second barrier, and the buffers swap.  DevState at
// the end is what the sweep and apply kernels leave after the same moves: moves,
// total_moves, sweeps and nbr_sweeps (one per sweep, the converging one included),
// converged, cur, the move log, kErrMoveLimit at max_moves, kErrBadKey on an
// out-of-range key.
template <bool OR, int NT>
__global__ void __launch_bounds__(NT, 1) coop_nbr_kernel(NbrLaunch L, CoopSync* cs) {
    constexpr int NW = NT / 32;
    constexpr NbrPick kNoPick{~0u, ~0ull, 0u, 0u};
    // positions in hand
    __shared__ uint32_t at[NT], city_of[NT];
    __shared__ int bases[OR ? 5 : 1][NT];
    __shared__ uint32_t taken[2];
    __shared__ NbrPick wbest[NW];
    __shared__ NbrPick best;
    __shared__ uint2 seeds[32];  // cities of entries of the lists (equal: none)
    __shared__ int bound;
    __shared__ bool ok_s;
    DevState* st = L.st;
    const uint32_t n = L.n, K = L.K;
    uint32_t cur = *(volatile unsigned int*)&st->cur;
    const unsigned long long max_moves = *(volatile unsigned long long*)&st->max_moves;
    unsigned long long moves = *(volatile unsigned long long*)&st->moves;
    const unsigned long long moves0 = moves;
    const bool start_done = *(volatile unsigned int*)&st->converged;
    GridBarrier barrier{&cs->arrived, st, &ok_s, kCoopWaitNs};
    if (threadIdx.x == 0) barrier.start(gridDim.x);
    uint32_t sweeps = 0;
    bool limit = false, bad = false, timeout = false;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // positions are dealt 32 at a time: those that can take part often lie together
    const uint32_t chunk = 32 * gridDim.x, share = (n + chunk - 1) / chunk * 32;
    if (threadIdx.x < 2) taken[threadIdx.x] = 0;
    if (threadIdx.x < 32) seeds[threadIdx.x] = make_uint2(0u, 0u);
    __syncthreads();
    for (uint32_t sw = 0; !start_done; ++sw) {
        const OrderedCity* Q = cur ? L.Q1 : L.Q0;
        const uint32_t* R = cur ? L.R1 : L.R0;
        NbrPick pick = kNoPick;
        if (warp == NW - 1) {
            // (the last warp: only of large tours it has positions of its own)
            const uint2 seed = seeds[lane];
            if (seed.x != seed.y) {
                const uint32_t i = min(ld_u32(L.pos + min(seed.x, n - 1)), n - 1);
                const uint32_t q = min(ld_u32(L.pos + min(seed.y, n - 1)), n - 1);
                NbrBases s;
                nbr_bases<OR>(i, Q, n, s);
                nbr_entry<OR>(i, q, Q, n, L.margin, -1, s, pick);
            }
            const int known = __reduce_min_sync(0xffffffffu, pick.bound());
            if (lane == 0) bound = known;
        }
        uint32_t turn = 0;
        for (uint32_t base = 0; base < share; base += NT, turn ^= 1u) {
            const uint32_t t0 = base + threadIdx.x, i = (t0 / 32 * gridDim.x + blockIdx.x) * 32 + lane;
            NbrBases s;
            const int low = t0 < share && i < n ? nbr_bases<OR>(i, Q, n, s) : INT_MAX;
            if (base == 0) __syncthreads();  // the bound
            const int B = bound;
            const bool take = low <= B;
            const uint32_t votes = __ballot_sync(0xffffffffu, take);
            uint32_t to = 0;
            if (lane == 0 && votes) to = atomicAdd(&taken[turn], (uint32_t)__popc(votes));
            to = __shfl_sync(0xffffffffu, to, 0) + __popc(votes & ((1u << lane) - 1u));
            if (take) {
                at[to] = i;
                city_of[to] = min(ld_u32(R + i), n - 1);
                if (OR) {
                    bases[0][to] = s.b1;
                    bases[OR ? 1 : 0][to] = s.b2;
                    bases[OR ? 2 : 0][to] = s.b3;
                    bases[OR ? 3 : 0][to] = s.c2;
                    bases[OR ? 4 : 0][to] = s.c3;
                }
            }
            if (threadIdx.x == 0) taken[turn ^ 1u] = 0;  // the next positions'
            __syncthreads();
            const uint32_t entries = taken[turn] * K;
            for (uint32_t t = threadIdx.x; t < entries; t += NT) {
                const uint32_t o = t / K;
                const uint32_t v = min(L.nbr[(size_t)city_of[o] * K + (t - o * K)], n - 1);
                const uint32_t q = min(ld_u32(L.pos + v), n - 1);
                if (OR)
                    s = NbrBases{bases[0][o], bases[OR ? 1 : 0][o], bases[OR ? 2 : 0][o],
                                 bases[OR ? 3 : 0][o], bases[OR ? 4 : 0][o]};
                nbr_entry<OR>(at[o], q, Q, n, L.margin, min(B, pick.bound()), s, pick);
            }
            __syncthreads();
        }
        if (threadIdx.x < 2) taken[threadIdx.x] = 0;
        pick.reduce();
        if (lane == 0) wbest[warp] = pick;
        __syncthreads();
        if (warp == 0) {
            pick = lane < NW ? wbest[lane] : kNoPick;
            pick.reduce();
            if (lane == 0) {
                CoopBest b{};
                b.lo = pick.lo;
                b.hi = pick.hi;
                if (pick.hi != ~0u) {
                    b.city = ld_u32(R + pick.i);
                    b.near = ld_u32(R + pick.q);
                }
                cs->best[sw & 1][blockIdx.x] = b;
            }
        }
        ++sweeps;
        if (!barrier()) {
            timeout = true;
            break;
        }
        // the move, and a seed per lane for the next sweep
        if (warp == 0) {
            NbrPick all = kNoPick;
            uint2 seed = make_uint2(0u, 0u);
            for (uint32_t c = lane; c < gridDim.x; c += 32) {
                const CoopBest& b = cs->best[sw & 1][c];
                const uint32_t h = __ldcg(&b.hi);
                const uint64_t l = __ldcg(&b.lo);
                if (h < all.hi || (h == all.hi && l < all.lo)) {
                    all.hi = h;
                    all.lo = l;
                    seed = make_uint2(__ldcg(&b.city), __ldcg(&b.near));
                }
            }
            seeds[lane] = seed;
            all.reduce();
            if (lane == 0) best = all;
        }
        __syncthreads();
        const NbrPick move = best;
        if (move.hi == ~0u) break;  // converged (every CTA reads the same candidates)
        const int delta = move.bound(), vslot = (int)(move.hi & 7u) - 1;
        const uint32_t a = (uint32_t)(move.lo >> 21), b = (uint32_t)move.lo & 0x1FFFFFu;
        const uint32_t Lg = vslot >= 0 ? or_len(vslot) : 0u;
        const bool rev = vslot >= 0 && or_rev(vslot);
        const bool ok = vslot < 0 ? (a >= 1 && b < n && b >= a + 2)
                                  : (a >= 1 && a + Lg <= n - 1 &&
                                     (b + 2 <= a || (b >= a + Lg && b + 2 <= n)));
        if (!ok) {
            bad = true;
            break;
        }
        const OrderedCity* Qs = Q;
        OrderedCity* Qd = cur ? L.Q0w : L.Q1w;
        uint32_t* Rd = cur ? L.R0w : L.R1w;
        for (uint32_t k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
            const uint32_t km = k == 0 ? n - 1 : k - 1;
            const uint32_t src = vslot < 0 ? rotrev_src(k, a, b, n) : oropt_src(k, a, Lg, b, rev);
            const uint32_t srcm =
                vslot < 0 ? rotrev_src(km, a, b, n) : oropt_src(km, a, Lg, b, rev);
            const OrderedCity qa = ld_city(Qs + src), qb = ld_city(Qs + srcm);
            OrderedCity o;
            o.x = qa.x;
            o.y = qa.y;
            o.e = (float)exact_dist(qb.x, qb.y, qa.x, qa.y);
            o.pad = 0.f;
            Qd[k] = o;
            const uint32_t id = ld_u32(R + src);
            Rd[k] = id;
            L.pos[min(id, n - 1)] = k;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0 && st->move_log && moves < st->log_cap) {
            st->move_log[3 * moves + 0] = delta;
            st->move_log[3 * moves + 1] = vslot < 0 ? (int)a : -1 - (int)(a + ((uint32_t)vslot << 21));
            st->move_log[3 * moves + 2] = (int)b;
        }
        ++moves;
        cur ^= 1u;
        if (moves >= max_moves) limit = true;
        if (!barrier()) {
            timeout = true;
            break;
        }
        if (limit) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long made = moves - moves0;
        st->moves = moves;
        st->total_moves += made;
        st->sweeps += made + (limit || timeout || bad || start_done ? 0 : 1);
        st->nbr_sweeps += sweeps;
        st->cur = cur;
        st->best_key = kNoMove;
        for (int v = 0; v < kOrSlots; ++v) st->or_key[v] = kNoMove;
        st->converged = 1;
        if (limit) atomicOr(&st->status, kErrMoveLimit);
        if (bad) atomicOr(&st->status, kErrBadKey);
    }
}

// Test hook for the bounded wait: one CTA waits at a barrier sized for two,
// which nothing else will reach; the wait gives up after its budget and sets
// kErrTimeout in st->status.
__global__ void barrier_probe_kernel(CoopSync* cs, DevState* st) {
    __shared__ bool ok;
    GridBarrier barrier{&cs->arrived, st, &ok, kCoopWaitNs};
    if (threadIdx.x == 0) barrier.start(2u);
    barrier(2u);
}

}  // namespace

cudaError_t launch_barrier_probe(CoopSync* cs, DevState* st, cudaStream_t s) {
    barrier_probe_kernel<<<1, 32, 0, s>>>(cs, st);
    return cudaGetLastError();
}

template <bool OR, int NT>
static int coop_nbr_grid_t(int device) {
    int per_sm = 0, sms = 0, coop = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, coop_nbr_kernel<OR, NT>, NT, 0) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess)
        return 0;
    if (!coop || per_sm < 1) return 0;
    return std::min<int>(sms, (int)kGridMaxCtas);
}

int coop_nbr_grid(uint32_t n, bool oropt, int device) {
    const int cap = oropt ? coop_nbr_grid_t<true, kCoopNT>(device)
                          : std::min(coop_nbr_grid_t<false, kCoopNT>(device),
                                     coop_nbr_grid_t<false, kCoopWideNT>(device));
    const int want = (int)((n + kCoopLeast - 1) / kCoopLeast);
    return cap < 1 ? 0 : (want < cap ? (want < 1 ? 1 : want) : cap);
}

cudaError_t launch_coop_nbr(const NbrLaunch& L, CoopSync* cs, int grid, cudaStream_t s) {
    // a cooperative launch through the launch attribute, which stream capture
    // records as a cooperative kernel node (the device-run ILS graph)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    const bool wide = !L.oropt && L.n > (uint32_t)grid * kCoopNT;
    cfg.blockDim = dim3(wide ? kCoopWideNT : kCoopNT);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (L.oropt) return cudaLaunchKernelEx(&cfg, coop_nbr_kernel<true, kCoopNT>, L, cs);
    if (wide) return cudaLaunchKernelEx(&cfg, coop_nbr_kernel<false, kCoopWideNT>, L, cs);
    return cudaLaunchKernelEx(&cfg, coop_nbr_kernel<false, kCoopNT>, L, cs);
}

}  // namespace logo
