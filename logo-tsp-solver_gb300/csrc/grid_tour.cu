// Descents and ILS calls of large tours (n > kSoloMaxN) as cooperative launches over
// the whole device (sm_103a).
//
// The tour is the ring of near_tour.cuh in global memory (L2: 20 bytes a city);
// the slots of a sweep are dealt to all warps of the grid, and a move is the
// reversal of the shorter arc, in place, by all threads.  So a move costs a sweep
// of a few dependent L2 reads and two grid barriers instead of four kernels that
// go over windows, tiles and the whole tour (n = 100,000: 86 us a move).
//
// Every CTA leaves its best key before a grid barrier (grid_barrier.cuh), reads the
// same keys after it and so does the same.
//
// The launch holds every SM (a CTA's registers are all that an SM has), so nothing
// else runs beside it: after quantum_ns it ends, between two moves, with everything
// in the state, and the host launches it again behind whatever else is waiting.
//
// As a whole call the launch also loads and checks the caller's route and leaves
// result and state in host memory: one launch and one wait.  Against route load,
// three sweep kernels and move (us a best move, the other path first): NN tour of
// n = 6,200 41, 48; 7,000 54, 53; 20,000 70, 55; 40,009 72, 73; 100,000 83, 66; 200,000
// 132, 86; random tour 65, 42; 79, 42; 45, 49; 46, 59; 58, 66; 84, 75; some hundred
// moves on 41, 31; 41, 33; 74, 40; 73, 49; 95, 57; 146, 101.  Which of these a caller's
// route is does not show before the sweep, so no rule of a dispatch chooses.
//
// Up to A.spread cities a CTA goes through its large discs itself, above (SPREAD) they
// are dealt to all CTAs after one more barrier: with more slots a CTA, one had up to
// 20 discs while the others waited (best move of an NN tour of n = 100,000: 95 -> 66
// us, of 1,000,000: 247 -> 165; of a random one 81 -> 66 and 163 -> 109; a sweep early
// in a descent of n = 100,000: 57 -> 43.  Below, the barrier costs more: n = 20,000
// clustered 23 -> 26 us a sweep, 1 of it by the kernel's size alone, so there are two;
// n = 40,009 35 -> 35, later in the descent 26 -> 31).
//
// Discs of more than kGridDisc cities (long edges of a tour far from a local
// optimum) are put off to all CTAs: the few edges against every edge that can
// take part, after one more barrier.  One CTA going through them held up the rest
// (best move of the 1,000,000-city tour: 375 us).  Dealing out every slot
// whose list was too short the same way costs the barrier in each sweep and was
// slower (n = 20,000: 18.9 -> 20.8 us a sweep).
#include <cstddef>

#include "grid_barrier.cuh"
#include "logo_device.cuh"
#include "logo_internal.h"
#include "near_tour.cuh"

namespace logo {

namespace {

constexpr int kGridNT = 1024;  // one CTA per SM
constexpr unsigned long long kGridWaitNs = 20000000000ull;  // other kernels may hold SMs for long

using GridTour = NearTour<uint32_t, kCtxNear>;

// Slot k = position k = city route[k], by all threads; a barrier must follow.
__device__ __forceinline__ void grid_place(GridTour& T, const uint32_t* route, const float2* xy,
                                           uint32_t tid, uint32_t threads) {
    T.o = 0;
    T.rev = false;
    for (uint32_t k = tid; k < T.n; k += threads) {
        const uint32_t v = __ldcg(route + k), w = __ldcg(route + (k == 0 ? T.n - 1 : k - 1));
        const float2 p = xy[v];
        T.xy[k] = p;
        T.E[k] = near_dist(xy[w], p);
        T.id[k] = v;
        T.pos[v] = k;
    }
}

// The pairs of `count` edges with every edge, by `threads` threads.
__device__ __forceinline__ void grid_edges(const GridTour& T, const uint32_t* edges,
                                           uint32_t count, uint32_t z, NearBest& nb, uint32_t tid,
                                           uint32_t threads) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t base = tid - lane; base < T.n; base += threads) {  // whole warps
        const uint32_t g = base + lane;
        near_edges(T, edges, count,
                   g < T.n && g != z && 2.f * T.E[min(g, T.n - 1)] + 8.f >= -nb.B, g, z, nb);
    }
}

// The caller's route as grid_place, with the check that it is a permutation
// (load_route_kernel in tour.cu) and the tour's other copy; true when this
// thread met a city twice or none.
__device__ __forceinline__ bool grid_load(GridTour& T, const SoloArgs& A,
                                          unsigned long long* length, uint32_t tid,
                                          uint32_t threads) {
    const uint32_t n = T.n, lane = threadIdx.x & 31;
    T.o = 0;
    T.rev = false;
    bool bad = false;
    unsigned long long sum = 0;
    for (uint32_t base = tid - lane; base < n; base += threads) {  // whole warps
        const uint32_t k = base + lane;
        uint32_t v = k < n ? A.call.src[k] : 0u;
        uint32_t w = __shfl_up_sync(0xffffffffu, v, 1);
        if (lane == 0) w = A.call.src[k == 0 ? n - 1 : k - 1];
        if (k >= n) continue;
        const bool miss = v >= n || atomicExch(&A.call.seen[v], A.call.epoch) == A.call.epoch;
        bad |= miss;
        if (A.R0 != A.call.src) A.R0[k] = v;
        v = min(v, n - 1);
        w = min(w, n - 1);
        const float2 p = A.xy[v];
        const float e = near_dist(A.xy[w], p);
        A.Q0[k] = OrderedCity{p.x, p.y, e, 0.f};
        T.xy[k] = p;
        T.E[k] = e;
        T.id[k] = v;
        T.pos[v] = k;
        sum += (unsigned long long)e;
    }
    if (length) {
        sum = warp_sum_u64(sum);
        if (lane == 0 && sum) atomicAdd(length, sum);
    }
    return bad;
}

template <bool ILS, bool SPREAD>
__global__ void __launch_bounds__(kGridNT, 1) near_grid_kernel(GridArgs A) {
    constexpr int NT = kGridNT, NW = NT / 32;
    __shared__ NearShared<NT, 1, uint32_t> S;
    __shared__ bool bar_ok;
    __shared__ uint2 seeds[32];
    __shared__ unsigned long long best_key;
    __shared__ uint32_t wide_count, disc_count, pause_now;
    // (in shared memory for the sweep's registers; one thread uses them)
    __shared__ uint32_t most[3];
    __shared__ unsigned long long begun;
    DevState* st = A.solo.st;
    const bool whole = !ILS && A.solo.call.src != nullptr;
    // set before the launch and identical for every CTA
    if (!whole && *(volatile unsigned int*)&st->converged) return;
    const uint32_t n = A.solo.n, rank = blockIdx.x, ranks = gridDim.x;
    const uint32_t tid = rank * NT + threadIdx.x, threads = ranks * NT;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        begun = global_timer_ns();
        most[0] = most[1] = most[2] = 0;
    }
    const uint32_t cur = whole ? 0u : *(volatile unsigned int*)&st->cur;
    OrderedCity* Qg = cur ? A.solo.Q1 : A.solo.Q0;
    uint32_t* Rg = cur ? A.solo.R1 : A.solo.R0;
    // the ring lies in the other tour buffer: xy, E, id by slot
    unsigned char* ring = reinterpret_cast<unsigned char*>(cur ? A.solo.Q0 : A.solo.Q1);
    GridTour T;
    T.n = n;
    T.kc = min(n - 1, kCtxNear);
    T.whole = n - 1 <= kCtxNear;
    T.xy = reinterpret_cast<float2*>(ring);
    T.E = reinterpret_cast<float*>(ring + 8 * (size_t)n);
    T.id = reinterpret_cast<uint32_t*>(ring + 12 * (size_t)n);
    T.pos = A.solo.pos;
    T.nbr = reinterpret_cast<NearEntry<uint32_t>*>(A.solo.near.nbr);
    T.cell = A.solo.near.cell;
    T.cellid = A.solo.near.cellid;
    T.g = A.solo.near.g;
    GridBarrier barrier{&A.gs->arrived, st, &bar_ok, kGridWaitNs};
    S.init();
    // this CTA's best key, and the counters of the next sweep
    uint32_t parity = 0;
    auto publish = [&](unsigned long long* keys, uint64_t key) {
        const uint64_t mine = warp_min_u64(key);
        if (lane == 0) S.wbest[0][warp] = mine;
        __syncthreads();
        if (warp == 0) {
            const uint64_t best = warp_min_u64(lane < NW ? S.wbest[0][lane] : kNoMove);
            if (lane == 0) {
                keys[rank] = best;
                S.reset(parity ^ 1);
            }
        }
    };
    // a whole call's state goes to the host with the last CTA, so that a wait of any
    // CTA that ran out is in it
    auto leave = [&] {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            bar_ok = atomicAdd(&A.gs->left, 1u) == ranks - 1;
            __threadfence();
        }
        __syncthreads();
        if (bar_ok) leave_call(st, A.solo.call.mirror);
    };
    const bool step = whole && A.solo.call.step, lengths = whole && A.solo.call.lengths;
    if (whole && tid == 0) start_call(st, A.solo.call.max_moves);
    if (whole) {
        if (grid_load(T, A.solo, lengths ? &A.gs->start_length : nullptr, tid, threads))
            atomicExch(&A.gs->bad, 1ull);
    } else {
        grid_place(T, Rg, A.solo.xy, tid, threads);
    }
    bool ok = barrier();
    if (whole && ok && ld_acquire_u64(&A.gs->bad)) {  // the same in every CTA
        if (tid == 0) {
            st->bad_route = 1;
            st->converged = 1;
        }
        leave();
        return;
    }
    NearSeed seed;
    unsigned long long m0 = whole ? 0ull : *(volatile unsigned long long*)&st->moves;
    const unsigned long long maxm =
        whole ? A.solo.call.max_moves : *(volatile unsigned long long*)&st->max_moves;
    unsigned long long step_key = kNoMove;
    unsigned long long m = 0, sweeps = 0, total_m = 0;
    unsigned long long best_len = 0, accepted = 0, kicks = 0;
    uint64_t rng = 0;
    if (ILS) {
        best_len = *(volatile unsigned long long*)&st->best_length;
        rng = *(volatile unsigned long long*)&st->rng;
    }
    bool limit = false, bad = false, paused = false;
    for (uint32_t it = ILS ? (uint32_t)*(volatile unsigned long long*)&st->kicks : 0u; ok; ++it) {
        m = 0;
        for (;;) {
            NearBest nb{near_scan<NT, false, SPREAD>(T, S, seed, parity, rank, ranks, A.disc),
                        -1.f};
            const uint32_t z = T.closing();
            auto& put = A.gs->put[parity];
            __syncthreads();
            // (the same for every thread)
            const uint32_t huges = SPREAD ? min(S.big[parity], kNearWide) : S.huges[parity];
            if (huges) {
                // (the CTA's bound, not the lane's own best: near_far wants one for the warp)
                nb.B = fminf((float)S.bound[parity], (float)S.far_bound[parity]);
                const float h = near_half((float)S.bound[parity]);
                for (uint32_t o = warp; o < huges; o += NW) {
                    const uint32_t j = SPREAD ? S.wide[o] : S.huge[o];
                    // its disc, or where that is too large its edges that reach beyond its list
                    const bool disc = SPREAD && !near_large(T, j, z, A.disc, nb.B);
#pragma unroll 1
                    for (uint32_t s = 0; s < (disc ? 1u : 2u); ++s) {
                        const uint32_t f = s ? T.wrap(j + 1) : j;
                        if (!disc && (f == z || T.last_sq(j) > near_limit(T.E[f] + h))) continue;
                        uint32_t at = 0;
                        if (lane == 0)
                            at = atomicAdd(disc ? &put.discs : &put.wides, 1u);
                        at = __shfl_sync(0xffffffffu, at, 0);
                        if (at >= (disc ? A.discs : A.wide))
                            near_far(T, j, z, ~0u, nb.B, nb);  // no room for this one
                        else if (lane == 0)
                            (disc ? A.disc_list + parity * kGridDiscs : A.gs->wide[parity])[at] = f;
                    }
                }
            }
            // (the clock is slow to read)
            if (tid == 0 && ((sweeps & 15u) == 15u || A.quantum_ns < 1000000u) &&
                global_timer_ns() - begun > A.quantum_ns)
                put.pause = 1u;
            publish(A.gs->keys[parity], nb.key);
            if (!(ok = barrier())) break;
            ++sweeps;
            if (tid == 0) {  // the next sweep's
                auto& next = A.gs->put[parity ^ 1];
                next.wides = next.discs = next.takers = 0;
            }
            // one warp per CTA reads the keys (all of them reading the same few
            // lines queued up at L2 for 7 us)
            if (warp == 0) {
                const uint4 p = __ldcg(reinterpret_cast<const uint4*>(&put));
                const uint64_t k = near_pick(T, A.gs->keys[parity], ranks, seed);
                seeds[lane] = make_uint2(seed.a, seed.b);
                if (lane == 0) {
                    best_key = k;
                    wide_count = p.x;
                    pause_now = p.y;
                    disc_count = p.z;
                }
            }
            __syncthreads();
            uint64_t key = best_key;
            const uint32_t wides = min(wide_count, A.wide);
            const uint32_t discs = SPREAD ? min(disc_count, A.discs) : 0u;
            if (wides || discs) {
                if (tid == 0) {
                    most[0] = max(most[0], wide_count);
                    most[2] = max(most[2], SPREAD ? disc_count : 0u);
                }
                const float known = key == kNoMove ? -1.f : (float)key_delta(key);
                NearBest more{key, known};
                if constexpr (SPREAD) {
                    // discs put off, a CTA each
                    for (uint32_t d = rank; d < discs; d += ranks) {
                        const uint32_t j = A.disc_list[parity * kGridDiscs + d], jn = T.wrap(j + 1);
                        const float m =
                            fmaxf(j == z ? kNoEdge : T.E[j], jn == z ? kNoEdge : T.E[jn]);
                        if (2.f * m + 8.f >= -known &&
                            T.last_sq(j) <= near_limit(m + near_half(known)))
                            near_far(T, j, z, ~0u, known, more, warp, NW);
                    }
                }
                // edges put off, with every edge that can take part: listed first,
                // so that the pairs can be dealt evenly, unless those are too many
                if (wides) {
                    for (uint32_t base = tid - lane; base < n; base += threads) {
                        const uint32_t g = base + lane;
                        const bool takes = g < n && g != z && 2.f * T.E[g] + 8.f >= -known;
                        const uint32_t votes = __ballot_sync(0xffffffffu, takes);
                        if (votes == 0) continue;
                        uint32_t at = 0;
                        if (lane == 0)
                            at = atomicAdd(&put.takers, (uint32_t)__popc(votes));
                        at = __shfl_sync(0xffffffffu, at, 0) + __popc(votes & ((1u << lane) - 1u));
                        if (takes && at < A.takers) A.gs->taker[at] = g;
                    }
                    if (!(ok = barrier())) break;
                    const uint32_t takers = *(volatile uint32_t*)&put.takers;
                    if (tid == 0) most[1] = max(most[1], takers);
                    if (takers <= A.takers) {
                        for (uint32_t base = tid - lane; base < wides * takers; base += threads) {
                            const uint32_t t = base + lane;
                            const bool in = t < wides * takers;
                            near_edges(T, &A.gs->wide[parity][in ? t / takers : 0], 1u, in,
                                       A.gs->taker[in ? t % takers : 0], z, more);
                        }
                    } else {
                        grid_edges(T, A.gs->wide[parity], wides, z, more, tid, threads);
                    }
                }
                publish(A.gs->wide_keys[parity], more.key);
                if (!(ok = barrier())) break;
                if (warp == 0) {
                    NearSeed other;
                    const uint64_t k = near_pick(T, A.gs->wide_keys[parity], ranks, other);
                    if (lane == 0) best_key = k;
                }
                __syncthreads();
                key = best_key;
            }
            seed.a = seeds[lane].x;
            seed.b = seeds[lane].y;
            parity ^= 1u;
            if (key == kNoMove) break;  // local optimum
            if (step) {
                step_key = key;
                break;
            }
            // reported move (i, j+1): p = i < q = j+1 (twoOptLocalSolver.cpp:41-48)
            const uint32_t p = key_i(key), q = key_j(key);
            if (!(p >= 1 && q < n && q >= p + 2)) {
                bad = true;
                break;
            }
            if (!ILS && tid == 0) {
                int* log = st->move_log;
                const unsigned long long idx = m0 + m;
                if (log && idx < st->log_cap) {
                    log[3 * idx + 0] = key_delta(key);
                    log[3 * idx + 1] = (int)p;
                    log[3 * idx + 2] = (int)q;
                }
            }
            near_move(T, p, q, tid, threads);
            ++m;
            if (!(ok = barrier())) break;
            if (m0 + m >= maxm) {
                limit = true;
                break;
            }
            if (pause_now) {  // (the same in every CTA)
                paused = true;
                break;
            }
        }
        total_m += m;
        if (!ILS || !ok || bad || paused) break;
        // length of the tour; keep it if strictly shorter than the best, else go back
        unsigned long long part = 0;
        for (uint32_t k = tid; k < n; k += threads) part += (unsigned long long)T.E[k];
        part = warp_sum_u64(part);
        if (lane == 0 && part) atomicAdd(&A.gs->length[it & 1], part);
        if (!(ok = barrier())) break;
        const unsigned long long len = ld_acquire_u64(&A.gs->length[it & 1]);
        if (tid == 0) A.gs->length[(it & 1) ^ 1] = 0;  // the next descent's (two barriers away)
        if (len < best_len) {
            for (uint32_t k = tid; k < n; k += threads) A.solo.route_best[k] = T.id[T.slot(k)];
            best_len = len;
            ++accepted;
        } else {
            grid_place(T, A.solo.route_best, A.solo.xy, tid, threads);
        }
        if (!(ok = barrier())) break;
        if (it == A.solo.kicks) break;
        // kick (the same draws as kick_kernel in tour.cu)
        if (A.solo.kick_kind == 1) {
            uint32_t c[3];
            for (int k = 0; k < 3; ++k) c[k] = 1 + uniform_below(rng, n - 1);
            uint32_t t;
            if (c[1] < c[0]) { t = c[0]; c[0] = c[1]; c[1] = t; }
            if (c[2] < c[1]) { t = c[1]; c[1] = c[2]; c[2] = t; }
            if (c[1] < c[0]) { t = c[0]; c[0] = c[1]; c[1] = t; }
            near_double_bridge(T, c[0], c[1], c[2], tid, threads,
                               [&] { ok = barrier() && ok; });
        } else {
            uint32_t a = uniform_below(rng, n);
            uint32_t b = uniform_below(rng, n);
            if (b < a) { const uint32_t t = a; a = b; b = t; }
            near_move(T, a, b, tid, threads);
            ok = barrier();
        }
        ++kicks;
        m0 = 0;
    }
    if (ok && !step) {  // (a step's tour went there as it was loaded)
        // the tour in its order, with the positions that other kernels keep
        unsigned long long part = 0;
        for (uint32_t k = tid; k < n; k += threads) {
            const uint32_t j = T.slot(k);
            const uint32_t id = T.id[j];
            const float2 c = T.xy[j];
            const OrderedCity o{c.x, c.y, T.E[T.rev ? T.wrap(j + 1) : j], 0.f};
            part += (unsigned long long)o.e;
            Rg[k] = id;
            Qg[k] = o;
            T.pos[id] = k;
            if (ILS && !paused) A.solo.Qbest[k] = o;
            if (whole && A.solo.call.out && !paused) A.solo.call.out[k] = id;
        }
        if (lengths && !paused) {
            part = warp_sum_u64(part);
            if (lane == 0 && part) atomicAdd(&A.gs->length[0], part);
            ok = barrier();
        }
    }
    if (lengths && tid == 0) {
        st->start_length = ld_acquire_u64(&A.gs->start_length);
        if (!paused) st->length = ld_acquire_u64(&A.gs->length[0]);
    }
    if (tid == 0) {
        if (ok) {
            st->moves = m0 + m;
            st->total_moves += total_m;
            if (!step) st->sweeps += sweeps;
            st->best_key = step_key;
            if (ILS) {
                st->rng = rng;
                st->best_length = best_len;
                st->accepted += accepted;
                st->kicks += kicks;
            }
            if (limit) atomicOr(&st->status, kErrMoveLimit);
            if (bad) atomicOr(&st->status, kErrBadKey);
        }
        st->converged = (step || paused) && ok ? 0u : 1u;
        A.gs->most_wides = most[0];
        A.gs->most_takers = most[1];
        A.gs->most_discs = most[2];
    }
    if (whole) leave();
}

template <bool ILS, bool SPREAD>
int grid_ctas_t(int device) {
    int per_sm = 0, sms = 0, coop = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, near_grid_kernel<ILS, SPREAD>, kGridNT, 0) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess)
        return 0;
    return coop && per_sm >= 1 ? (int)std::min<uint32_t>((uint32_t)sms, kGridMaxCtas) : 0;
}

}  // namespace

int near_grid_ctas(uint32_t n, int device) {
    if (n <= kSoloMaxN) return 0;
    return std::min({grid_ctas_t<false, false>(device), grid_ctas_t<true, false>(device),
                     grid_ctas_t<false, true>(device), grid_ctas_t<true, true>(device)});
}

cudaError_t launch_near_grid(const GridArgs& A, bool ils, int ctas, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(A.gs, 0, offsetof(GridSync, keys), s);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kGridNT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (A.solo.n > A.spread)
        return ils ? cudaLaunchKernelEx(&cfg, near_grid_kernel<true, true>, A)
                   : cudaLaunchKernelEx(&cfg, near_grid_kernel<false, true>, A);
    return ils ? cudaLaunchKernelEx(&cfg, near_grid_kernel<true, false>, A)
               : cudaLaunchKernelEx(&cfg, near_grid_kernel<false, false>, A);
}

}  // namespace logo
