// Descents and ILS calls of large tours (n > kSoloMaxN) as one cooperative
// launch (sm_103a).
//
// The tour is the ring of near_tour.cuh in global memory (L2: 20 bytes a city);
// the slots of a sweep are dealt to all warps of the grid, and a move is the
// reversal of the shorter arc, in place, by all threads.  So a move costs a sweep
// of a few dependent L2 reads and two grid barriers instead of four kernels that
// go over windows, tiles and the whole tour (n = 100,000: 86 us a move).
//
// A grid barrier: each CTA leaves its best key, thread 0 adds to a counter
// (release) and polls it (acquire, which also makes the SM's L1 current: the
// arrays are read through it, and other SMs rewrite them between barriers;
// bounded by %globaltimer, after which the CTA sets kErrTimeout and every CTA
// gives up in turn).  Every CTA reads the same keys and so does the same.
#include <mutex>

#include "logo_device.cuh"
#include "logo_internal.h"
#include "near_tour.cuh"

namespace logo {

namespace {

constexpr int kGridNT = 1024;  // one CTA per SM
constexpr unsigned long long kGridWaitNs = 20000000000ull;  // other kernels may hold SMs for long

using GridTour = NearTour<uint32_t, kCtxNear>;

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

struct GridBarrier {
    GridSync* gs;
    DevState* st;
    bool* ok;  // shared
    unsigned long long target = 0;

    // False when the wait ran out (the same in every thread of the CTA).
    __device__ __forceinline__ bool operator()() {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(&gs->arrived) : "memory");
            bool fine = true;
            unsigned long long t0 = 0;
            for (uint32_t it = 0; ld_acquire_u64(&gs->arrived) < target; ++it) {
                if ((it & 255u) == 255u) {
                    const unsigned long long now = global_timer_ns();
                    if (t0 == 0) t0 = now;
                    if (now - t0 > kGridWaitNs) {
                        atomicOr(&st->status, kErrTimeout);
                        fine = false;
                        break;
                    }
                }
            }
            *ok = fine;
        }
        __syncthreads();
        return *ok;
    }
};

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

template <bool ILS>
__global__ void __launch_bounds__(kGridNT, 1) near_grid_kernel(GridArgs A) {
    constexpr int NT = kGridNT, NW = NT / 32;
    __shared__ NearShared<NT, 1, uint32_t> S;
    __shared__ bool bar_ok;
    __shared__ uint2 seeds[32];
    __shared__ unsigned long long best_key;
    DevState* st = A.solo.st;
    // set before the launch and identical for every CTA
    if (*(volatile unsigned int*)&st->converged) return;
    const uint32_t n = A.solo.n, rank = blockIdx.x, ranks = gridDim.x;
    const uint32_t tid = rank * NT + threadIdx.x, threads = ranks * NT;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t cur = *(volatile unsigned int*)&st->cur;
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
    T.pos = A.pos;
    T.nbr = reinterpret_cast<NearEntry<uint32_t>*>(A.solo.near.nbr);
    T.cell = A.solo.near.cell;
    T.cellid = A.solo.near.cellid;
    T.g = A.solo.near.g;
    GridBarrier barrier{A.gs, st, &bar_ok};
    S.init();
    grid_place(T, Rg, A.solo.xy, tid, threads);
    bool ok = barrier();
    NearSeed seed;
    uint32_t parity = 0;
    unsigned long long m0 = *(volatile unsigned long long*)&st->moves;
    const unsigned long long maxm = *(volatile unsigned long long*)&st->max_moves;
    unsigned long long m = 0, sweeps = 0, total_m = 0;
    unsigned long long best_len = 0, accepted = 0, kicks = 0;
    uint64_t rng = 0;
    if (ILS) {
        best_len = *(volatile unsigned long long*)&st->best_length;
        rng = *(volatile unsigned long long*)&st->rng;
    }
    bool limit = false, bad = false;
    for (uint32_t it = 0; ok; ++it) {
        m = 0;
        for (;;) {
            const uint64_t mine =
                warp_min_u64(near_scan<NT, false>(T, S, seed, parity, rank, ranks));
            if (lane == 0) S.wbest[0][warp] = mine;
            __syncthreads();
            if (warp == 0) {
                const uint64_t best = warp_min_u64(lane < NW ? S.wbest[0][lane] : kNoMove);
                if (lane == 0) {
                    A.gs->keys[parity][rank] = best;
                    S.reset(parity ^ 1);  // the next sweep's
                }
            }
            if (!(ok = barrier())) break;
            ++sweeps;
            // one warp per CTA reads the keys (all of them reading the same few
            // lines queued up at L2 for 7 us)
            if (warp == 0) {
                const uint64_t k = near_pick(T, A.gs->keys[parity], ranks, seed);
                seeds[lane] = make_uint2(seed.a, seed.b);
                if (lane == 0) best_key = k;
            }
            __syncthreads();
            const uint64_t key = best_key;
            seed.a = seeds[lane].x;
            seed.b = seeds[lane].y;
            parity ^= 1u;
            if (key == kNoMove) break;  // local optimum
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
        }
        total_m += m;
        if (!ILS || !ok || bad) break;
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
    if (ok) {
        // the tour in its order, with the positions that other kernels keep
        for (uint32_t k = tid; k < n; k += threads) {
            const uint32_t j = T.slot(k);
            const uint32_t id = T.id[j];
            const float2 c = T.xy[j];
            const OrderedCity o{c.x, c.y, T.E[T.rev ? T.wrap(j + 1) : j], 0.f};
            Rg[k] = id;
            Qg[k] = o;
            T.pos[id] = k;
            if (ILS) A.solo.Qbest[k] = o;
        }
    }
    if (tid == 0) {
        if (ok) {
            st->moves = m0 + m;
            st->total_moves += total_m;
            st->sweeps += sweeps;
            st->best_key = kNoMove;
            if (ILS) {
                st->rng = rng;
                st->best_length = best_len;
                st->accepted += accepted;
                st->kicks += kicks;
            }
            if (limit) atomicOr(&st->status, kErrMoveLimit);
            if (bad) atomicOr(&st->status, kErrBadKey);
        }
        st->converged = 1;
    }
}

template <bool ILS>
int grid_ctas_t(int device) {
    int per_sm = 0, sms = 0, coop = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, near_grid_kernel<ILS>, kGridNT, 0) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess)
        return 0;
    return coop && per_sm >= 1 ? (int)std::min<uint32_t>((uint32_t)sms, kGridMaxCtas) : 0;
}

}  // namespace

int near_grid_ctas(uint32_t n, int device) {
    if (n <= kSoloMaxN) return 0;
    return std::min(grid_ctas_t<false>(device), grid_ctas_t<true>(device));
}

cudaError_t launch_near_grid(const GridArgs& A, bool ils, int ctas, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(A.gs, 0, sizeof(GridSync), s);
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
    if (ils) return cudaLaunchKernelEx(&cfg, near_grid_kernel<true>, A);
    return cudaLaunchKernelEx(&cfg, near_grid_kernel<false>, A);
}

}  // namespace logo
