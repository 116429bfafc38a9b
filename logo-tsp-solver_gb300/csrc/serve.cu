// Serving rounds: continuous batching of independent requests at the
// granularity of a bounded work quantum (sm_103a).
//
// Every admitted request owns a slot: its coordinates, current tour and best
// tour stay resident in a device arena between rounds, and a small state
// record (phase, counters, PRNG state, lengths) in ServeSlot.  A round kernel
// hands the active slots to CTAs through an atomic queue; a CTA loads its
// slot's tour into shared memory and advances the request's ILS -- the same
// descent / accept-or-revert / kick sequence as logo_ils and the batched
// solver (src/solvers/ILSGlobalSolverSequential.cpp:60-100) -- until it has
// spent `budget_pairs` pair evaluations (checked between sweeps) or the
// request is finished, then writes the state back.  Between rounds the host
// retires finished requests and admits new ones, so requests that arrive while
// others run join the next round and share the GPU with them.
//
// A slot's computation depends only on its own input, never on which other
// slots share a round, so a request's result is the same alone and in any mix.
#include <cstdint>

#include "batch_internal.h"
#include "logo_device.cuh"
#include "near_tour.cuh"
#include "serve_internal.h"

namespace logo {

namespace {

// Pair evaluations charged per city and sweep: a sweep looks at a few listed
// neighbours of each city (near_tour.cuh counts them), 16 is what its lists
// hold.  (The default quantum is then 305 sweeps at n = 4,096, a round of 23 ms of
// which 2 go into the lists of clustered cities, built anew in every round; charged
// 48, rounds of 11 ms and a burst of 64 requests up to 15 % slower.)
constexpr unsigned long long kServePairsPerCity = 16;

template <int NT>
__global__ void __launch_bounds__(NT, kNearWarpsPerSm * 32 / NT)
    serve_round_kernel(ServeArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ NearShared<NT, 1, uint16_t> S;

    for (;;) {
        if (threadIdx.x == 0) S.idx = atomicAdd(A.queue, 1u);
        __syncthreads();
        const uint32_t unit = S.idx;
        __syncthreads();
        if (unit >= A.nunits) break;
        const uint32_t slot = A.units[unit];
        ServeSlot st = A.slots[slot];
        if (st.phase == kServeDone) continue;
        const uint32_t n = st.n;
        const float2* xy = A.coords + st.off;
        uint32_t* rio = A.route + st.off;
        uint32_t* bio = A.best + st.off;
        CtaTour T = near_carve(smem_raw, n);
        NearSeed seed;
        uint32_t parity = 0;
        S.init();  // (the last slot's sweeps need not have left it so)

        // load the resident tour into shared memory (the best one stays in the arena)
        for (uint32_t k = threadIdx.x; k < n; k += NT) {
            const uint32_t c = rio[k];
            T.id[k] = (uint16_t)c;
            if (st.phase == kServeInit) bio[k] = c;
        }
        __syncthreads();
        near_build<NT>(T, S, xy);
        near_place<NT>(T, xy);
        if (st.phase == kServeInit) {
            st.start_len = near_length<NT>(T, S);
            st.best_len = st.start_len;
            st.phase = kServeDescent;
        }
        const unsigned long long move_cap = 64ull * n * n + 1024;
        unsigned long long spent = 0;
        uint64_t rng = st.rng;
        while (st.phase != kServeDone && spent < A.budget_pairs) {
            if (st.phase == kServeDescent) {
                const unsigned long long key = near_sweep<NT, false>(T, S, seed, parity);
                parity ^= 1u;
                ++st.sweeps;
                spent += kServePairsPerCity * n;
                if (key == kNoMove) {
                    st.phase = kServeAccept;
                    continue;
                }
                const uint32_t p = key_i(key), q = key_j(key);
                if (!(p >= 1 && q < n && q >= p + 2)) {
                    st.status |= kErrBadKey;
                    st.phase = kServeDone;
                    break;
                }
                near_move<NT>(T, p, q);
                ++st.moves;
                if (++st.descent_moves >= move_cap) {
                    st.status |= kErrMoveLimit;
                    st.phase = kServeDone;
                }
            } else {  // kServeAccept: keep if strictly shorter, else revert
                const unsigned long long len = near_length<NT>(T, S);
                if (len < st.best_len) {
                    st.best_len = len;
                    ++st.accepted;
                    for (uint32_t k = threadIdx.x; k < n; k += NT) bio[k] = T.id[T.slot(k)];
                    __syncthreads();
                } else {
                    for (uint32_t k = threadIdx.x; k < n; k += NT) T.id[k] = (uint16_t)bio[k];
                    __syncthreads();
                    near_place<NT>(T, xy);
                }
                if (st.kicks_done == st.kicks_total) {
                    st.phase = kServeDone;
                    break;
                }
                if (st.kick_kind == 1) {
                    uint32_t c0 = 1 + uniform_below(rng, n - 1);
                    uint32_t c1 = 1 + uniform_below(rng, n - 1);
                    uint32_t c2 = 1 + uniform_below(rng, n - 1);
                    uint32_t t;
                    if (c1 < c0) { t = c0; c0 = c1; c1 = t; }
                    if (c2 < c1) { t = c1; c1 = c2; c2 = t; }
                    if (c1 < c0) { t = c0; c0 = c1; c1 = t; }
                    near_double_bridge<NT>(T, c0, c1, c2);
                } else {
                    uint32_t a = uniform_below(rng, n);
                    uint32_t b = uniform_below(rng, n);
                    if (b < a) { const uint32_t t = a; a = b; b = t; }
                    near_move<NT>(T, a, b);
                }
                ++st.kicks_done;
                st.descent_moves = 0;
                st.phase = kServeDescent;
            }
        }
        st.rng = rng;
        // write the resident state back, in tour order
        for (uint32_t k = threadIdx.x; k < n; k += NT) rio[k] = T.id[T.slot(k)];
        if (threadIdx.x == 0) A.slots[slot] = st;
        __syncthreads();
    }
}

}  // namespace

size_t serve_smem_bytes(uint32_t max_n) { return near_layout(max_n).bytes; }

constexpr int kServeNT = 256;

cudaError_t launch_serve_round(const ServeArgs& A, int grid, cudaStream_t s, int* occupancy) {
    const size_t smem = serve_smem_bytes(A.max_n);
    auto kern = serve_round_kernel<kServeNT>;
    if (occupancy) {
        // for the largest request: the attribute is shared by every server
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)serve_smem_bytes(kBatchMaxN));
        if (e != cudaSuccess) return e;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occupancy, kern, kServeNT, smem);
    }
    kern<<<grid, kServeNT, smem, s>>>(A);
    return cudaGetLastError();
}

}  // namespace logo
