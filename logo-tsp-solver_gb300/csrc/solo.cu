// One small instance solved by one thread-block cluster (n <= kSoloMaxN), and
// the neighbour lists of a single-instance context (sm_103a).
//
// A descent is a chain of sweeps and moves, so its time is the latency of one
// link.  A cluster holds the tour in every CTA's shared memory (near_tour.cuh),
// deals the sweep's slots to all of its warps, and needs one hardware cluster
// barrier per move: the warps' best keys go straight into every CTA's shared
// memory, and each CTA applies the same move to its own copy.  The CTAs of a
// cluster are resident together by construction, so nothing waits on memory.
//
// As a whole call the launch loads and checks the caller's route as well, each
// CTA handing its share to the others, and leaves result and state in host
// memory: one launch and one wait (best move of 52 cities: 29 -> 20.5 us, of which
// a 1 KB memset with its wait takes 8).
//
// The bookkeeping is that of sweep.cu + apply_move_kernel
// (src/solvers/twoOptLocalSolver.cpp:22-64): moves, total_moves, sweeps (+1 for
// the converging sweep), the move log, kErrMoveLimit at max_moves, kErrBadKey
// on an out-of-range key; the final tour goes back to buffer `cur`.
#include <cmath>

#include "logo_device.cuh"
#include "logo_internal.h"
#include "near_tour.cuh"

namespace logo {

namespace {

constexpr uint32_t kSoloMaxCtas = 16;  // largest cluster (needs the non-portable opt-in)

struct SoloLayout {
    uint32_t xy, e, id, pos, best, bytes;
};
__host__ __device__ constexpr SoloLayout solo_layout(uint32_t n) {
    SoloLayout l{};
    l.xy = 0;                                    // float2[n]
    l.e = near_pad16(l.xy + 8 * n);              // float[n]
    l.id = near_pad16(l.e + 4 * n);              // uint32[n]
    l.pos = near_pad16(l.id + 4 * n);            // uint32[n]
    l.best = near_pad16(l.pos + 4 * n);          // uint32[n] (ILS)
    l.bytes = near_pad16(l.best + 4 * n);
    return l;
}

// ILS == false: one descent (or, as a whole call, one sweep).  ILS == true: a
// whole ILS call, every CTA doing the same length, accept/revert and kick on its
// own copy (ILSGlobalSolverSequential.cpp:87-94, ILSGlobalSolver.cpp:37-48 and the
// double bridge).
template <int NT, bool ILS>
__global__ void __launch_bounds__(NT) near_solo_kernel(SoloArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ NearShared<NT, (int)kSoloMaxCtas, uint32_t> S;
    DevState* st = A.st;
    const bool whole = !ILS && A.call.src != nullptr;
    // set before the launch and identical for every CTA
    if (!whole && *(volatile unsigned int*)&st->converged) return;
    const uint32_t rank = cluster_rank(), ranks = cluster_ctas();
    const uint32_t cur = whole ? 0u : *(volatile unsigned int*)&st->cur;
    OrderedCity* Qg = cur ? A.Q1 : A.Q0;
    uint32_t* Rg = cur ? A.R1 : A.R0;
    const SoloLayout l = solo_layout(A.n);
    NearTour<uint32_t, kCtxNear> T;
    T.n = A.n;
    T.o = 0;
    T.rev = false;
    T.kc = min(A.n - 1, kCtxNear);
    T.whole = A.n - 1 <= kCtxNear;
    T.xy = reinterpret_cast<float2*>(smem_raw + l.xy);
    T.E = reinterpret_cast<float*>(smem_raw + l.e);
    T.id = reinterpret_cast<uint32_t*>(smem_raw + l.id);
    T.pos = reinterpret_cast<uint32_t*>(smem_raw + l.pos);
    T.nbr = reinterpret_cast<NearEntry<uint32_t>*>(A.near.nbr);
    T.cell = A.near.cell;
    T.cellid = A.near.cellid;
    T.g = A.near.g;
    uint32_t* best = reinterpret_cast<uint32_t*>(smem_raw + l.best);
    const uint32_t n = T.n;
    S.init();
    if (whole) {
        // each CTA reads its share of the route and hands it to all; each then
        // checks and places the whole tour
        for (uint32_t k = threadIdx.x; k < n; k += NT) T.pos[k] = ~0u;
        cluster_barrier();  // every CTA runs before any is written to
        for (uint32_t k = rank * NT + threadIdx.x; k < n; k += ranks * NT) {
            const uint32_t v = A.call.src[k];
            if (Rg != A.call.src) Rg[k] = v;
            for (uint32_t c = 0; c < ranks; ++c) cluster_store(T.id + k, c, v);
        }
        cluster_barrier();
        bool bad_id = false;
        for (uint32_t k = threadIdx.x; k < n; k += NT) {
            uint32_t v = T.id[k];
            if (v >= n || atomicExch(&T.pos[v], k) != ~0u) {
                bad_id = true;
                v = min(v, n - 1);
            }
            T.xy[k] = A.xy[v];
        }
        if (__syncthreads_or(bad_id)) {  // the same in every CTA
            if (rank == 0 && threadIdx.x == 0) {
                start_call(st, A.call.max_moves);
                st->bad_route = 1;
                st->converged = 1;
            }
            if (rank == 0) leave_call(st, A.call.mirror);
            return;
        }
        for (uint32_t k = threadIdx.x; k < n; k += NT)
            T.E[k] = near_dist(T.xy[k == 0 ? n - 1 : k - 1], T.xy[k]);
        __syncthreads();
    } else {
        for (uint32_t k = threadIdx.x; k < n; k += NT) {
            T.id[k] = Rg[k];
            if (ILS) best[k] = A.route_best[k];
        }
        __syncthreads();
        near_place<NT>(T, A.xy);
        cluster_barrier();  // every CTA's result slots exist before any is written
    }
    NearSeed seed;
    uint32_t parity = 0;
    unsigned long long m0 = whole ? 0ull : *(volatile unsigned long long*)&st->moves;
    const unsigned long long maxm =
        whole ? A.call.max_moves : *(volatile unsigned long long*)&st->max_moves;
    unsigned long long start_len = 0, step_key = kNoMove;
    if (whole && A.call.lengths) start_len = near_length<NT>(T, S);
    unsigned long long m = 0, sweeps = 0, total_m = 0;
    unsigned long long best_len = 0, accepted = 0, kicks = 0;
    uint64_t rng = 0;
    if (ILS) {
        best_len = *(volatile unsigned long long*)&st->best_length;
        rng = *(volatile unsigned long long*)&st->rng;
    }
    bool limit = false, bad = false;
    for (uint32_t it = 0;; ++it) {
        m = 0;
        for (;;) {
            const unsigned long long key = near_sweep<NT, true>(T, S, seed, parity, rank, ranks);
            parity ^= 1u;
            ++sweeps;
            if (key == kNoMove) break;  // local optimum
            if (whole && A.call.step) {
                step_key = key;
                break;
            }
            // reported move (i, j+1): p = i < q = j+1 (twoOptLocalSolver.cpp:41-48)
            const uint32_t p = key_i(key), q = key_j(key);
            if (!(p >= 1 && q < n && q >= p + 2)) {
                bad = true;
                break;
            }
            if (!ILS && rank == 0 && threadIdx.x == 0) {
                int* log = st->move_log;
                const unsigned long long idx = m0 + m;
                if (log && idx < st->log_cap) {
                    log[3 * idx + 0] = key_delta(key);
                    log[3 * idx + 1] = (int)p;
                    log[3 * idx + 2] = (int)q;
                }
            }
            near_move<NT>(T, p, q);
            ++m;
            if (m0 + m >= maxm) {
                limit = true;
                break;
            }
        }
        total_m += m;
        if (!ILS || bad) break;
        // keep the tour if it is strictly shorter than the best, else go back
        const unsigned long long len = near_length<NT>(T, S);
        if (len < best_len) {
            for (uint32_t k = threadIdx.x; k < n; k += NT) best[k] = T.id[T.slot(k)];
            best_len = len;
            ++accepted;
        } else {
            for (uint32_t k = threadIdx.x; k < n; k += NT) T.id[k] = best[k];
            __syncthreads();
            near_place<NT>(T, A.xy);
        }
        __syncthreads();
        if (it == A.kicks) break;
        // kick (the same draws as kick_kernel in tour.cu)
        if (A.kick_kind == 1) {
            uint32_t c[3];
            for (int k = 0; k < 3; ++k) c[k] = 1 + uniform_below(rng, n - 1);
            uint32_t t;
            if (c[1] < c[0]) { t = c[0]; c[0] = c[1]; c[1] = t; }
            if (c[2] < c[1]) { t = c[1]; c[1] = c[2]; c[2] = t; }
            if (c[1] < c[0]) { t = c[0]; c[0] = c[1]; c[1] = t; }
            near_double_bridge<NT>(T, c[0], c[1], c[2]);
        } else {
            uint32_t a = uniform_below(rng, n);
            uint32_t b = uniform_below(rng, n);
            if (b < a) { const uint32_t t = a; a = b; b = t; }
            near_move<NT>(T, a, b);
        }
        ++kicks;
        m0 = 0;
    }
    // each CTA writes its share of the tour
    for (uint32_t k = rank * NT + threadIdx.x; k < n; k += ranks * NT) {
        const uint32_t j = T.slot(k);
        const uint32_t id = T.id[j];
        const float2 c = T.xy[j];
        const float e = T.E[T.rev ? T.wrap(j + 1) : j];
        Rg[k] = id;
        Qg[k] = OrderedCity{c.x, c.y, e, 0.f};
        if (ILS) {
            A.route_best[k] = id;
            A.Qbest[k] = OrderedCity{c.x, c.y, e, 0.f};
        }
        if (whole && A.call.out) A.call.out[k] = id;
        if (A.pos) A.pos[id] = k;
    }
    unsigned long long end_len = 0;
    if (whole && A.call.lengths) end_len = near_length<NT>(T, S);
    cluster_barrier();  // no CTA leaves while another may still write to it
    if (rank == 0 && threadIdx.x == 0) {
        if (whole) start_call(st, maxm);
        st->moves = m0 + m;
        st->total_moves += total_m;
        if (!(whole && A.call.step)) st->sweeps += sweeps;
        st->best_key = step_key;
        st->converged = whole && A.call.step ? 0u : 1u;
        if (whole && A.call.lengths) {
            st->start_length = start_len;
            st->length = end_len;
        }
        if (ILS) {
            st->rng = rng;
            st->best_length = best_len;
            st->accepted += accepted;
            st->kicks += kicks;
        }
        if (limit) atomicOr(&st->status, kErrMoveLimit);
        if (bad) atomicOr(&st->status, kErrBadKey);
    }
    if (whole && rank == 0) leave_call(st, A.call.mirror);
}

// ---- neighbour lists of a context ----------------------------------------------
// Counting sort of the cities into the grid's cells, then one thread per city.
__device__ __forceinline__ uint32_t cell_of(const float2 p, const NearGrid& g) {
    return (uint32_t)near_cell(p.y - g.y0, g.inv, g.gy) * (uint32_t)g.gx +
           (uint32_t)near_cell(p.x - g.x0, g.inv, g.gx);
}

__global__ void near_count_kernel(const float2* __restrict__ xy, uint32_t n, NearGrid g,
                                  uint32_t* count) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) atomicAdd(&count[cell_of(xy[v], g)], 1u);
}

// Exclusive scan of count[0 .. cells) into cell[0 .. cells] and back into
// count, by one CTA of 1,024 threads; *crowd (host memory) gets the sum of the
// squared counts.
__global__ void __launch_bounds__(1024) near_scan_kernel(uint32_t* count, uint32_t* cell,
                                                         uint32_t cells,
                                                         unsigned long long* crowd) {
    __shared__ uint32_t part[32];
    __shared__ unsigned long long squares[32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    unsigned long long mine = 0;
    for (uint32_t base = 0; base < cells; base += 1024) {
        const uint32_t c = base + threadIdx.x;
        const uint32_t own = c < cells ? count[c] : 0u;
        mine += (unsigned long long)own * own;
        uint32_t run = own;
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, run, s);
            if (lane >= (uint32_t)s) run += u;
        }
        if (lane == 31) part[warp] = run;
        __syncthreads();
        uint32_t before = carry, all = 0;
        for (uint32_t w = 0; w < 32; ++w) {
            const uint32_t u = part[w];
            before += w < warp ? u : 0u;
            all += u;
        }
        if (c < cells) cell[c] = count[c] = before + run - own;
        carry += all;
        __syncthreads();
    }
    mine = warp_sum_u64(mine);
    if (lane == 0) squares[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        cell[cells] = carry;
        for (uint32_t w = 1; w < 32; ++w) mine += squares[w];
        *(volatile unsigned long long*)crowd = mine;
        __threadfence_system();
    }
}

__global__ void near_scatter_kernel(const float2* __restrict__ xy, uint32_t n, NearGrid g,
                                    uint32_t* count, uint32_t* cellid) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) cellid[atomicAdd(&count[cell_of(xy[v], g)], 1u)] = v;
}

__global__ void near_lists_kernel(const float2* __restrict__ xy, uint32_t n, NearIndex I) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    near_search<uint32_t, kCtxNear>(v, xy, I.g, I.cell, I.cellid,
                                    reinterpret_cast<NearEntry<uint32_t>*>(I.nbr));
    for (uint32_t k = 0; k < kSeedNeighbours; ++k)
        I.seeds[(size_t)v * kSeedNeighbours + k] = I.nbr[(size_t)v * kCtxNear + min(k, n - 2)].x;
}

// Without lists: the seeds alone.
__global__ void near_seeds_kernel(const float2* __restrict__ xy, uint32_t n, NearIndex I) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    float ds[kSeedNeighbours];
    uint32_t vs[kSeedNeighbours];
    near_nearest<uint32_t, kSeedNeighbours>(v, xy, I.g, I.cell, I.cellid, ds, vs);
    for (uint32_t k = 0; k < kSeedNeighbours; ++k)
        I.seeds[(size_t)v * kSeedNeighbours + k] = vs[min(k, n - 2)];
}

void solo_config(uint32_t n, int nt, uint32_t ctas, cudaLaunchConfig_t* cfg,
                 cudaLaunchAttribute* attr, cudaStream_t s) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(ctas);
    cfg->blockDim = dim3((unsigned)nt);
    cfg->dynamicSmemBytes = solo_layout(n).bytes;
    cfg->stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

template <int NT, bool ILS>
int solo_ctas_t(uint32_t n, uint32_t max_n) {
    // the limits are shared by every context: set for the largest n
    if (cudaFuncSetAttribute(near_solo_kernel<NT, ILS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)solo_layout(max_n).bytes) != cudaSuccess ||
        cudaFuncSetAttribute(near_solo_kernel<NT, ILS>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return 0;
    for (uint32_t ctas = solo_wanted_ctas(n); ctas >= 1; ctas /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        solo_config(n, NT, ctas, &cfg, attr, nullptr);
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, near_solo_kernel<NT, ILS>, &cfg) ==
                cudaSuccess &&
            clusters >= 1)
            return (int)ctas;
        cudaGetLastError();
    }
    return 0;
}

template <int NT, bool ILS>
cudaError_t launch_solo_t(const SoloArgs& A, int ctas, cudaStream_t s) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    solo_config(A.n, NT, (uint32_t)ctas, &cfg, attr, s);
    return cudaLaunchKernelEx(&cfg, near_solo_kernel<NT, ILS>, A);
}

constexpr uint32_t kSoloSmallN = 2048;  // 256 threads a CTA up to here, 512 above

}  // namespace

// A CTA per 64 slots (two warps' worth of lists each), up to 16.
uint32_t solo_wanted_ctas(uint32_t n) {
    uint32_t c = 1;
    while (c < kSoloMaxCtas && c * 64 < n) c *= 2;
    return c;
}

int solo_ctas(uint32_t n, bool ils) {
    if (n < 8 || n > kSoloMaxN) return 0;
    if (n <= kSoloSmallN)
        return ils ? solo_ctas_t<256, true>(n, kSoloSmallN) : solo_ctas_t<256, false>(n, kSoloSmallN);
    return ils ? solo_ctas_t<512, true>(n, kSoloMaxN) : solo_ctas_t<512, false>(n, kSoloMaxN);
}

cudaError_t launch_solo(const SoloArgs& A, bool ils, int ctas, cudaStream_t s) {
    if (A.n <= kSoloSmallN)
        return ils ? launch_solo_t<256, true>(A, ctas, s) : launch_solo_t<256, false>(A, ctas, s);
    return ils ? launch_solo_t<512, true>(A, ctas, s) : launch_solo_t<512, false>(A, ctas, s);
}

// Words of the lists, or without them of the seeds; either holds the sort's counters first.
static size_t near_first_words(uint32_t n, bool lists) {
    return std::max<size_t>((size_t)n * (lists ? kCtxNear * 2 : kSeedNeighbours),
                            near_cells_max(n));
}

size_t near_index_words(uint32_t n, bool lists) {
    // lists, cells and their end, cities by cell, seeds
    return near_first_words(n, lists) + near_cells_max(n) + 1 + n +
           (lists ? (size_t)n * kSeedNeighbours : 0);
}

void near_index_carve(NearIndex& I, uint32_t* words, uint32_t n, bool lists) {
    I.nbr = lists ? reinterpret_cast<uint2*>(words) : nullptr;
    I.cell = words + near_first_words(n, lists);
    I.cellid = I.cell + near_cells_max(n) + 1;
    I.seeds = lists ? I.cellid + n : words;
}

cudaError_t launch_near_index(const NearIndex& I, const float2* xy, uint32_t n,
                              unsigned long long* crowd, cudaStream_t s) {
    const uint32_t cells = (uint32_t)I.g.gx * (uint32_t)I.g.gy;
    const uint32_t grid = (n + 255) / 256;
    uint32_t* count = I.nbr ? reinterpret_cast<uint32_t*>(I.nbr) : I.seeds;
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(uint32_t) * cells, s);
    if (e != cudaSuccess) return e;
    near_count_kernel<<<grid, 256, 0, s>>>(xy, n, I.g, count);
    near_scan_kernel<<<1, 1024, 0, s>>>(count, I.cell, cells, crowd);
    near_scatter_kernel<<<grid, 256, 0, s>>>(xy, n, I.g, count, I.cellid);
    if (I.nbr)
        near_lists_kernel<<<(n + 127) / 128, 128, 0, s>>>(xy, n, I);
    else
        near_seeds_kernel<<<(n + 127) / 128, 128, 0, s>>>(xy, n, I);
    return cudaGetLastError();
}

}  // namespace logo
