// Host-side declarations shared by the translation units of liblogo_gpu.so.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/logo_gpu.h"
#include "logo_device.cuh"
#include "near_grid.h"

namespace logo {

// Programmatic dependent launches for the step chain (see chain_wait in
// logo_device.cuh) when launched on a stream; inside stream capture (the
// descent and ILS graphs, whose launches the graph already pipelines) the
// launches stay ordinary.  Measured on GB300 at n = 100k: a step launched
// on a stream 0.0769 -> 0.0730 ms (the sweep's three launches 0.0642 ->
// 0.0604 ms); captured descents unchanged with the exhaustive search and
// 15 % slower with the neighbour search.  Off when the environment sets
// LOGO_CHAINED_LAUNCH=0.
bool chained_launch_enabled();
template <typename... KArgs, typename... Args>
cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                           cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) cap = cudaStreamCaptureStatusActive;
    cfg.numAttrs = chained_launch_enabled() && cap == cudaStreamCaptureStatusNone ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// ---- single-instance sweep (sweep.cu) ---------------------------------------
struct SweepLaunch {
    const OrderedCity* Q0;
    const OrderedCity* Q1;
    uint32_t n;
    const uint2* tiles;  // (row0, col0) per CTA
    uint32_t ntiles;
    uint32_t cb;         // columns per tile
    int R, NW;           // rows per thread, warps per CTA
    int variant;         // LOGO_SWEEP_* (0 MUFU, 4 fused, 5 local, 6 boxed; 1-3 retired)
    float margin;        // filter margin M
    DevState* st;
    // boxed variant (6): per 32-column window (columns 3 + 32g ..) its coordinate
    // bounding box and largest edge (sweep_windows(n) entries), the same per
    // 32-row window (rows 1 + 32g .., sweep_row_windows(n) entries), the list
    // of (tile, column-window mask) that pass the window test (ntiles entries)
    // and its three counters (tiles listed from the start, claimed, listed from the end)
    float4* wbox;
    float* wmax;
    float4* rbox;
    float* rmax;
    uint4* work;         // ntiles entries
    uint32_t* workctl;   // tiles listed from the start, claimed, listed from the end
    // boxed variant: the tour's city ids (both buffers), the tour position of
    // every city (kept by every kernel that moves the tour) and the nearest
    // kSeedNeighbours cities of each (NearIndex), whose pairs seed the sweep's best
    // delta
    const uint32_t* R0;
    const uint32_t* R1;
    uint32_t* pos;
    const uint32_t* nbr;
};
constexpr uint32_t kSeedNeighbours = 5;
// k nearest other cities of every city, out[v * k + j] (construct.cpp).
void knn_grid(const ::logo_xy* p, uint32_t n, uint32_t k, uint32_t* out);
// Windows of the boxed variant: columns 3 + 32 g .. 3 + 32 g + 31 (< n) and
// rows 1 + 32 g .. 1 + 32 g + 31 (rows with pairs: i + 3 <= n).
__host__ __device__ inline uint32_t sweep_windows(uint32_t n) {
    return n < 4 ? 1 : (n - 3 + 31) / 32;
}
__host__ __device__ inline uint32_t sweep_row_windows(uint32_t n) {
    return n < 4 ? 1 : (n - 3 + 31) / 32;
}
// The boxed variant needs tile widths that are multiples of 32 (tile column
// starts are then 3 + 32k) and at most 1024 (one mask bit per window).
inline bool sweep_cols_supported(int variant, uint32_t cb) {
    return variant != 6 || (cb % 32 == 0 && cb <= 1024);
}
cudaError_t launch_sweep(const SweepLaunch& L, cudaStream_t s);
// Sets the kernel attributes of L's shape; call before any stream capture.
cudaError_t launch_sweep_prepare(const SweepLaunch& L);
bool sweep_shape_supported(int R, int NW, int variant);
size_t sweep_smem_bytes(uint32_t cb);

struct CoopSync;  // coop.cu's grid barrier and key slots (below)

// ---- neighbour-list search (neighbour.cu) ------------------------------------
struct NbrLaunch {
    const OrderedCity* Q0;
    const OrderedCity* Q1;
    const uint32_t* R0;
    const uint32_t* R1;
    OrderedCity* Q0w;     // the same buffers, writable (the cooperative phase moves the tour)
    OrderedCity* Q1w;
    uint32_t* R0w;
    uint32_t* R1w;
    uint32_t* pos;        // tour position of every city (exact: kept by every tour move)
    const uint32_t* nbr;  // K nearest other cities per city, nearest first
    uint32_t K;
    uint32_t n;
    DevState* st;
    bool oropt;           // also the Or-opt candidates (into st->or_key)
    float margin;         // filter_margin of the instance (Or-opt estimate test)
};
// Default and largest neighbour-list length of LOGO_SEARCH_NEIGHBOUR.
constexpr uint32_t kSearchNeighbours = 8, kSearchNeighboursMax = 16;
// One neighbour sweep: the lowest improving candidate key into st->best_key
// (the apply kernel then moves or marks convergence), st->nbr_sweeps += 1.
cudaError_t launch_nbr_sweep(const NbrLaunch& L, cudaStream_t s);
// Recomputes pos from the current tour.
cudaError_t launch_fill_pos(const NbrLaunch& L, cudaStream_t s);
// The whole neighbour phase of a descent as one cooperative launch
// (coop.cu): moves until no candidate improves or st->max_moves; cs->arrived
// must be 0 or what a launch of as many CTAs left.  coop_nbr_grid: its CTAs
// for this n (0: cooperative launches unavailable).
int coop_nbr_grid(uint32_t n, bool oropt, int device);
cudaError_t launch_coop_nbr(const NbrLaunch& L, CoopSync* cs, int grid, cudaStream_t s);

// ---- tour maintenance (tour.cu) --------------------------------------------
struct TourBufs {
    OrderedCity* Q[2];
    uint32_t* route[2];
    OrderedCity* Qbest;
    uint32_t* route_best;
    const float2* xy;
    uint32_t n;
    DevState* st;
    uint32_t* seen;  // n words: number of the last route load that met each city
    // tour position of every city (boxed sweep's seed pass; null otherwise),
    // kept current by every kernel that moves the tour
    uint32_t* pos;
};
// Neighbours per city in a context's lists: few walks run off 40 (counted on
// the CPU, slots whose list is too short per sweep of the descent with 16 and
// with 32: n = 1,000 from the NN tour 12.5 and 3.5, n = 6,000 clustered 105
// and 34, after a kick at n = 1,500 4.8 and 1.4).
constexpr uint32_t kCtxNear = 40;
// Neighbour lists and search grid of a context's cities (near_tour.cuh),
// built on the device once per context.
struct NearIndex {
    uint2* nbr;  // kCtxNear entries per city: city, squared distance (near_tour.cuh)
    uint32_t* cell;
    uint32_t* cellid;
    uint32_t* seeds;  // kSeedNeighbours per city: the lists' first cities (sweep.cu)
    NearGrid g;
};
// 32-bit words behind nbr (null without lists), cell, cellid and seeds.
size_t near_index_words(uint32_t n, bool lists);
void near_index_carve(NearIndex& I, uint32_t* words, uint32_t n, bool lists);  // words 8-byte aligned
// *crowd (pinned host memory): over all cities, the cities of its cell, summed.
cudaError_t launch_near_index(const NearIndex& I, const float2* xy, uint32_t n,
                              unsigned long long* crowd, cudaStream_t s);

// A whole call as one launch: the route is loaded (and checked) by the launch
// itself, and its state and result are left in host memory.
struct WholeCall {
    const uint32_t* src;   // the caller's route, or a device copy of it; null: the resident tour
    uint32_t* out;         // where the resulting tour also goes (null: nowhere)
    DevState* mirror;      // pinned host memory: *st as the launch leaves it
    unsigned long long max_moves;
    uint32_t* seen;        // grid-wide launch: the last load that met each city
    uint32_t epoch;        // number of this load (see launch_load_route)
    bool step;             // one sweep, no move: its key stays in st->best_key
    bool lengths;          // also st->start_length and st->length
};

// One cluster runs a whole descent, or a whole ILS call, of a tour of 8 to
// kSoloMaxN cities (solo.cu).
constexpr uint32_t kSoloMaxN = 6144;
struct SoloArgs {
    OrderedCity* Q0;
    OrderedCity* Q1;
    uint32_t* R0;
    uint32_t* R1;
    uint32_t n;
    DevState* st;
    const float2* xy;  // coordinates by city id
    NearIndex near;
    // ILS only: the best tour (also the start: route_best/Qbest and
    // st->best_length are set before the launch), the kick count and kind
    OrderedCity* Qbest;
    uint32_t* route_best;
    uint32_t kicks;
    int kick_kind;
    WholeCall call;  // descents only
    uint32_t* pos;   // tour position of every city, where the context keeps it
};
// CTAs of the cluster for this n on the current device (0: not available).
uint32_t solo_wanted_ctas(uint32_t n);
int solo_ctas(uint32_t n, bool ils);
// Without ils: a descent to a local optimum or st->max_moves.  With ils:
// descent, length, accept/revert and kicks for A.kicks kicks
// (ILSGlobalSolverSequential::optimize with a kick count).
cudaError_t launch_solo(const SoloArgs& A, bool ils, int ctas, cudaStream_t s);

// A descent or an ILS call of a larger tour as one cooperative launch over the
// whole device (grid_tour.cu): one CTA per SM.
constexpr uint32_t kGridMaxCtas = 256;
constexpr uint32_t kGridWide = 1024, kGridTakers = 8192;
constexpr uint32_t kGridDisc = 4096;  // cities of a disc that one CTA goes through
constexpr uint32_t kGridDiscs = 4096;  // discs put off that are listed
constexpr uint32_t kGridSpread = 50000;  // default of GridArgs::spread (see grid_tour.cu)
struct GridSync {
    unsigned long long arrived;    // barrier arrivals so far
    unsigned long long length[2];  // tour length of the descent in hand, by its parity
    unsigned long long start_length;
    unsigned long long bad;        // the route is not a permutation
    uint32_t left;  // CTAs that have left a whole call
    // by the sweep's parity, read with one load: edges put off, whether the launch is to
    // end after the sweep's move, slots whose discs are put off; and edges that can take
    // part in pairs with those put off (more of each may have been offered than fit)
    struct __align__(16) {
        uint32_t wides, pause, discs, takers;
    } put[2];
    // (set to zero up to here before a launch)
    unsigned long long keys[2][kGridMaxCtas];  // best key per CTA, by the sweep's parity
    unsigned long long wide_keys[2][kGridMaxCtas];  // best key per CTA after those put off
    uint32_t wide[2][kGridWide];
    uint32_t taker[kGridTakers];
    uint32_t most_wides, most_takers, most_discs;  // largest counts of a sweep of the last launch
};
struct GridArgs {
    SoloArgs solo;  // pos: slot of every city meanwhile
    GridSync* gs;
    uint32_t* disc_list;  // kGridDiscs for each of the two parities
    // limits, at most (a test's are smaller) kGridWide, kGridTakers, kGridDisc, kGridDiscs
    uint32_t wide, takers, disc, discs;
    uint32_t spread;  // tours above as many cities have their large discs dealt to all CTAs
    unsigned long long quantum_ns;  // a launch that has run for longer ends after its next move
};
// Default of quantum_ns: how long other work on the device (another context's call, a
// serving round) waits for one launch.  Going on costs a launch, the tour's way into
// the ring and back, and a first sweep without the last one's seeds (every 2 ms 6 %, every
// 20 ms 0.2 % of an ILS call at n = 20,000).
constexpr unsigned long long kGridQuantumNs = 20000000ull;
// CTAs of the launch (0: n is not above kSoloMaxN, or not available).  The state it
// leaves is not converged when it paused: the next launch goes on from it (of an ILS
// call in the middle of a descent, after st->kicks kicks).
int near_grid_ctas(uint32_t n, int device);
cudaError_t launch_near_grid(const GridArgs& A, bool ils, int ctas, cudaStream_t s);

// State of a cooperative launch (coop.cu).
// A CTA's best candidate of a sweep: its order (NbrPick in coop.cu), and the cities
// of the list entry it came from.
struct CoopBest {
    unsigned long long lo;
    uint32_t hi, city, near, pad;
};
struct CoopSync {
    unsigned long long arrived;  // barrier arrivals so far; 0 before the first launch
    CoopBest best[2][kGridMaxCtas];  // by the sweep's parity
};
// One CTA waits at the cooperative grid barrier sized for two (test hook).
cudaError_t launch_barrier_probe(CoopSync* cs, DevState* st, cudaStream_t s);

// Loads a tour from src (a host buffer the device reads in place, or a
// device copy) into route[0] and Q[0], with pos and the permutation check
// (st->bad_route = 1 if src is not a permutation of 0..n-1; `epoch` must
// differ from every value seen holds, i.e. count loads from 1 with seen
// zeroed at the start and on wrap-around); cur = 0.  With reset_moves != 0
// also what launch_reset_descent(reset_moves) does.
cudaError_t launch_load_route(const TourBufs& T, const uint32_t* src, uint32_t epoch,
                              unsigned long long reset_moves, cudaStream_t s);
// Writes the current tour (best: the ILS best) to dst (host buffer written
// in place, or device memory).
cudaError_t launch_store_route(const TourBufs& T, uint32_t* dst, bool best, cudaStream_t s);
// Prepares *st for a new descent: cur = 0 kept, counters cleared.
cudaError_t launch_reset_descent(const TourBufs& T, unsigned long long max_moves,
                                 cudaStream_t s);
// Applies the move in st->best_key (or marks convergence); with out, also
// writes the resulting current tour there (moved or not).
cudaError_t launch_apply_move(const TourBufs& T, cudaStream_t s, uint32_t* out = nullptr);
// The same for the neighbour search with Or-opt moves: the best of
// st->best_key and st->or_key[].
cudaError_t launch_apply_nbr_move(const TourBufs& T, cudaStream_t s);
// After a converged neighbour phase: continue the same descent (moves and
// limit kept) with full sweeps, unless it stopped on an error or the limit.
cudaError_t launch_resume_descent(const TourBufs& T, cudaStream_t s);
// st->length = length of the current tour.
cudaError_t launch_tour_length(const TourBufs& T, cudaStream_t s);
// ILS pieces.
cudaError_t launch_kick(const TourBufs& T, int kind, cudaStream_t s);
cudaError_t launch_accept(const TourBufs& T, cudaStream_t s);
cudaError_t launch_save_best(const TourBufs& T, cudaStream_t s);
// Kick of the kind in st->kick_kind.
inline cudaError_t launch_kick_dev(const TourBufs& T, cudaStream_t s) { return launch_kick(T, -1, s); }
// Set the WHILE conditions of the device-run ILS graph (see tour.cu).
cudaError_t launch_descent_cond(DevState* st, cudaGraphConditionalHandle h, bool first,
                                cudaStream_t s);
cudaError_t launch_kick_cond(DevState* st, cudaGraphConditionalHandle h, bool first,
                             cudaStream_t s);

// logo_ctx_create; without lists the context takes 320 bytes a city less and runs
// the graph-driven descents, which need none.
logo_status create_context(int device, const logo_xy* coords, uint32_t n, bool lists,
                           logo_ctx** out);

// Upper bound of |exact delta - approximate delta| for coordinates whose
// bounding-box diagonal is `diag` (see filter_margin in capi.cu).
float filter_margin(double diag);

}  // namespace logo
