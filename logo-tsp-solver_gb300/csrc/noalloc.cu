// logo_best_move_noalloc: the best-improvement sweep for callers that must not
// allocate device memory.
//
// Who needs it: callers that account for every device byte in their own pool
// allocator (a framework's caching allocator, a budgeted multi-tenant
// service), and latency-sensitive callers for whom cudaMalloc/cudaFree are off
// limits because those calls can synchronize the whole device.  Such a caller
// allocates the inputs and the output itself and passes device pointers; this
// entry point then launches four kernels on the caller's stream and performs
// no allocation of any kind.
//
// A pair changes the tour by d(i, c) + d(i-1, c-1) - e[i] - e[c], so with the
// bounding boxes of two windows of 32 consecutive cities (each with the city
// before it) and their longest edges most pairs of windows are out at once, and
// of the others only edges with e[i] + e[c] >= -B take part, B being the best
// delta so far.  B is good before the sweep begins: every window's longest edge
// is paired with every other's first.  The sweep is bound by the latency of its
// four dependent launches then, not by the pairs (n = 20,011, clustered, NN tour:
// 128 -> 51 us; a random tour 191 -> 41; a local optimum 128 -> 73; n = 65,536:
// 810 -> 72, random 1,320 -> 62; n = 52: 29.5 -> 26.4).
//
// Its working memory (the tour-ordered cities, the argmin key, the bounding
// box and a status word) lives in one file-scope __device__ array of fixed
// size, logo_noalloc_scratch, sized for LOGO_NOALLOC_MAX_CITIES cities
// (1 MiB plus an 8.25 KiB header).  The array exists once per GPU that loads
// the library and stays allocated until the process exits.  Host code cannot
// use the array's name as a device address, so the first call on each device
// looks the address up with cudaGetSymbolAddress (with that device current)
// and caches it; make that first call before any stream capture.  The cache
// is keyed by the device's current context (its driver-assigned unique id),
// so a call after cudaDeviceReset, which re-creates the primary context and
// with it the array, looks the address up again instead of using the old
// one.
//
// The coordinates are read as 8-byte (x, y) pairs, so coords must be 8-byte
// aligned (any cudaMalloc'd array and any even element offset into one);
// route, out and status_out must be 4-byte aligned.  Misaligned pointers are
// refused on the host with LOGO_ERR_INVALID_ARG before any work is enqueued.
//
// Every call shares the array and the array keeps the previous call's
// contents: each call clears the key, bounding box and status first.  Calls
// whose kernels overlap on the GPU (different streams, or different host
// threads on the same device) race on the array and must be serialised by
// the caller.
#include <cmath>
#include <cstdint>
#include <mutex>

#include <cudaTypedefs.h>

#include "../../include/logo_gpu.h"
#include "logo_device.cuh"
#include "logo_internal.h"
#include "sweep_core.cuh"

namespace {

using namespace logo;

constexpr uint32_t kNoAllocMax = LOGO_NOALLOC_MAX_CITIES;

struct __align__(256) NoAllocHeader {
    unsigned long long key;  // argmin of this call
    unsigned int bbox[4];    // min x, min y, max x, max y as ordered integers
    unsigned int status;     // 0, or LOGO_ERR_INVALID_ARG
    float margin;            // filter margin of the box
    unsigned int done;       // CTAs of the sweep that have finished
    unsigned int seen[kNoAllocMax / 32];  // one bit per city id: permutation check
};

constexpr size_t kScratchBytes =
    sizeof(NoAllocHeader) + sizeof(OrderedCity) * (size_t)kNoAllocMax;

static __device__ __align__(256) unsigned char logo_noalloc_scratch[kScratchBytes];

// float <-> integer whose unsigned order matches the float order
__device__ __forceinline__ unsigned int ordered_bits(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(unsigned int o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

constexpr uint32_t kWindow = 32;
static_assert(kNoAllocMax % kWindow == 0, "the last window's pads lie in the array");

// What the pads of a window's first cities hold.
enum { kMinX, kMinY, kMaxX, kMaxY, kLongest, kLongestAt, kPads };

// Same exactness margin as the library's other sweeps, from the box diagonal.
__device__ __forceinline__ float noalloc_margin(double diag) {
    const double rel = 9.5367431640625e-07;  // 2^-20
    const double u = 5.9604644775390625e-08;  // 2^-24
    return (float)(1.0 + 2.0 * diag * (3.0 * u + rel) + 2.0 * 1.1920928955078125e-07 +
                   3.0 * u * 4.0 * diag + 1.0);
}

__global__ void noalloc_reset(unsigned char* scratch) {
    chain_release();
    NoAllocHeader* h = reinterpret_cast<NoAllocHeader*>(scratch);
    for (uint32_t w = threadIdx.x; w < kNoAllocMax / 32; w += blockDim.x) h->seen[w] = 0u;
    if (threadIdx.x == 0) {
        h->key = kNoMove;
        h->bbox[0] = 0xFFFFFFFFu;
        h->bbox[1] = 0xFFFFFFFFu;
        h->bbox[2] = 0u;
        h->bbox[3] = 0u;
        h->status = 0u;
        h->done = 0u;
    }
}

// Tour-ordered cities with exact incoming edges; bounding box; what the sweep
// wants of every window; route and coordinate checks (out-of-range or repeated
// ids and non-finite coordinates set the status word; out-of-range ids are
// clamped so no access leaves the caller's arrays).  A thread per city.
// (Reset, this and the seeds as one cluster of 8 CTAs save two launches, 1 us at
// n = 52, and cost 9 us at n = 20,011 and 120 us at n = 65,536: too few SMs.)
__global__ void noalloc_prepare(const float2* __restrict__ xy, const uint32_t* __restrict__ route,
                                uint32_t n, unsigned char* scratch) {
    chain_wait();
    chain_release();
    NoAllocHeader* h = reinterpret_cast<NoAllocHeader*>(scratch);
    OrderedCity* Q = reinterpret_cast<OrderedCity*>(scratch + sizeof(NoAllocHeader));
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    if (k - lane >= n) return;  // whole warps
    const bool in = k < n;
    unsigned int v[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u};
    unsigned int longest = 0u;  // (edges are not negative: ordered as integers)
    OrderedCity o{};
    bool bad = false;
    if (in) {
        uint32_t c = route[k], p = route[k == 0 ? n - 1 : k - 1];
        if (c >= n || p >= n) {
            bad = true;
            c = c < n ? c : 0;
            p = p < n ? p : 0;
        } else if (atomicOr(&h->seen[c >> 5], 1u << (c & 31)) & (1u << (c & 31))) {
            bad = true;  // a repeated city id: not a permutation
        }
        const float2 a = xy[c], b = xy[p];
        if (!isfinite(a.x) || !isfinite(a.y)) bad = true;
        o.x = a.x;
        o.y = a.y;
        o.e = (float)exact_dist(b.x, b.y, a.x, a.y);
        v[0] = min(ordered_bits(a.x), ordered_bits(b.x));
        v[1] = min(ordered_bits(a.y), ordered_bits(b.y));
        v[2] = max(ordered_bits(a.x), ordered_bits(b.x));
        v[3] = max(ordered_bits(a.y), ordered_bits(b.y));
        if (k >= 1) longest = __float_as_uint(o.e);  // (no pair has the edge into city 0)
    }
    v[0] = __reduce_min_sync(0xffffffffu, v[0]);
    v[1] = __reduce_min_sync(0xffffffffu, v[1]);
    v[2] = __reduce_max_sync(0xffffffffu, v[2]);
    v[3] = __reduce_max_sync(0xffffffffu, v[3]);
    const unsigned int most = __reduce_max_sync(0xffffffffu, longest);
    const uint32_t at = k - lane + __ffs(__ballot_sync(0xffffffffu, in && longest == most)) - 1;
    if (lane < kLongest) {
        const unsigned int mine = lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : v[3];
        if (lane < kMaxX)
            atomicMin(&h->bbox[lane], mine);
        else
            atomicMax(&h->bbox[lane], mine);
        o.pad = from_ordered(mine);
    } else if (lane == kLongest) {
        o.pad = __uint_as_float(most);
    } else if (lane == kLongestAt) {
        o.pad = __uint_as_float(at);
    }
    if (in)
        Q[k] = o;
    else if (lane < kPads)
        Q[k].pad = o.pad;
    if (bad) atomicExch(&h->status, (unsigned int)LOGO_ERR_INVALID_ARG);
}

// The longest edges of all windows, in pairs: a warp per 32 x 32 windows, a lane
// per row.  Also the margin, and the check of the diagonal (each thread of the
// sweep had worked them out in 64 bits).
constexpr uint32_t kSeedThreads = 128;
__global__ void __launch_bounds__(kSeedThreads) noalloc_seed(uint32_t n, unsigned char* scratch) {
    chain_wait();
    chain_release();
    NoAllocHeader* h = reinterpret_cast<NoAllocHeader*>(scratch);
    const OrderedCity* Q = reinterpret_cast<const OrderedCity*>(scratch + sizeof(NoAllocHeader));
    const uint32_t windows = (n + kWindow - 1) / kWindow, groups = (windows + 31) / 32;
    const uint32_t pair = blockIdx.x * (kSeedThreads / 32) + threadIdx.x / 32;
    const uint32_t lane = threadIdx.x & 31, row = pair / groups, col = pair % groups;
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kSeedThreads - 1) {
        const double dx = (double)from_ordered(h->bbox[2]) - (double)from_ordered(h->bbox[0]);
        const double dy = (double)from_ordered(h->bbox[3]) - (double)from_ordered(h->bbox[1]);
        const double diag = sqrt(dx * dx + dy * dy);
        if (n >= 4 && !(diag < LOGO_MAX_DIAGONAL))  // (three cities have no move, at any distance)
            atomicExch(&h->status, (unsigned int)LOGO_ERR_INVALID_ARG);
        h->margin = noalloc_margin(diag);
    }
    if (row > col || row >= groups) return;  // whole warps
    const uint32_t rw = row * 32 + lane, cw = col * 32 + lane;
    const uint32_t a = rw < windows ? __float_as_uint(Q[rw * kWindow + kLongestAt].pad) : 0u;
    const uint32_t b = cw < windows ? __float_as_uint(Q[cw * kWindow + kLongestAt].pad) : 0u;
    const OrderedCity qa = Q[a], qam = Q[a ? a - 1 : 0], qb = Q[b], qbm = Q[b ? b - 1 : 0];
    uint64_t best = kNoMove;
    for (int o = 0; o < 32; ++o) {
        const uint32_t c = __shfl_sync(0xffffffffu, b, o);
        const float cx = __shfl_sync(0xffffffffu, qb.x, o), cy = __shfl_sync(0xffffffffu, qb.y, o);
        const float ce = __shfl_sync(0xffffffffu, qb.e, o);
        const float px = __shfl_sync(0xffffffffu, qbm.x, o);
        const float py = __shfl_sync(0xffffffffu, qbm.y, o);
        if (a == 0 || c == 0) continue;
        const int delta = exact_dist(qa.x, qa.y, cx, cy) + exact_dist(qam.x, qam.y, px, py) -
                          (int)qa.e - (int)ce;
        const uint32_t i = min(a, c), j = max(a, c);
        if (delta < 0 && j >= i + 2) {
            const uint64_t key = pack_key(delta, i, j);
            best = key < best ? key : best;
        }
    }
    best = warp_min_u64(best);
    if (lane == 0 && best != kNoMove) atomicMin(&h->key, best);
}

constexpr int kR = 4;
constexpr int kNW = 4;
constexpr uint32_t kRowsPerWarp = 32u * kR;           // 128
constexpr uint32_t kRowsPerCta = kRowsPerWarp * kNW;  // 512
constexpr uint32_t kRowWindows = kRowsPerWarp / kWindow;
constexpr uint32_t kColWindowsMost = 32 / kRowWindows;  // a pair of windows per lane

// Windows of columns per CTA: up to 8192 cities the sweep is as long as its
// longest warp, so warps get few (n = 1,000 from an NN tour: 34 us, with 8 windows 41);
// above, what each warp does before its first pair counts.
constexpr uint32_t kColWindowsFew = 2, kFewMax = 8192;

constexpr int kCols = 4;  // columns whose loads are in flight together

// Steps (32 rows and a column) of a warp's tile above which all of it is walked,
// four rows a lane: a step costs 2.4 times what the walk spends on as many pairs.
template <uint32_t COLS>
constexpr uint32_t kWalkStepsOf = kRowWindows * COLS * 10 / 24;

// CTAs of the sweep at most, about two waves; above, each takes several column
// chunks.  (Many CTAs cost more than their work, as they count themselves out on
// one word: n = 65,536 with one chunk each 170 us; half as many CTAs leave too few
// warps for long tiles, n = 20,011 at a local optimum 73 -> 86 us.)
constexpr uint32_t kSweepCtas = 2736;

// grid (group of `chunks` column chunks, row block); groups entirely below the
// diagonal exit, and the last of the `tiles` others leaves the result.
template <uint32_t kColWindows>
__global__ void __launch_bounds__(kNW * 32)
    noalloc_sweep(uint32_t n, uint32_t chunks, uint32_t tiles, unsigned char* scratch,
                  logo_move* out, int32_t* status_out) {
    constexpr uint32_t kColsPerCta = kColWindows * kWindow, kWalkSteps = kWalkStepsOf<kColsPerCta>;
    static_assert(kRowWindows * kColWindows <= 32, "a pair of windows per lane");
    chain_wait();
    NoAllocHeader* h = reinterpret_cast<NoAllocHeader*>(scratch);
    const OrderedCity* Q = reinterpret_cast<const OrderedCity*>(scratch + sizeof(NoAllocHeader));
    __shared__ unsigned long long wbest[kNW];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t row0 = blockIdx.y * kRowsPerCta, group = chunks * kColsPerCta;
    if ((blockIdx.x + 1) * group <= row0) return;
    uint64_t best = kNoMove;
    if (!*(volatile unsigned int*)&h->status) {
        const float margin = h->margin;
        const unsigned long long known = *(volatile unsigned long long*)&h->key;
        int B = known == kNoMove ? -1 : key_delta(known);
        const uint32_t rows = row0 + warp * kRowsPerWarp;
        const uint32_t end = min((blockIdx.x + 1) * group, n);
        for (uint32_t col0 = blockIdx.x * group; col0 < end; col0 += kColsPerCta) {
            if (col0 + kColsPerCta <= rows) continue;
            // a lane per pair of windows
            const uint32_t r0 = rows + lane / kColWindows * kWindow;
            const uint32_t c0 = col0 + lane % kColWindows * kWindow;
            float er = 0.f, ec = 0.f;  // their longest edges
            bool hit = false;
            if (lane < kRowWindows * kColWindows && r0 < n && c0 < n && c0 >= r0) {
                const OrderedCity *R = Q + r0, *C = Q + c0;
                er = R[kLongest].pad;
                ec = C[kLongest].pad;
                const float dx = fmaxf(fmaxf(C[kMinX].pad - R[kMaxX].pad, R[kMinX].pad - C[kMaxX].pad),
                                       0.f);
                const float dy = fmaxf(fmaxf(C[kMinY].pad - R[kMaxY].pad, R[kMinY].pad - C[kMaxY].pad),
                                       0.f);
                // (the two new edges, rounded, are no shorter than 2 d less 1 and the
                // rounding of the differences, squares and roots)
                const float d = sqrtf(dx * dx + dy * dy) * (1.f - 4e-6f);
                hit = 2.f * d - 4.f <= er + ec + (float)B;
            }
            const uint32_t hits = __ballot_sync(0xffffffffu, hit);
            uint32_t steps = 0;
            if (__popc(hits) * kWindow > kWalkSteps) {
                for (uint32_t t = 0; t < 32; ++t) {
                    if (!(hits >> t & 1u)) continue;
                    const uint32_t c = col0 + t % kColWindows * kWindow + lane;
                    const float e = __shfl_sync(0xffffffffu, er, t);
                    steps += __popc(__ballot_sync(
                        0xffffffffu, c < n && Q[min(c, n - 1)].e + e + (float)B >= 0.f));
                }
            }
            if (steps > kWalkSteps) {
                const uint32_t ib = rows + lane * kR;
                RowBlock<kR> rb;
                load_rows<kR>(rb, Q, ib, n);
                refresh_thresholds<kR>(rb, Q, ib, n, B, margin);
                walk_columns<kR>(rb, Q, 0, col0, min(col0 + kColsPerCta, n), ib, n, Q, margin, B,
                                 best);
            } else {
                for (uint32_t g = 0; g < kRowWindows; ++g) {
                    uint32_t left = hits >> (g * kColWindows) & ((1u << kColWindows) - 1u);
                    if (left == 0) continue;
                    const uint32_t i = rows + g * kWindow + lane;
                    const bool row = i >= 1 && i + 3 <= n;
                    const OrderedCity q = Q[min(i, n - 1)], qm = Q[row ? i - 1 : 0];
                    const float longest =  // (any pair that is in has read it)
                        __shfl_sync(0xffffffffu, er, g * kColWindows + __ffs(left) - 1);
                    for (; left; left &= left - 1) {
                        const uint32_t w = __ffs(left) - 1;
                        const float e = __shfl_sync(0xffffffffu, ec, g * kColWindows + w);
                        if (!__any_sync(0xffffffffu, row && q.e + e + (float)B >= 0.f)) continue;
                        const uint32_t first = col0 + w * kWindow, c = first + lane;
                        uint32_t cols = __ballot_sync(
                            0xffffffffu,
                            c >= 1 && c < n && Q[min(c, n - 1)].e + longest + (float)B >= 0.f);
                        while (cols) {  // kCols at a time, at the end the last one again
                            uint32_t j[kCols];
                            OrderedCity p[kCols], pm[kCols];
#pragma unroll
                            for (int u = 0; u < kCols; ++u) {
                                j[u] = cols ? first + __ffs(cols) - 1 : j[u ? u - 1 : 0];
                                cols &= cols - 1;
                                p[u] = Q[j[u]];
                                pm[u] = Q[j[u] - 1];
                            }
#pragma unroll
                            for (int u = 0; u < kCols; ++u) {
                                const float v = approx_dist(q.x, q.y, p[u].x, p[u].y) +
                                                (approx_dist(qm.x, qm.y, pm[u].x, pm[u].y) - p[u].e);
                                if (row && j[u] >= i + 2 && v < (float)(B + (int)q.e) + margin) {
                                    const int delta = exact_dist(q.x, q.y, p[u].x, p[u].y) +
                                                      exact_dist(qm.x, qm.y, pm[u].x, pm[u].y) -
                                                      (int)q.e - (int)p[u].e;
                                    if (delta <= B) {
                                        const uint64_t key = pack_key(delta, i, j[u]);
                                        best = key < best ? key : best;
                                        B = delta;
                                    }
                                }
                            }
                        }
                        B = __reduce_min_sync(0xffffffffu, B);
                    }
                }
            }
        }
    }
    best = warp_min_u64(best);
    if (lane == 0) wbest[warp] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long m = wbest[0];
        for (int w = 1; w < kNW; ++w) m = wbest[w] < m ? wbest[w] : m;
        if (m != kNoMove) atomicMin(&h->key, m);
        __threadfence();
        if (atomicAdd(&h->done, 1u) == tiles - 1) {
            __threadfence();
            const unsigned int status = *(volatile unsigned int*)&h->status;
            const unsigned long long k = *(volatile unsigned long long*)&h->key;
            logo_move move{};
            if (!status && k != kNoMove) {
                move.i = key_i(k);
                move.j = key_j(k);
                move.minchange = key_delta(k);
            }
            *out = move;
            if (status_out) *status_out = (int32_t)status;
        }
    }
}

// The scratch array's device address per device, with the id of the context
// it was looked up in (0: not looked up yet).
struct ScratchAddr {
    unsigned long long ctx_id;
    void* ptr;
};
std::mutex g_mu;
ScratchAddr g_scratch[64] = {};
PFN_cuCtxGetCurrent_v4000 g_ctx_current = nullptr;
PFN_cuCtxGetId_v12000 g_ctx_id = nullptr;
bool g_ctx_fns_tried = false;

// Unique id of the calling thread's current context; 0 if the driver cannot
// tell, in which case the address is looked up on every call.
unsigned long long current_ctx_id() {
    if (!g_ctx_fns_tried) {
        g_ctx_fns_tried = true;
        cudaDriverEntryPointQueryResult q1, q2;
        void* f1 = nullptr;
        void* f2 = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 4000, cudaEnableDefault,
                                             &q1) == cudaSuccess &&
            q1 == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault,
                                             &q2) == cudaSuccess &&
            q2 == cudaDriverEntryPointSuccess) {
            g_ctx_current = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(f1);
            g_ctx_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(f2);
        }
    }
    if (!g_ctx_current || !g_ctx_id) return 0ull;
    CUcontext ctx = nullptr;
    unsigned long long id = 0ull;
    if (g_ctx_current(&ctx) != CUDA_SUCCESS || !ctx) return 0ull;
    if (g_ctx_id(ctx, &id) != CUDA_SUCCESS) return 0ull;
    return id;
}

}  // namespace

extern "C" logo_status logo_best_move_noalloc(const logo_xy* coords, const uint32_t* route,
                                              uint32_t n, logo_move* out, int32_t* status_out,
                                              void* stream) {
    if (!coords || !route || !out) return LOGO_ERR_INVALID_ARG;
    if (n < 3 || n > kNoAllocMax) return LOGO_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(coords) & 7u) || (reinterpret_cast<uintptr_t>(route) & 3u) ||
        (reinterpret_cast<uintptr_t>(out) & 3u) || (reinterpret_cast<uintptr_t>(status_out) & 3u))
        return LOGO_ERR_INVALID_ARG;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return LOGO_ERR_NO_DEVICE;
    if (dev >= 64) return LOGO_ERR_INVALID_ARG;
    void* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        const unsigned long long id = current_ctx_id();
        ScratchAddr& a = g_scratch[dev];
        if (!a.ptr || id == 0ull || a.ctx_id != id) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, logo_noalloc_scratch) != cudaSuccess || !p)
                return LOGO_ERR_CUDA;
            a.ptr = p;
            a.ctx_id = id;
        }
        scratch = a.ptr;
    }
    cudaStream_t s = (cudaStream_t)stream;
    unsigned char* sc = static_cast<unsigned char*>(scratch);
    const bool few = n <= kFewMax;
    const uint32_t cols = (few ? kColWindowsFew : kColWindowsMost) * kWindow;
    const uint32_t rows = (n + kRowsPerCta - 1) / kRowsPerCta;
    uint32_t chunks = 1, tiles = 0;
    dim3 grid;
    for (;; chunks *= 2) {
        grid = dim3((n + cols * chunks - 1) / (cols * chunks), rows);
        tiles = 0;
        for (uint32_t y = 0; y < rows; ++y) tiles += grid.x - y * kRowsPerCta / (cols * chunks);
        if (tiles <= kSweepCtas) break;
    }
    const float2* xy = reinterpret_cast<const float2*>(coords);
    const uint32_t groups = ((n + kWindow - 1) / kWindow + 31) / 32;
    constexpr uint32_t kPairs = kSeedThreads / 32;
    noalloc_reset<<<1, 256, 0, s>>>(sc);
    if (launch_chained(noalloc_prepare, (n + 255) / 256, 256, 0, s, xy, route, n, sc) !=
            cudaSuccess ||
        launch_chained(noalloc_seed, (groups * groups + kPairs - 1) / kPairs, kSeedThreads, 0, s,
                       n, sc) != cudaSuccess ||
        launch_chained(few ? noalloc_sweep<kColWindowsFew> : noalloc_sweep<kColWindowsMost>, grid,
                       kNW * 32, 0, s, n, chunks, tiles, sc, out, status_out) != cudaSuccess)
        return LOGO_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? LOGO_OK : LOGO_ERR_CUDA;
}
