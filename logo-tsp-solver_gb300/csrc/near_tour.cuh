// A tour as a ring of slots and the exact best-improvement sweep over its near
// neighbours: held by one CTA's shared memory in the batched solver (batch.cu) and
// the serving rounds (serve.cu), by each CTA of a cluster (solo.cu), and by global
// memory where the whole device shares it (grid_tour.cu).
//
// What bounds it.  A local search is a chain of sweeps, each followed by one
// move, so a CTA is as fast as one sweep's latency.  Walking all n^2/2 pairs
// (even with whole windows skipped) made that latency grow with n^2; here a
// sweep looks only at the pairs that can be the best move.
//
// Which pairs those are.  A pair of tour edges f = (a, b), g = (c, d) has
//     delta = [D(b, d) - |f|] + [D(a, c) - |g|]
// in whole numbers (D the exact per-edge distance, D(b, d) and D(a, c) the two
// new edges, b and d the later ends).  If delta <= B, one bracket is at most
// floor(B / 2).  So with h = floor(B / 2), every pair with delta <= B is met by
// looking, from the later end of each edge, for cities within D <= |f| + h, and
// from the earlier end of each edge likewise (each pair once: from the later
// end of the edge with the lower index, from the earlier end of the other).  B
// is the best delta met so far (at first -1), so the pairs that tie with the
// final best are all met and the packed key's minimum is the exact lowest
// (delta, i, j).  A pair's delta is also at least -2 min(|f|, |g|) - 3 by the
// triangle inequality and the rounding of four distances, so an edge with
// 2 |f| + 8 < -B cannot take part and its ends are not looked at.
//
// How they are found.  Each city has its kNearK nearest cities in order of the
// squared distance s as sweeps compute it; the walk along the list ends at the
// first s > (|f| + h + 1)^2 (a city at or beyond it has a distance above
// |f| + h + 0.5 even after rounding: coordinates are below 2e6 apart, so s and
// its root are off by less than 0.25).  A walk that reaches the end of the list
// goes on as a search of the cell grid in a disc of that radius by the whole
// warp.  Counted on the CPU (n = 1,000 uniform, random start tour, 16
// neighbours): 2.0 list entries a city and sweep, 16 discs a sweep in the
// descent and 1.4 after a kick, against 498,501 pairs.
//
// The tour is a ring: slot j holds a city, E[j] is the exact length of the
// edge between slots j - 1 and j, and (o, rev) say which slot is position 0
// and in which direction positions count.  A move
//     new = old[p..q) ++ rev(old[0..p)) ++ rev(old[q..n))
// (src/solvers/twoOptLocalSolver.cpp:41-48; the kick is the same permutation,
// src/solvers/ILSGlobalSolver.cpp:37-48) keeps the cyclic order but for one
// arc, so it reverses the shorter of [p, q) and its complement in place and
// changes (o, rev): on average under 0.15 n slots are written instead of n.
// Positions matter only where the reference lets them: in the tie rule and in
// the closing edge (n - 1, 0), which is never part of a pair.
//
// Shared memory of a CTA that has the lists there too: 51 bytes a city (209 KB at the
// largest, n = 4,096); the best tour of an iterated search stays in global memory.
#pragma once
#include <cstdint>

#include "logo_device.cuh"
#include "near_grid.h"

namespace logo {

constexpr uint32_t kNearK = 16;       // neighbours per list of a CTA's instance
constexpr uint32_t kNearMaxN = 4096;  // largest instance one CTA holds
// Warps per SM that kernels over NearTour are compiled for (64 registers a
// thread): a sweep is a chain of dependent shared-memory reads, so an SM is
// kept busy by the other CTAs on it.
constexpr int kNearWarpsPerSm = 32;
constexpr uint32_t kNoSeed = 0xFFFFFFFFu;
constexpr float kNoEdge = -2.7e8f;    // stands for an edge that takes part in nothing

// Byte offsets of the arrays, for an instance of n cities.
struct NearLayout {
    uint32_t xy, e, nbr, id, pos, cell, cellid, bytes;
};
__host__ __device__ constexpr uint32_t near_pad16(uint32_t b) { return (b + 15u) & ~15u; }
__host__ __device__ constexpr NearLayout near_layout(uint32_t n) {
    NearLayout l{};
    l.nbr = 0;                                               // uint16[n][kNearK]
    l.xy = l.nbr + 2 * kNearK * n;                           // float2[n]
    l.e = near_pad16(l.xy + 8 * n);                          // float[n]
    l.id = near_pad16(l.e + 4 * n);                          // uint16[n]
    l.pos = near_pad16(l.id + 2 * n);                        // uint16[n]
    l.cellid = near_pad16(l.pos + 2 * n);                    // uint16[n]
    l.cell = near_pad16(l.cellid + 2 * n);                   // uint16[cells + 1]
    l.bytes = near_pad16(l.cell + 2 * (near_cells_max(n) + 1));
    return l;
}

// The squared distance whose rounded root the per-edge distance is
// (exact_dist in logo_device.cuh).
__device__ __forceinline__ float near_sq(float2 a, float2 b) {
    const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y);
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
}
// Lengths are whole numbers below 2^21 kept in binary32: sums of four are exact,
// and nothing on the way needs a conversion.
__device__ __forceinline__ float near_len(float s) {
    return truncf(__fadd_rn(__fsqrt_rn(s), 0.5f));
}
__device__ __forceinline__ float near_dist(float2 a, float2 b) { return near_len(near_sq(a, b)); }

// An entry of a neighbour list.  In global memory it carries its squared distance,
// so that an entry out of reach costs one dependent read, not three; in shared
// memory, where reads are quick and room is short, it does not.
template <typename IX>
struct NearEntry {
    IX id;
};
template <>
struct __align__(8) NearEntry<uint32_t> {
    uint32_t id;
    float s;
};

// IX: what a city or slot number is stored as (uint16_t where all arrays are in
// one CTA's shared memory, else uint32_t); KN: neighbours per list.
template <typename IX, uint32_t KN>
struct NearTour {
    static_assert(KN == 16 || KN == 40, "near_sweep goes over 8 entries and 8 or 32 more");
    using Index = IX;
    static constexpr uint32_t kList = KN;
    uint32_t n;
    uint32_t o;     // slot of position 0
    bool rev;       // positions count downwards
    bool whole;     // the lists hold every other city
    uint32_t kc;    // entries per list
    float2* xy;     // by slot
    float* E;       // by slot: the length of the edge between slots j - 1 and j
    IX* id;     // city in slot j
    IX* pos;    // slot of city v
    NearEntry<IX>* nbr;
    IX* cell;    // first entry of every cell in cellid (row major), and the end
    IX* cellid;  // cities by cell
    NearGrid g;

    __device__ __forceinline__ uint32_t wrap(uint32_t j) const { return j >= n ? j - n : j; }
    // slot of position k < n
    __device__ __forceinline__ uint32_t slot(uint32_t k) const {
        return rev ? (o >= k ? o - k : o + n - k) : wrap(o + k);
    }
    // position index of the edge in E[j] (its later end's position; 0 = closing edge)
    __device__ __forceinline__ uint32_t edge_index(uint32_t j) const {
        if (!rev) return j >= o ? j - o : j + n - o;
        const uint32_t t = o + 1;  // (o + 1 - j) mod n
        return t >= j ? (t - j == n ? 0u : t - j) : t + n - j;
    }
    // squared distance of the last entry of the list of the city in slot j
    __device__ __forceinline__ float last_sq(uint32_t j) const {
        const NearEntry<IX> e = nbr[id[j] * KN + KN - 1];
        if constexpr (sizeof(IX) == 4)
            return e.s;
        else
            return near_sq(xy[j], xy[pos[e.id]]);
    }
    // where E holds the closing edge
    __device__ __forceinline__ uint32_t closing() const { return rev ? wrap(o + 1) : o; }
};

constexpr uint32_t kNearFar = 256;   // discs of a sweep's CTA that may wait for their warps
constexpr uint32_t kNearWide = 64;   // discs that may be put off again, to the whole CTA
constexpr uint32_t kNearDisc = 256;  // cities that a warp goes through of a disc

// MAXC: CTAs that share the sweeps (a cluster, each with its own copy of the tour).
template <int NT, int MAXC, typename IX>
struct NearShared {
    static constexpr int kKeys = MAXC * (NT / 32);
    unsigned long long wbest[2][kKeys];  // best key of every warp, by the sweep's parity
    unsigned long long part[NT / 32];
    float red[4][NT / 32];
    uint32_t scan[NT / 32];
    // by the sweep's parity: best delta met, entries of far and wide (more may
    // have been offered than fit)
    int bound[2], far_bound[2];  // (of its lists, and of its discs)
    uint32_t fars[2], big[2], huges[2];
    IX far[kNearFar];         // slots whose lists were too short
    IX wide[kNearWide];       // those of them whose discs are large
    IX huge[kNearWide];       // and those too large for one CTA
    // each warp's slots in hand: slot, its city, its longer edge
    struct Slots {
        IX j[32], id[32], open[32];
        float m[32];
    } slots[NT / 32];
    // each warp's pairs of slots that are in reach of one another: slot, slot of
    // the other city (uint32_t: the other city), squared distance
    struct Reach {
        IX j[64], p[64];
        float s[64];
    } reach[NT / 32];
    uint32_t idx;
    unsigned int flag, seq;

    __device__ __forceinline__ void reset(uint32_t parity) {
        bound[parity] = far_bound[parity] = -1;
        fars[parity] = big[parity] = huges[parity] = 0;
    }
    // once per instance, between barriers: sweeps (parity from 0) leave the counters of
    // one parity as they are
    __device__ __forceinline__ void init() {
        if (threadIdx.x < 2) reset(threadIdx.x);
    }
};

// The cities at the ends of a new edge of a pair that was nearly the best in
// the last sweep, one pair per lane (the same in every warp).
struct NearSeed {
    uint32_t a = 0, b = 0;  // a == b: none
};

using CtaTour = NearTour<uint16_t, kNearK>;
__device__ __forceinline__ CtaTour near_carve(unsigned char* smem, uint32_t n) {
    const NearLayout l = near_layout(n);
    CtaTour T;
    T.n = n;
    T.o = 0;
    T.rev = false;
    T.kc = n - 1 < kNearK ? n - 1 : kNearK;
    T.whole = n - 1 <= kNearK;
    T.xy = reinterpret_cast<float2*>(smem + l.xy);
    T.E = reinterpret_cast<float*>(smem + l.e);
    T.id = reinterpret_cast<uint16_t*>(smem + l.id);
    T.pos = reinterpret_cast<uint16_t*>(smem + l.pos);
    T.nbr = reinterpret_cast<NearEntry<uint16_t>*>(smem + l.nbr);
    T.cell = reinterpret_cast<uint16_t*>(smem + l.cell);
    T.cellid = reinterpret_cast<uint16_t*>(smem + l.cellid);
    return T;
}

// Cell column (or row) of a coordinate u counted from the box's corner:
// monotone in u, clamped to the grid.  (Differences from the corner are below
// 2e6 and good to 0.12 wherever the box lies; the coordinates themselves may be
// much larger.)
__device__ __forceinline__ int near_cell(float u, float inv, int cells) {
    const int c = (int)fminf(fmaxf(u * inv, 0.f), 1.0e6f);
    return c < cells ? c : cells - 1;
}

// ---- the search grid and the neighbour lists ---------------------------------
// City v's KN nearest cities from the filled cells, by one thread: rings of
// cells around its own, until the nearest are certain (after ring r every city
// nearer than r cells has been seen; a little less, for rounding).
template <typename IX, uint32_t KN>
__device__ __forceinline__ void near_nearest(uint32_t v, const float2* __restrict__ gxy,
                                             const NearGrid& g, const IX* cell, const IX* cellid,
                                             float (&ds)[KN], uint32_t (&vs)[KN]) {
    const float2 p = gxy[v];
    const int cx = near_cell(p.x - g.x0, g.inv, g.gx), cy = near_cell(p.y - g.y0, g.inv, g.gy);
#pragma unroll
    for (uint32_t k = 0; k < KN; ++k) {
        ds[k] = INFINITY;
        vs[k] = v;
    }
    const int rings = max(max(cx, g.gx - 1 - cx), max(cy, g.gy - 1 - cy));
    for (int r = 0; r <= rings; ++r) {
        const float sure = (float)(r - 1) * g.side * 0.999f;  // rings below r are done
        if (r >= 1 && ds[KN - 1] < sure * sure) break;
        for (int yy = max(cy - r, 0); yy <= min(cy + r, g.gy - 1); ++yy) {
            const bool edge_row = yy == cy - r || yy == cy + r;
            for (int part = 0; part < 2; ++part) {
                // whole row of the ring, or its two end cells
                int xa, xb;
                if (edge_row) {
                    if (part) break;
                    xa = max(cx - r, 0);
                    xb = min(cx + r, g.gx - 1);
                } else {
                    xa = xb = part ? cx + r : cx - r;
                    if (xa < 0 || xa >= g.gx) continue;
                }
                const uint32_t a = cell[yy * g.gx + xa], b = cell[yy * g.gx + xb + 1];
                for (uint32_t k = a; k < b; ++k) {
                    const uint32_t u = cellid[k];
                    if (u == v) continue;
                    float d = near_sq(p, gxy[u]);
                    if (d >= ds[KN - 1]) continue;
                    uint32_t c = u;
#pragma unroll
                    for (uint32_t q = 0; q < KN; ++q) {
                        const bool less = d < ds[q];
                        const float td = ds[q];
                        const uint32_t tv = vs[q];
                        ds[q] = less ? d : td;
                        vs[q] = less ? c : tv;
                        d = less ? td : d;
                        c = less ? tv : c;
                    }
                }
            }
        }
    }
}
// The same as city v's list.
template <typename IX, uint32_t KN>
__device__ void near_search(uint32_t v, const float2* __restrict__ gxy, const NearGrid& g,
                            const IX* cell, const IX* cellid, NearEntry<IX>* nbr) {
    float ds[KN];
    uint32_t vs[KN];
    near_nearest<IX, KN>(v, gxy, g, cell, cellid, ds, vs);
#pragma unroll
    for (uint32_t k = 0; k < KN; ++k) {
        NearEntry<IX> e;
        e.id = (IX)vs[k];
        if constexpr (sizeof(IX) == 4) e.s = ds[k];
        nbr[(size_t)v * KN + k] = e;
    }
}

// Once per instance of a CTA: bounding box, counting sort of the cities into
// cells, then one thread per city.  The list area serves as the sort's 32-bit
// counters first.
template <int NT, typename SH>
__device__ void near_build(CtaTour& T, SH& S, const float2* __restrict__ gxy) {
    const uint32_t n = T.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        const float2 p = gxy[v];
        x0 = fminf(x0, p.x);
        x1 = fmaxf(x1, p.x);
        y0 = fminf(y0, p.y);
        y1 = fmaxf(y1, p.y);
    }
    for (int s = 16; s; s >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, s));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, s));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, s));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, s));
    }
    if (lane == 0) {
        S.red[0][warp] = x0;
        S.red[1][warp] = x1;
        S.red[2][warp] = y0;
        S.red[3][warp] = y1;
    }
    __syncthreads();
    for (int w = 0; w < NT / 32; ++w) {
        x0 = fminf(x0, S.red[0][w]);
        x1 = fmaxf(x1, S.red[1][w]);
        y0 = fminf(y0, S.red[2][w]);
        y1 = fmaxf(y1, S.red[3][w]);
    }
    T.g = near_grid(n, x0, y0, x1 - x0, y1 - y0);
    const NearGrid g = T.g;
    const uint32_t cells = (uint32_t)(g.gx * g.gy);
    uint32_t* count = reinterpret_cast<uint32_t*>(T.nbr);  // cells <= n / 2 + 64 words
    for (uint32_t c = threadIdx.x; c < cells; c += NT) count[c] = 0;
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        const float2 p = gxy[v];
        atomicAdd(&count[near_cell(p.y - y0, g.inv, g.gy) * g.gx + near_cell(p.x - x0, g.inv, g.gx)],
                  1u);
    }
    __syncthreads();
    // exclusive scan: each thread a run of cells, then the threads' sums
    const uint32_t per = (cells + NT - 1) / NT;
    const uint32_t c0 = min(threadIdx.x * per, cells), c1 = min(c0 + per, cells);
    uint32_t sum = 0;
    for (uint32_t c = c0; c < c1; ++c) sum += count[c];
    uint32_t run = sum;
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, run, s);
        if (lane >= (uint32_t)s) run += u;
    }
    if (lane == 31) S.scan[warp] = run;
    __syncthreads();
    uint32_t before = run - sum;
    for (uint32_t k = 0; k < warp; ++k) before += S.scan[k];
    for (uint32_t c = c0; c < c1; ++c) {
        const uint32_t k = count[c];
        T.cell[c] = (uint16_t)before;
        count[c] = before;
        before += k;
    }
    if (threadIdx.x == 0) T.cell[cells] = (uint16_t)n;
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        const float2 p = gxy[v];
        const uint32_t c =
            near_cell(p.y - y0, g.inv, g.gy) * g.gx + near_cell(p.x - x0, g.inv, g.gx);
        T.cellid[atomicAdd(&count[c], 1u)] = (uint16_t)v;
    }
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < n; v += NT)
        near_search<uint16_t, kNearK>(v, gxy, g, T.cell, T.cellid, T.nbr);
    __syncthreads();
}

// ---- the tour -------------------------------------------------------------------
// Slot k = position k = id[k] (already written): coordinates, slots of cities,
// edges.
template <int NT, typename TOUR>
__device__ __forceinline__ void near_place(TOUR& T, const float2* __restrict__ gxy) {
    T.o = 0;
    T.rev = false;
    for (uint32_t k = threadIdx.x; k < T.n; k += NT) {
        const uint32_t v = T.id[k];
        T.xy[k] = gxy[v];
        T.pos[v] = (typename TOUR::Index)k;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < T.n; k += NT)
        T.E[k] = near_dist(T.xy[k == 0 ? T.n - 1 : k - 1], T.xy[k]);
    __syncthreads();
}

// Length of the tour (routeLength, src/headers.h:170-189); every thread has it.
template <int NT, typename TOUR, typename SH>
__device__ __forceinline__ unsigned long long near_length(const TOUR& T, SH& S) {
    unsigned long long s = 0;
    for (uint32_t k = threadIdx.x; k < T.n; k += NT) s += (unsigned long long)T.E[k];
    s = warp_sum_u64(s);
    if ((threadIdx.x & 31) == 0) S.part[threadIdx.x >> 5] = s;
    __syncthreads();
    s = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) s += S.part[w];
    __syncthreads();
    return s;
}

// Reverses the arc of len slots from slot u (len < n), by `threads` threads of
// which this is number `tid`.  Slots and the inner edges swap pairwise, the two
// outer edges get their new lengths from the thread that holds the arc's ends.
// A barrier of all of them must follow.
template <typename TOUR>
__device__ __forceinline__ void near_reverse(TOUR& T, uint32_t u, uint32_t len, uint32_t tid,
                                             uint32_t threads) {
    const uint32_t n = T.n;
    if (len == 0) return;
    for (uint32_t t = tid; t < (len + 1) / 2; t += threads) {
        const uint32_t a = T.wrap(u + t), b = T.wrap(u + len - 1 - t);
        const float2 pa = T.xy[a], pb = T.xy[b];
        if (t == 0) {
            T.E[a] = near_dist(T.xy[a == 0 ? n - 1 : a - 1], pb);
            T.E[T.wrap(b + 1)] = near_dist(pa, T.xy[T.wrap(b + 1)]);
        }
        const typename TOUR::Index va = T.id[a], vb = T.id[b];
        T.xy[a] = pb;
        T.xy[b] = pa;
        T.id[a] = vb;
        T.id[b] = va;
        T.pos[vb] = (typename TOUR::Index)a;
        T.pos[va] = (typename TOUR::Index)b;
    }
    for (uint32_t t = tid + 1; 2 * t < len; t += threads) {
        const uint32_t a = T.wrap(u + t), b = T.wrap(u + len - t);
        const float ea = T.E[a], eb = T.E[b];
        T.E[a] = eb;
        T.E[b] = ea;
    }
}

// Reverses positions [a, b) in place.
template <typename TOUR>
__device__ __forceinline__ void near_reverse_positions(TOUR& T, uint32_t a, uint32_t b,
                                                       uint32_t tid, uint32_t threads) {
    if (b > a) near_reverse(T, T.rev ? T.slot(b - 1) : T.slot(a), b - a, tid, threads);
}

// new = old[p..q) ++ rev(old[0..p)) ++ rev(old[q..n)), p <= q < n; a barrier of
// all threads must follow.
template <typename TOUR>
__device__ __forceinline__ void near_move(TOUR& T, uint32_t p, uint32_t q, uint32_t tid,
                                          uint32_t threads) {
    const uint32_t n = T.n, len = q - p;
    if (2 * len <= n) {
        // reversed arc [p, q), read the other way round from its far end
        const uint32_t first = T.slot(p), last = T.slot(q == 0 ? n - 1 : q - 1);
        near_reverse(T, T.rev ? last : first, len, tid, threads);
        T.o = last;
        T.rev = !T.rev;
    } else {
        // the complement: positions q .. n - 1, 0 .. p - 1
        const uint32_t o = T.slot(p);
        near_reverse(T, T.rev ? T.slot(p == 0 ? n - 1 : p - 1) : T.slot(q), n - len, tid, threads);
        T.o = o;
    }
}
template <int NT, typename TOUR>
__device__ __forceinline__ void near_move(TOUR& T, uint32_t p, uint32_t q) {
    near_move(T, p, q, threadIdx.x, NT);
    __syncthreads();
}

// new = old[0,p1) old[p2,p3) old[p1,p2) old[p3,n): three reversals in place, with
// a barrier of all threads after each.
template <typename TOUR, typename BAR>
__device__ __forceinline__ void near_double_bridge(TOUR& T, uint32_t p1, uint32_t p2, uint32_t p3,
                                                   uint32_t tid, uint32_t threads, BAR barrier) {
    near_reverse_positions(T, p1, p3, tid, threads);
    barrier();
    const uint32_t m = p1 + (p3 - p2);
    near_reverse_positions(T, p1, m, tid, threads);
    barrier();
    near_reverse_positions(T, m, p3, tid, threads);
    barrier();
}
template <int NT, typename TOUR>
__device__ __forceinline__ void near_double_bridge(TOUR& T, uint32_t p1, uint32_t p2,
                                                   uint32_t p3) {
    near_double_bridge(T, p1, p2, p3, threadIdx.x, NT, [] { __syncthreads(); });
}

// ---- the sweep --------------------------------------------------------------------
// (V + 1)^2: above it a squared distance stands for more than V; -1 for V < 0.
__device__ __forceinline__ float near_limit(float V) {
    const float l = V + 1.f;
    return V < 0.f ? -1.f : l * l;
}
__device__ __forceinline__ float near_half(float B) { return floorf(0.5f * B); }

// ---- clusters: another CTA's shared memory, and the barrier of all CTAs ----------
__device__ __forceinline__ void cluster_store(unsigned long long* p, uint32_t cta, uint64_t v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(p)), "r"(cta));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t* p, uint32_t cta, uint32_t v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(p)), "r"(cta));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(v) : "memory");
}
// (the aligned form wants whole warps: a loop or branch before it may have left the
// warp's threads apart)
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                     : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_ctas() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

struct NearBest {
    uint64_t key;  // this lane's best pair
    float B;       // best delta its warp met, at most -1 (the same in every lane)
};

// The pair of the edges in E[f] and E[g], neither the closing edge, with new
// edges of squared lengths s and s2; true when it lowers the bound.  The test
// in front of the two square roots lets every pair with delta <= B through:
// the approximate root is within 2^-20 of the true one (2 at most), a rounded
// distance within 0.7, so D2 <= B + ef + eg - D1 implies
// sqrt(s2) <= B + ef + eg - approx + 3.4.
template <typename TOUR>
__device__ __forceinline__ bool near_pair(const TOUR& T, uint32_t f, uint32_t g, float s,
                                          float s2, float ef, float eg, NearBest& nb,
                                          float& lowest) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    const float t = (nb.B + ef + eg + 4.f) - r;
    if (t < 0.f || s2 > t * t) return false;
    const float delta = near_len(s) + near_len(s2) - ef - eg;
    if (delta > nb.B) return false;
    const uint32_t i = T.edge_index(f), c = T.edge_index(g);
    const uint64_t key = pack_key((int)delta, min(i, c), max(i, c));
    nb.key = key < nb.key ? key : nb.key;
    lowest = fminf(lowest, delta);
    return true;
}

// The warp's bound after lanes met pairs.
__device__ __forceinline__ void near_share(NearBest& nb, bool met, float lowest) {
    if (__any_sync(0xffffffffu, met))
        nb.B = (float)__reduce_min_sync(0xffffffffu, (int)fminf(nb.B, lowest));
}

// A city in slot p at squared distance s from the city in slot j: a later
// slot may meet the edge before j (both later ends), an earlier one the edge
// after j (both earlier ends); the last slot's next edge is E[0], so it may
// also do the latter.  True when the bound was lowered.
template <typename TOUR>
__device__ __forceinline__ bool near_meet(const TOUR& T, bool in, uint32_t j, uint32_t p,
                                          float s, float ej, float en, uint32_t z,
                                          NearBest& nb, float& lowest) {
    const uint32_t n = T.n, jn = T.wrap(j + 1);
    const float h = near_half(nb.B);
    const bool later = p > j;
    const uint32_t f = later ? j : jn, g = later ? p : p + 1;
    const float ef = later ? ej : en;
    bool met = false;
    if (in && p != j && (later || jn != 0) && g != z && s <= near_limit(ef + h))
        met = near_pair(T, f, g, s,
                        near_sq(T.xy[later ? (j == 0 ? n - 1 : j - 1) : jn], T.xy[later ? p - 1 : g]),
                        ef, T.E[g], nb, lowest);
    if (in && p == n - 1 && later && z != 0 && s <= near_limit(en + h))
        met |= near_pair(T, jn, 0, s, near_sq(T.xy[jn], T.xy[0]), en, T.E[0], nb, lowest);
    return met;
}

// Whether the disc of slot j under bound B has more than `most` cities (as near_far
// sees it); the whole warp, j and B the same in every lane.
template <typename TOUR>
__device__ __forceinline__ bool near_large(const TOUR& T, uint32_t j, uint32_t z, uint32_t most,
                                           float B) {
    const uint32_t jn = T.wrap(j + 1);
    const float ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
    const float V = fmaxf(ej, en) + near_half(B), r = V + 2.f;
    if (V < 0.f) return false;
    const float ux = T.xy[j].x - T.g.x0, uy = T.xy[j].y - T.g.y0;
    const int xa = near_cell(ux - r, T.g.inv, T.g.gx), xb = near_cell(ux + r, T.g.inv, T.g.gx);
    const int ya = near_cell(uy - r, T.g.inv, T.g.gy), yb = near_cell(uy + r, T.g.inv, T.g.gy);
    if (2u * (uint32_t)((xb - xa + 1) * (yb - ya + 1)) > most) return true;
    uint32_t held = 0;
    for (int y = ya + (int)(threadIdx.x & 31); y <= yb; y += 32)
        held += T.cell[y * T.g.gx + xb + 1] - T.cell[y * T.g.gx + xa];
    return __reduce_add_sync(0xffffffffu, held) > most;
}

// A slot whose list was too short, looked at by the whole warp: the grid's
// cells in the disc that bound B gives, of whose cities this warp takes part
// `part` of `parts` (B has to be the same in all of those warps: they number the
// disc's cities alike).  j, most, B and nb.B are the same in every lane: the warp
// goes through the cells together.  A disc of more than `most` cities, or of as many
// cells as hold `most` on average, is left alone, and the result is true.  (The
// cities are counted: where a few cities far from the rest stretch the box, one
// cell may hold nearly all of them.)
template <typename TOUR>
__device__ __forceinline__ bool near_far(const TOUR& T, uint32_t j, uint32_t z,
                                         uint32_t most, float B, NearBest& nb,
                                         uint32_t part = 0, uint32_t parts = 1) {
    const uint32_t lane = threadIdx.x & 31, jn = T.wrap(j + 1);
    const float ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
    const float V = fmaxf(ej, en) + near_half(B);
    if (V < 0.f) return false;
    const float2 p = T.xy[j];
    const float r = V + 2.f, lim = near_limit(V);
    const float ux = p.x - T.g.x0, uy = p.y - T.g.y0;
    const int xa = near_cell(ux - r, T.g.inv, T.g.gx), xb = near_cell(ux + r, T.g.inv, T.g.gx);
    const int ya = near_cell(uy - r, T.g.inv, T.g.gy), yb = near_cell(uy + r, T.g.inv, T.g.gy);
    if (2u * (uint32_t)((xb - xa + 1) * (yb - ya + 1)) > most) return true;
    // up to 32 rows of cells, one per lane: each a run of cellid
    uint32_t first = 0, len = 0;
    auto row_of = [&](int y) {
        first = len = 0;
        if (y <= yb) {
            first = T.cell[y * T.g.gx + xa];
            len = T.cell[y * T.g.gx + xb + 1] - first;
        }
    };
    row_of(ya + (int)lane);
    if (most != ~0u) {
        uint32_t held = len;
        for (int y = ya + 32 + (int)lane; y <= yb; y += 32)
            held += T.cell[y * T.g.gx + xb + 1] - T.cell[y * T.g.gx + xa];
        if (__reduce_add_sync(0xffffffffu, held) > most) return true;
    }
    for (int y0 = ya; y0 <= yb; y0 += 32) {
        if (y0 != ya) row_of(y0 + (int)lane);
        uint32_t end = len;
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, end, s);
            if (lane >= (uint32_t)s) end += u;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
        for (uint32_t t0 = part * 32; t0 < total; t0 += parts * 32) {
            const uint32_t t = t0 + lane;
            // the row of entry t: the first whose end is above t
            uint32_t row = 0;
#pragma unroll
            for (int s = 16; s; s >>= 1) {
                const uint32_t e = __shfl_sync(0xffffffffu, end, row + s - 1);
                if (e <= t) row += s;
            }
            const uint32_t rf = __shfl_sync(0xffffffffu, first, row);
            const uint32_t rb = __shfl_sync(0xffffffffu, end - len, row);
            const uint32_t q = t < total ? T.pos[T.cellid[rf + (t - rb)]] : j;
            const float s = near_sq(p, T.xy[q]);
            float lowest = 0.f;
            const bool met = near_meet(T, s <= lim, j, q, s, ej, en, z, nb, lowest);
            near_share(nb, met, lowest);
        }
    }
    return false;
}

// Pairs in reach wait in the warp's queue until there is one for every lane.
template <typename TOUR, typename SH>
struct NearQueue {
    const TOUR& T;
    typename SH::Reach& q;
    NearBest& nb;
    uint32_t z;
    uint32_t count = 0;

    // SETS times 32 of the queue's last entries, fewer at the end
    template <int SETS>
    __device__ __forceinline__ void take() {
        const uint32_t lane = threadIdx.x & 31;
        uint32_t j[SETS], p[SETS];
        float s[SETS];
        bool in[SETS];
        const uint32_t from = count > 32u * SETS ? count - 32u * SETS : 0u;
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            const uint32_t t = from + 32 * u + lane;
            in[u] = t < count;
            j[u] = q.j[in[u] ? t : 0];
            p[u] = q.p[in[u] ? t : 0];
            s[u] = q.s[in[u] ? t : 0];
        }
        if constexpr (sizeof(typename TOUR::Index) == 4) {
#pragma unroll
            for (int u = 0; u < SETS; ++u) p[u] = T.pos[p[u]];
        }
        bool met = false;
        float lowest = 0.f;
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            const uint32_t jn = T.wrap(j[u] + 1);
            const float ej = j[u] == z ? kNoEdge : T.E[j[u]], en = jn == z ? kNoEdge : T.E[jn];
            met |= near_meet(T, in[u], j[u], p[u], s[u], ej, en, z, nb, lowest);
        }
        near_share(nb, met, lowest);
        count = from;
        __syncwarp();
    }
    __device__ __forceinline__ void add(bool in, uint32_t j, uint32_t p, float s) {
        const uint32_t lane = threadIdx.x & 31;
        const uint32_t votes = __ballot_sync(0xffffffffu, in);
        if (votes == 0) return;
        if (in) {
            const uint32_t t = count + __popc(votes & ((1u << lane) - 1u));
            q.j[t] = (typename TOUR::Index)j;
            q.p[t] = (typename TOUR::Index)p;
            q.s[t] = s;
        }
        count += __popc(votes);
        __syncwarp();
        if (count > 32) take<1>();
    }
    __device__ __forceinline__ void rest() {
        if (count) take<1>();
    }
};

// The pairs of `count` edges with the edges of 32 slots, a lane per slot g (in: g
// is a slot whose edge can take part), whole warps.
template <typename TOUR>
__device__ __forceinline__ void near_edges(const TOUR& T, const typename TOUR::Index* edges,
                                           uint32_t count, bool in, uint32_t g, uint32_t z,
                                           NearBest& nb) {
    if (!__any_sync(0xffffffffu, in)) return;
    const uint32_t n = T.n, gs = in ? g : 0;
    const float2 head = T.xy[gs], tail = T.xy[gs == 0 ? n - 1 : gs - 1];
    const float eg = T.E[gs];
    bool met = false;
    float lowest = 0.f;
    for (uint32_t o = 0; o < count; ++o) {
        const uint32_t f = edges[o];
        if (in && f != g && f != z)
            met |= near_pair(T, f, g, near_sq(T.xy[f], head),
                             near_sq(T.xy[f == 0 ? n - 1 : f - 1], tail), T.E[f], eg, nb, lowest);
    }
    near_share(nb, met, lowest);
}

// Entries FIRST .. FIRST + WIDTH - 1 of the lists of `count` of the warp's slots
// (slots w.open[0 .. count), or with FIRST == 0 all), a lane per entry and
// 32 / WIDTH slots at a time (a long list keeps no other slot waiting), SETS
// times that many in flight.  Pairs in reach go to the queue; the slots whose
// entries were all in reach are left in w.open, and their number is returned.
template <uint32_t FIRST, uint32_t WIDTH, int SETS, typename TOUR, typename SLOTS, typename QUEUE>
__device__ __forceinline__ uint32_t near_lists(const TOUR& T, SLOTS& w, uint32_t count,
                                               QUEUE& queue, const NearBest& nb) {
    using IX = typename TOUR::Index;
    constexpr uint32_t PER = 32 / WIDTH;
    const uint32_t lane = threadIdx.x & 31, k = FIRST + lane % WIDTH;
    uint32_t open = 0;
    for (uint32_t t0 = 0; t0 < count; t0 += PER * SETS) {
        uint32_t i[SETS], j[SETS], p[SETS];
        float s[SETS];
        bool in[SETS];
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            const uint32_t t = t0 + PER * u + lane / WIDTH;
            in[u] = t < count && k < T.kc;
            i[u] = FIRST == 0 ? min(t, count - 1) : w.open[min(t, count - 1)];
            j[u] = w.j[i[u]];
            const NearEntry<IX> e = T.nbr[w.id[i[u]] * TOUR::kList + (in[u] ? k : 0)];
            if constexpr (sizeof(IX) == 4) {
                p[u] = e.id;
                s[u] = e.s;
            } else {
                p[u] = T.pos[e.id];
            }
        }
        const float h = near_half(nb.B);
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            if constexpr (sizeof(IX) != 4) s[u] = near_sq(T.xy[j[u]], T.xy[p[u]]);
            in[u] = in[u] && s[u] <= near_limit(w.m[i[u]] + h);
        }
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            // open <= t0 + PER * u: entries still to be read are not written
            const uint32_t ends =
                __ballot_sync(0xffffffffu, in[u] && lane % WIDTH == WIDTH - 1);
            if (ends >> lane & 1u) w.open[open + __popc(ends & ((1u << lane) - 1u))] = (IX)i[u];
            open += __popc(ends);
            queue.add(in[u], j[u], p[u], s[u]);
        }
        __syncwarp();
    }
    return open;
}

// One best-improvement sweep; the packed key of the best move (kNoMove if
// none).  parity alternates from sweep to sweep (it names the counters).
//
// near_scan is the sweep of one CTA's share: the slots are dealt to the warps of
// `ranks` CTAs, of which this is number `rank`; each lane's best key comes back.
// With ALL_EDGES (a tour in shared memory) large discs are replaced by the whole
// tour's edges.
//
// 1. Each warp re-evaluates the best pairs that the warps met in the last
//    sweep, where their cities are now: real pairs of this tour, and most of
//    them still nearly the best, so the bound is good from the start.
// 2. A warp takes up to 32 slots at a time, drops those whose edges are too
//    short to take part, and goes through the lists of the others.
// 3. Slots whose lists were too short are dealt to the CTA's warps, a disc
//    each, or a part of one where there are fewer discs than warps.  They wait
//    until every list has been looked at because a disc costs what its radius
//    says and the radius shrinks with the bound, which the CTA's warps share.
// 4. Large discs are put off to all warps of the CTA, which take a part each
//    (those beyond `huge` stay in S.huge for the caller), or with ALL_EDGES go
//    over the edges that can take part instead (long edges of a tour far from a
//    local optimum: the bound is large then, and most edges too short).  With LEAVE
//    they stay in S.wide for the caller.
template <int NT, bool ALL_EDGES, bool LEAVE = false, typename TOUR, typename SH>
__device__ __forceinline__ uint64_t near_scan(const TOUR& T, SH& S, const NearSeed& seed,
                                              uint32_t parity, uint32_t rank, uint32_t ranks,
                                              uint32_t huge = ~0u) {
    using IX = typename TOUR::Index;
    constexpr int NW = NT / 32;
    const uint32_t n = T.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t z = T.closing();
    NearBest nb{kNoMove, -1.f};
    {
        bool met = false;
        float lowest = 0.f;
        if (seed.a != seed.b) {
            const uint32_t a = T.pos[seed.a], b = T.pos[seed.b];
            const uint32_t an = T.wrap(a + 1), bn = T.wrap(b + 1);
            const float s = near_sq(T.xy[a], T.xy[b]);
            if (a != z && b != z)
                met = near_pair(T, a, b, s,
                                near_sq(T.xy[a == 0 ? n - 1 : a - 1], T.xy[b == 0 ? n - 1 : b - 1]),
                                T.E[a], T.E[b], nb, lowest);
            if (an != z && bn != z)
                met |= near_pair(T, an, bn, s, near_sq(T.xy[an], T.xy[bn]), T.E[an], T.E[bn], nb,
                                 lowest);
        }
        near_share(nb, met, lowest);
    }
    auto& w = S.slots[warp];
    NearQueue<TOUR, SH> queue{T, S.reach[warp], nb, z};
    // the bound that the CTA's warps share
    auto exchange = [&] {
        const float shared = (float)*(volatile int*)&S.bound[parity];
        if (lane == 0 && nb.B < shared) atomicMin(&S.bound[parity], (int)nb.B);
        nb.B = __shfl_sync(0xffffffffu, fminf(nb.B, shared), 0);
    };
    auto put_off = [&](uint32_t j) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&S.big[parity], 1u);
        at = __shfl_sync(0xffffffffu, at, 0);
        if (at >= kNearWide)
            near_far(T, j, z, ~0u, nb.B, nb);  // no room to wait
        else if (lane == 0)
            S.wide[at] = (IX)j;
    };
    // slots per warp and turn: as even as eights allow
    constexpr uint32_t kMost = 32;
    const uint32_t warps = NW * ranks, turns = (n + kMost * warps - 1) / (kMost * warps);
    const uint32_t turn = ((n + turns * warps - 1) / (turns * warps) + 7u) & ~7u;
    for (uint32_t base = (warp * ranks + rank) * turn; base < n; base += warps * turn) {
        const uint32_t j = base + lane;
        bool take = false;
        float m = 0.f;
        if (lane < turn && j < n) {
            const uint32_t jn = T.wrap(j + 1);
            const float ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
            m = fmaxf(ej, en);
            take = 2.f * m + 8.f >= -nb.B;
        }
        const uint32_t votes = __ballot_sync(0xffffffffu, take);
        if (votes == 0) continue;
        if (take) {
            const uint32_t t = __popc(votes & ((1u << lane) - 1u));
            w.j[t] = (IX)j;
            w.id[t] = T.id[j];
            w.m[t] = m;
        }
        __syncwarp();
        uint32_t open = near_lists<0, 8, 2>(T, w, __popc(votes), queue, nb);
        if (open) {
            if constexpr (TOUR::kList == 16)
                open = near_lists<8, 8, 1>(T, w, open, queue, nb);
            else
                open = near_lists<8, 32, ALL_EDGES ? 2 : 4>(T, w, open, queue, nb);
        }
        queue.rest();
        if (open && !T.whole) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&S.fars[parity], open);
            at = __shfl_sync(0xffffffffu, at, 0);
            if (lane < open && at + lane < kNearFar) S.far[at + lane] = w.j[w.open[lane]];
            for (uint32_t o = at < kNearFar ? kNearFar - at : 0u; o < open; ++o)
                near_far(T, w.j[w.open[o]], z, ~0u, nb.B, nb);  // no room to wait
            __syncwarp();
        }
        exchange();
    }
    __syncthreads();
    const uint32_t fars = min(S.fars[parity], kNearFar);  // the same for every thread
    const float list_bound = (float)S.bound[parity];     // likewise: final since the barrier
    nb.B = fminf(nb.B, list_bound);
    if (fars) {
        uint32_t parts = 1;
        while (2 * parts * fars <= NW) parts *= 2;
        for (uint32_t t = warp / parts; t < fars; t += NW / parts) {
            const uint32_t j = S.far[t], jn = T.wrap(j + 1);
            const float ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
            const float m = fmaxf(ej, en);
            // still too short a list?
            if (2.f * m + 8.f < -nb.B || T.last_sq(j) > near_limit(m + near_half(nb.B))) continue;
            const uint32_t part = warp % parts;
            // (part 0 decides for all parts: the size depends on list_bound alone)
            if (near_far(T, j, z, parts * kNearDisc, list_bound, nb, part, parts) && part == 0)
                put_off(j);
        }
        if (lane == 0 && nb.B < list_bound) atomicMin(&S.far_bound[parity], (int)nb.B);
    }
    __syncthreads();
    if (LEAVE) return nb.key;
    const uint32_t big = min(S.big[parity], kNearWide);  // the same for every thread
    const float bound = fminf(list_bound, (float)S.far_bound[parity]);
    nb.B = fminf(nb.B, bound);
    if (!ALL_EDGES) {
        // (alike in all warps: the size depends on `bound` alone)
        for (uint32_t o = 0; o < big; ++o)
            if (near_far(T, S.wide[o], z, huge, bound, nb, warp, NW) && threadIdx.x == 0)
                S.huge[S.huges[parity]++] = S.wide[o];
    } else if (big) {
        for (uint32_t base = warp * 32; base < n; base += NT) {  // whole warps
            const uint32_t g = base + lane;
            const bool take = g < n && g != z && 2.f * T.E[g] + 8.f >= -nb.B;
            if (!__any_sync(0xffffffffu, take)) continue;
            const uint32_t gs = min(g, n - 1);
            const float2 head = T.xy[gs], tail = T.xy[gs == 0 ? n - 1 : gs - 1];
            const float eg = T.E[gs];
            for (uint32_t o = 0; o < big; ++o) {
                // later edges can only meet the edge before j (at their later
                // ends), the others only the edge after j (at their earlier ends)
                const uint32_t j = S.wide[o], jn = T.wrap(j + 1);
                const bool later = g > j;
                const uint32_t f = later ? j : jn;
                const float s = near_sq(T.xy[j], later ? head : tail);
                const float ef = f == z ? kNoEdge : T.E[f];
                bool met = false;
                float lowest = 0.f;
                if (take && (later || jn > g) && s <= near_limit(ef + near_half(nb.B)))
                    met = near_pair(T, f, g, s,
                                    later ? near_sq(T.xy[j == 0 ? n - 1 : j - 1], tail)
                                          : near_sq(T.xy[jn], head),
                                    ef, eg, nb, lowest);
                near_share(nb, met, lowest);
            }
        }
    }
    return nb.key;
}

// A lane's share of the warps' keys and its seed for the next sweep; the best
// key, in every lane.
template <typename TOUR>
__device__ __forceinline__ uint64_t near_pick(const TOUR& T, const unsigned long long* keys,
                                              uint32_t count, NearSeed& seed) {
    uint64_t k = kNoMove;
    for (uint32_t w = threadIdx.x & 31; w < count; w += 32) {
        const uint64_t o = *(volatile const unsigned long long*)&keys[w];
        k = o < k ? o : k;
    }
    seed.a = seed.b = 0;
    if (k != kNoMove) {
        seed.a = T.id[T.slot(key_i(k))];
        seed.b = T.id[T.slot(key_j(k))];
    }
    return warp_min_u64(k);
}

// The sweep of one CTA, or of a cluster (CL) whose CTAs all hold the same tour:
// the warps leave their best keys in every CTA's shared memory, and one cluster
// barrier closes the sweep.
template <int NT, bool CL, typename TOUR, typename SH>
__device__ __forceinline__ uint64_t near_sweep(const TOUR& T, SH& S, NearSeed& seed,
                                               uint32_t parity, uint32_t rank = 0,
                                               uint32_t ranks = 1) {
    constexpr int NW = NT / 32;
    const uint32_t lane = threadIdx.x & 31, mine = rank * NW + (threadIdx.x >> 5);
    if (T.n < 4) return kNoMove;
    const uint64_t best = warp_min_u64(near_scan<NT, true>(T, S, seed, parity, rank, ranks));
    if constexpr (CL) {
        if (lane < ranks) cluster_store(&S.wbest[parity][mine], lane, best);
    } else {
        if (lane == 0) S.wbest[parity][mine] = best;
    }
    if (threadIdx.x == 0) S.reset(parity ^ 1);  // the next sweep's
    if constexpr (CL) {
        cluster_barrier();
    } else {
        __syncthreads();
    }
    return near_pick(T, S.wbest[parity], ranks * NW, seed);
}

}  // namespace logo
