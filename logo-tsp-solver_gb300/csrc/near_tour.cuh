// A whole instance held by one CTA (shared memory) and the exact
// best-improvement sweep over its near neighbours.  Used by the batched solver
// (batch.cu) and the serving rounds (serve.cu).
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
// Shared memory: 56 bytes a city (230 KB at the largest, n = 4,096); the best
// tour of an iterated search stays in global memory.
#pragma once
#include <cstdint>

#include "logo_device.cuh"

namespace logo {

constexpr uint32_t kNearK = 16;       // neighbours per list (two 16-byte loads)
constexpr uint32_t kNearMaxN = 4096;  // largest instance one CTA holds
// Warps per SM that kernels over NearTour are compiled for (64 registers a
// thread): a sweep is a chain of dependent shared-memory reads, so an SM is
// kept busy by the other CTAs on it.
constexpr int kNearWarpsPerSm = 32;
constexpr uint32_t kNoSeed = 0xFFFFFFFFu;
constexpr int kNoEdge = -(1 << 28);   // stands for an edge that takes part in nothing

// Cells of the search grid: about two cities per cell; never more than this.
__host__ __device__ constexpr uint32_t near_cells_max(uint32_t n) { return n / 2 + 64; }

// Byte offsets of the arrays, for an instance of n cities.
struct NearLayout {
    uint32_t xy, e, nbr, id, pos, near1, queue, far, cell, cellid, bytes;
};
__host__ __device__ constexpr uint32_t near_pad16(uint32_t b) { return (b + 15u) & ~15u; }
__host__ __device__ constexpr NearLayout near_layout(uint32_t n) {
    NearLayout l{};
    l.nbr = 0;                                               // uint16[n][kNearK]
    l.xy = l.nbr + 2 * kNearK * n;                           // float2[n]
    l.e = near_pad16(l.xy + 8 * n);                          // int[n]
    l.id = near_pad16(l.e + 4 * n);                          // uint16[n]
    l.pos = near_pad16(l.id + 2 * n);                        // uint16[n]
    l.near1 = near_pad16(l.pos + 2 * n);                     // uint16[n]
    l.queue = near_pad16(l.near1 + 2 * n);                   // uint16[n]
    l.far = near_pad16(l.queue + 2 * n);                     // uint16[n / 2]
    l.cellid = near_pad16(l.far + 2 * (n / 2));              // uint16[n]
    l.cell = near_pad16(l.cellid + 2 * n);                   // uint16[cells + 1]
    l.bytes = near_pad16(l.cell + 2 * (near_cells_max(n) + 1));
    return l;
}

struct NearTour {
    uint32_t n;
    uint32_t o;     // slot of position 0
    bool rev;       // positions count downwards
    bool whole;     // the lists hold every other city
    uint32_t kc;    // entries per list
    float2* xy;     // by slot
    int* E;         // by slot: the edge between slots j - 1 and j
    uint16_t* id;   // city in slot j
    uint16_t* pos;  // slot of city v
    uint16_t* near1;  // distance of city v to its nearest city (upper half of the float)
    uint16_t* queue;  // slots to be looked at, later the edges that take part
    uint16_t* far;    // slots whose lists were too short (up to n / 2)
    uint16_t* nbr;
    uint16_t* cell;    // first entry of every cell in cellid (row major), and the end
    uint16_t* cellid;  // cities by cell
    int gx, gy;
    float x0, y0, inv;  // a coordinate x lies in column (x - x0) * inv, truncated

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
    // where E holds the closing edge
    __device__ __forceinline__ uint32_t closing() const { return rev ? wrap(o + 1) : o; }
};

template <int NT>
struct NearShared {
    unsigned long long wbest[2][NT / 32];
    unsigned long long part[NT / 32];
    float red[4][NT / 32];
    uint32_t scan[NT / 32];
    // per sweep, by its parity: best delta met, entries of NearTour::queue and
    // ::far, discs put off, edges listed for those
    int bound[2];
    uint32_t queued[2], far[2], big[2], active[2];
    // cities at the ends of a new edge of each warp's best pair in the last sweep
    uint32_t seed[NT / 32];
    uint16_t scratch[NT / 32][32];  // each warp's slots in hand
    uint32_t idx;
    unsigned int flag, seq;
};

template <int NT>
__device__ __forceinline__ void near_reset(NearShared<NT>& S, uint32_t parity) {
    S.bound[parity] = -1;
    S.queued[parity] = S.far[parity] = S.big[parity] = S.active[parity] = 0;
}

// Once per kernel; a barrier must follow before the first sweep.
template <int NT>
__device__ __forceinline__ void near_init(NearShared<NT>& S) {
    if (threadIdx.x < 2) near_reset<NT>(S, threadIdx.x);
}

__device__ __forceinline__ NearTour near_carve(unsigned char* smem, uint32_t n) {
    const NearLayout l = near_layout(n);
    NearTour T;
    T.n = n;
    T.o = 0;
    T.rev = false;
    T.kc = n - 1 < kNearK ? n - 1 : kNearK;
    T.whole = n - 1 <= kNearK;
    T.xy = reinterpret_cast<float2*>(smem + l.xy);
    T.E = reinterpret_cast<int*>(smem + l.e);
    T.id = reinterpret_cast<uint16_t*>(smem + l.id);
    T.pos = reinterpret_cast<uint16_t*>(smem + l.pos);
    T.near1 = reinterpret_cast<uint16_t*>(smem + l.near1);
    T.queue = reinterpret_cast<uint16_t*>(smem + l.queue);
    T.far = reinterpret_cast<uint16_t*>(smem + l.far);
    T.nbr = reinterpret_cast<uint16_t*>(smem + l.nbr);
    T.cell = reinterpret_cast<uint16_t*>(smem + l.cell);
    T.cellid = reinterpret_cast<uint16_t*>(smem + l.cellid);
    T.gx = T.gy = 1;
    T.x0 = T.y0 = T.inv = 0.f;
    return T;
}

// The squared distance whose rounded root the per-edge distance is
// (exact_dist in logo_device.cuh).
__device__ __forceinline__ float near_sq(float2 a, float2 b) {
    const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y);
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
}
__device__ __forceinline__ int near_len(float s) {
    return __float2int_rz(__fadd_rn(__fsqrt_rn(s), 0.5f));
}
__device__ __forceinline__ int near_dist(float2 a, float2 b) { return near_len(near_sq(a, b)); }

// Cell column (or row) of a coordinate u counted from the box's corner:
// monotone in u, clamped to the grid.  (Differences from the corner are below
// 2e6 and good to 0.12 wherever the box lies; the coordinates themselves may be
// much larger.)
__device__ __forceinline__ int near_cell(float u, float inv, int cells) {
    const int c = (int)fminf(fmaxf(u * inv, 0.f), 1.0e6f);
    return c < cells ? c : cells - 1;
}

// ---- the search grid and the neighbour lists ---------------------------------
// Once per instance: bounding box, counting sort of the cities into cells, then
// one thread per city searches rings of cells until its kNearK nearest are
// certain.  The list area serves as the sort's 32-bit counters first.
template <int NT>
__device__ void near_build(NearTour& T, NearShared<NT>& S, const float2* __restrict__ gxy) {
    const uint32_t n = T.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < NT / 32) S.seed[threadIdx.x] = kNoSeed;  // no pair of this instance yet
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
    // square cells of about two cities; a thin box gets fewer, longer ones
    const float w = x1 - x0, h = y1 - y0;
    const float cap = (float)(n / 2 + 1);
    float side = fmaxf(sqrtf(w / cap * h), fmaxf(w, h) / cap);
    const uint32_t cells_max = near_cells_max(n);
    int gx = 1, gy = 1;
    float inv = 0.f;
    if (side > 0.f) {
        for (int t = 0; t < 64; ++t) {
            inv = 1.0f / side;
            gx = (int)fminf(w * inv, 65536.f) + 1;
            gy = (int)fminf(h * inv, 65536.f) + 1;
            if ((uint64_t)gx * (uint64_t)gy <= cells_max) break;
            side *= 1.125f;
        }
        if ((uint64_t)gx * (uint64_t)gy > cells_max) {
            gx = gy = 1;
            inv = 0.f;
        }
    }
    T.gx = gx;
    T.gy = gy;
    T.x0 = x0;
    T.y0 = y0;
    T.inv = inv;
    const uint32_t cells = (uint32_t)(gx * gy);
    uint32_t* count = reinterpret_cast<uint32_t*>(T.nbr);  // cells <= n / 2 + 64 words
    for (uint32_t c = threadIdx.x; c < cells; c += NT) count[c] = 0;
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        const float2 p = gxy[v];
        atomicAdd(&count[near_cell(p.y - y0, inv, gy) * gx + near_cell(p.x - x0, inv, gx)], 1u);
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
        const uint32_t c = near_cell(p.y - y0, inv, gy) * gx + near_cell(p.x - x0, inv, gx);
        T.cellid[atomicAdd(&count[c], 1u)] = (uint16_t)v;
    }
    __syncthreads();
    // lists: rings of cells around the city's own; after ring r every city
    // nearer than r cells has been seen (a little less, for rounding)
    for (uint32_t v = threadIdx.x; v < n; v += NT) {
        const float2 p = gxy[v];
        const int cx = near_cell(p.x - x0, inv, gx), cy = near_cell(p.y - y0, inv, gy);
        float ds[kNearK];
        uint32_t vs[kNearK];
#pragma unroll
        for (uint32_t k = 0; k < kNearK; ++k) {
            ds[k] = INFINITY;
            vs[k] = v;
        }
        const int rings = max(max(cx, gx - 1 - cx), max(cy, gy - 1 - cy));
        for (int r = 0; r <= rings; ++r) {
            const float sure = (float)(r - 1) * side * 0.999f;  // rings below r are done
            if (r >= 1 && ds[kNearK - 1] < sure * sure) break;
            for (int yy = max(cy - r, 0); yy <= min(cy + r, gy - 1); ++yy) {
                const bool edge_row = yy == cy - r || yy == cy + r;
                for (int part = 0; part < 2; ++part) {
                    // whole row of the ring, or its two end cells
                    int xa, xb;
                    if (edge_row) {
                        if (part) break;
                        xa = max(cx - r, 0);
                        xb = min(cx + r, gx - 1);
                    } else {
                        xa = xb = part ? cx + r : cx - r;
                        if (xa < 0 || xa >= gx) continue;
                    }
                    const uint32_t a = T.cell[yy * gx + xa], b = T.cell[yy * gx + xb + 1];
                    for (uint32_t k = a; k < b; ++k) {
                        const uint32_t u = T.cellid[k];
                        if (u == v) continue;
                        float d = near_sq(p, gxy[u]);
                        if (d >= ds[kNearK - 1]) continue;
                        uint32_t c = u;
#pragma unroll
                        for (uint32_t q = 0; q < kNearK; ++q) {
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
#pragma unroll
        for (uint32_t k = 0; k < kNearK; ++k) T.nbr[v * kNearK + k] = (uint16_t)vs[k];
        T.near1[v] = (uint16_t)(__float_as_uint(sqrtf(ds[0]) * 0.999999f) >> 16);  // rounded down
    }
    __syncthreads();
}

// ---- the tour -------------------------------------------------------------------
// Slot k = position k = id[k] (already written): coordinates, slots of cities,
// edges.
template <int NT>
__device__ __forceinline__ void near_place(NearTour& T, const float2* __restrict__ gxy) {
    T.o = 0;
    T.rev = false;
    for (uint32_t k = threadIdx.x; k < T.n; k += NT) {
        const uint32_t v = T.id[k];
        T.xy[k] = gxy[v];
        T.pos[v] = (uint16_t)k;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < T.n; k += NT)
        T.E[k] = near_dist(T.xy[k == 0 ? T.n - 1 : k - 1], T.xy[k]);
    __syncthreads();
}

// Length of the tour (routeLength, src/headers.h:170-189); every thread has it.
template <int NT>
__device__ __forceinline__ unsigned long long near_length(const NearTour& T, NearShared<NT>& S) {
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

// Reverses the arc of len slots from slot u (len < n).  Slots and the inner
// edges swap pairwise, the two outer edges get their new lengths from the
// thread that holds the arc's ends.  A barrier must follow.
template <int NT>
__device__ __forceinline__ void near_reverse(NearTour& T, uint32_t u, uint32_t len) {
    const uint32_t n = T.n;
    if (len == 0) return;
    for (uint32_t t = threadIdx.x; t < (len + 1) / 2; t += NT) {
        const uint32_t a = T.wrap(u + t), b = T.wrap(u + len - 1 - t);
        const float2 pa = T.xy[a], pb = T.xy[b];
        if (t == 0) {
            T.E[a] = near_dist(T.xy[a == 0 ? n - 1 : a - 1], pb);
            T.E[T.wrap(b + 1)] = near_dist(pa, T.xy[T.wrap(b + 1)]);
        }
        const uint16_t va = T.id[a], vb = T.id[b];
        T.xy[a] = pb;
        T.xy[b] = pa;
        T.id[a] = vb;
        T.id[b] = va;
        T.pos[vb] = (uint16_t)a;
        T.pos[va] = (uint16_t)b;
    }
    for (uint32_t t = threadIdx.x + 1; 2 * t < len; t += NT) {
        const uint32_t a = T.wrap(u + t), b = T.wrap(u + len - t);
        const int ea = T.E[a], eb = T.E[b];
        T.E[a] = eb;
        T.E[b] = ea;
    }
}

// Reverses positions [a, b) in place.
template <int NT>
__device__ __forceinline__ void near_reverse_positions(NearTour& T, uint32_t a, uint32_t b) {
    if (b <= a) return;
    near_reverse<NT>(T, T.rev ? T.slot(b - 1) : T.slot(a), b - a);
}

// new = old[p..q) ++ rev(old[0..p)) ++ rev(old[q..n)), p <= q < n.
template <int NT>
__device__ __forceinline__ void near_move(NearTour& T, uint32_t p, uint32_t q) {
    const uint32_t n = T.n, len = q - p;
    if (2 * len <= n) {
        // reversed arc [p, q), read the other way round from its far end
        const uint32_t first = T.slot(p), last = T.slot(q == 0 ? n - 1 : q - 1);
        near_reverse<NT>(T, T.rev ? last : first, len);
        T.o = last;
        T.rev = !T.rev;
    } else {
        // the complement: positions q .. n - 1, 0 .. p - 1
        const uint32_t o = T.slot(p);
        near_reverse<NT>(T, T.rev ? T.slot(p == 0 ? n - 1 : p - 1) : T.slot(q), n - len);
        T.o = o;
    }
    __syncthreads();
}

// new = old[0,p1) old[p2,p3) old[p1,p2) old[p3,n).
template <int NT>
__device__ __forceinline__ void near_double_bridge(NearTour& T, uint32_t p1, uint32_t p2,
                                                   uint32_t p3) {
    near_reverse_positions<NT>(T, p1, p3);
    __syncthreads();
    const uint32_t m = p1 + (p3 - p2);
    near_reverse_positions<NT>(T, p1, m);
    __syncthreads();
    near_reverse_positions<NT>(T, m, p3);
    __syncthreads();
}

// ---- the sweep --------------------------------------------------------------------
// (V + 1)^2: above it a squared distance stands for more than V; -1 for V < 0.
__device__ __forceinline__ float near_limit(int V) {
    const float l = (float)(V + 1);
    return V < 0 ? -1.f : l * l;
}

struct NearBest {
    uint64_t key;  // this lane's best pair
    int B;         // best delta its warp met, at most -1 (the same in every lane)
};

// The pair of the edges in E[f] and E[g], neither the closing edge, with new
// edges of squared lengths s and s2; true when it lowers the bound.  The test
// in front of the two square roots lets every pair with delta <= B through:
// the approximate root is within 2^-20 of the true one (2 at most), a rounded
// distance within 0.7, so D2 <= B + ef + eg - D1 implies
// sqrt(s2) <= B + ef + eg - approx + 3.4.
__device__ __forceinline__ bool near_pair(const NearTour& T, uint32_t f, uint32_t g, float s,
                                          float s2, int ef, int eg, NearBest& nb, int& lowest) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    const float t = (float)(nb.B + ef + eg + 4) - r;
    if (t < 0.f || s2 > t * t) return false;
    const int delta = near_len(s) + near_len(s2) - ef - eg;
    if (delta > nb.B) return false;
    const uint32_t i = T.edge_index(f), c = T.edge_index(g);
    const uint64_t key = pack_key(delta, min(i, c), max(i, c));
    nb.key = key < nb.key ? key : nb.key;
    lowest = min(lowest, delta);
    return true;
}

// The warp's bound after lanes met pairs.
__device__ __forceinline__ void near_share(NearBest& nb, bool met, int lowest) {
    if (__any_sync(0xffffffffu, met)) nb.B = __reduce_min_sync(0xffffffffu, min(nb.B, lowest));
}

// A city in slot p at squared distance s from the city in slot j: a later
// slot may meet the edge before j (both later ends), an earlier one the edge
// after j (both earlier ends); the last slot's next edge is E[0], so it may
// also do the latter.  True when the bound was lowered.
__device__ __forceinline__ bool near_meet(const NearTour& T, bool in, uint32_t j, uint32_t p,
                                          float s, int ej, int en, uint32_t z, NearBest& nb,
                                          int& lowest) {
    const uint32_t n = T.n, jn = T.wrap(j + 1);
    const int h = nb.B >> 1;
    const bool later = p > j;
    const uint32_t f = later ? j : jn, g = later ? p : p + 1;
    const int ef = later ? ej : en;
    bool met = false;
    if (in && p != j && (later || jn != 0) && g != z && s <= near_limit(ef + h))
        met = near_pair(T, f, g, s,
                        near_sq(T.xy[later ? (j == 0 ? n - 1 : j - 1) : jn], T.xy[later ? p - 1 : g]),
                        ef, T.E[g], nb, lowest);
    if (in && p == n - 1 && later && z != 0 && s <= near_limit(en + h))
        met |= near_pair(T, jn, 0, s, near_sq(T.xy[jn], T.xy[0]), en, T.E[0], nb, lowest);
    return met;
}

// A slot whose list was too short, looked at by the whole warp: over the grid's
// cells in the disc, or over the listed edges that can take part, where those
// are fewer than the disc's cities (long edges of a tour far from a local
// optimum: the bound is large then, and most edges too short).  j is the slot
// (the same in every lane); active is the number of listed edges.  With
// active = 0 none are listed yet: a large disc is then left alone and the
// result is true.
constexpr uint32_t kNearDisc = 256;  // cities that are always gone through
__device__ __forceinline__ bool near_far(const NearTour& T, uint32_t j, uint32_t z,
                                         uint32_t active, NearBest& nb) {
    const uint32_t lane = threadIdx.x & 31, n = T.n, jn = T.wrap(j + 1);
    const int ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
    const int V = max(ej, en) + (nb.B >> 1);
    if (V < 0) return false;
    const float2 p = T.xy[j];
    const float r = (float)(V + 2), lim = near_limit(V);
    const float ux = p.x - T.x0, uy = p.y - T.y0;
    const int xa = near_cell(ux - r, T.inv, T.gx), xb = near_cell(ux + r, T.inv, T.gx);
    const int ya = near_cell(uy - r, T.inv, T.gy), yb = near_cell(uy + r, T.inv, T.gy);
    const uint32_t cities = 2u * (uint32_t)((xb - xa + 1) * (yb - ya + 1));
    if (active == 0 && cities > kNearDisc) return true;
    if (active != 0 && cities > active) {
        const float2 before_j = T.xy[j == 0 ? n - 1 : j - 1], after_j = T.xy[jn];
        for (uint32_t t0 = 0; t0 < active; t0 += 32) {
            const uint32_t t = t0 + lane;
            bool met = false;
            int lowest = 0;
            if (t < active) {
                const uint32_t g = T.queue[t];
                const bool later = g > j;
                const float2 head = T.xy[g], tail = T.xy[g == 0 ? n - 1 : g - 1];
                const float s = near_sq(p, later ? head : tail);
                const int ef = later ? ej : en;
                if ((later || jn > g) && s <= near_limit(ef + (nb.B >> 1)))
                    met = near_pair(T, later ? j : jn, g, s,
                                    later ? near_sq(before_j, tail) : near_sq(after_j, head), ef,
                                    T.E[g], nb, lowest);
            }
            near_share(nb, met, lowest);
        }
        return false;
    }
    for (int y0 = ya; y0 <= yb; y0 += 32) {
        // up to 32 rows of cells, one per lane: each a run of cellid
        const int y = y0 + (int)lane;
        uint32_t first = 0, len = 0;
        if (y <= yb) {
            first = T.cell[y * T.gx + xa];
            len = T.cell[y * T.gx + xb + 1] - first;
        }
        uint32_t end = len;
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, end, s);
            if (lane >= (uint32_t)s) end += u;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
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
            int lowest = 0;
            const bool met = near_meet(T, s <= lim, j, q, s, ej, en, z, nb, lowest);
            near_share(nb, met, lowest);
        }
    }
    return false;
}

// Entries HALF * 8 .. HALF * 8 + 7 of the lists of the slots from[0 .. count),
// four slots at a time with a lane per entry (a long list keeps no other slot
// waiting), SETS such fours in flight.  Writes the slots whose entries were
// all in reach to out (which may be `from`) and returns their number.
template <int HALF, int SETS>
__device__ __forceinline__ uint32_t near_lists(const NearTour& T, const uint16_t* from,
                                               uint32_t count, uint16_t* out, uint32_t z,
                                               NearBest& nb) {
    const uint32_t lane = threadIdx.x & 31, k = HALF * 8 + (lane & 7);
    uint32_t open = 0;
    for (uint32_t t0 = 0; t0 < count; t0 += 4 * SETS) {
        uint32_t j[SETS], p[SETS];
        int ej[SETS], en[SETS];
        float s[SETS];
        bool in[SETS];
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            const uint32_t t = t0 + 4 * u + (lane >> 3);
            in[u] = t < count && k < T.kc;
            j[u] = from[min(t, count - 1)];
        }
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            const uint32_t jn = T.wrap(j[u] + 1);
            ej[u] = j[u] == z ? kNoEdge : T.E[j[u]];
            en[u] = jn == z ? kNoEdge : T.E[jn];
            p[u] = T.pos[T.nbr[T.id[j[u]] * kNearK + (in[u] ? k : 0)]];
        }
        bool met = false;
        int lowest = 0;
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            s[u] = near_sq(T.xy[j[u]], T.xy[p[u]]);
            in[u] = in[u] && s[u] <= near_limit(max(ej[u], en[u]) + (nb.B >> 1));
        }
#pragma unroll
        for (int u = 0; u < SETS; ++u)
            met |= near_meet(T, in[u], j[u], p[u], s[u], ej[u], en[u], z, nb, lowest);
        near_share(nb, met, lowest);
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
            // open <= t0 + 4 u: entries still to be read are not written
            const uint32_t ends = __ballot_sync(0xffffffffu, in[u] && (lane & 7) == 7);
            if (ends >> lane & 1u) out[open + __popc(ends & ((1u << lane) - 1u))] = (uint16_t)j[u];
            open += __popc(ends);
        }
        __syncwarp();
    }
    return open;
}

// One best-improvement sweep; the packed key of the best move (kNoMove if
// none).  parity alternates from sweep to sweep (it names the result slots).
//
// 1. Each warp re-evaluates the best pairs its CTA's warps met in the last
//    sweep, where their cities are now: real pairs of this tour, and most of
//    them still nearly the best, so the bound is good from the start.
// 2. A lane per slot: slots whose edges can take part and reach the nearest
//    city at least are queued.
// 3. The warps go through the queue's lists, eight slots at a time.
// 4. Slots whose lists were too short are dealt to the warps, a disc each.  They
//    wait until here because a disc costs what its radius says and the radius
//    shrinks with the bound.
// 5. Large discs that are left (a tour far from a local optimum) go over the
//    edges that can take part instead.
template <int NT>
__device__ __forceinline__ unsigned long long near_sweep(const NearTour& T, NearShared<NT>& S,
                                                         uint32_t parity) {
    constexpr int NW = NT / 32;
    const uint32_t n = T.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (n < 4) return kNoMove;
    const uint32_t z = T.closing();
    NearBest nb{kNoMove, -1};
    {
        bool met = false;
        int lowest = 0;
        if (lane < NW && S.seed[lane] != kNoSeed) {
            const uint32_t a = T.pos[S.seed[lane] & 0xffffu], b = T.pos[S.seed[lane] >> 16];
            if (a != b) {
                const uint32_t an = T.wrap(a + 1), bn = T.wrap(b + 1);
                const float s = near_sq(T.xy[a], T.xy[b]);
                if (a != z && b != z)
                    met = near_pair(T, a, b, s,
                                    near_sq(T.xy[a == 0 ? n - 1 : a - 1],
                                            T.xy[b == 0 ? n - 1 : b - 1]),
                                    T.E[a], T.E[b], nb, lowest);
                if (an != z && bn != z)
                    met |= near_pair(T, an, bn, s, near_sq(T.xy[an], T.xy[bn]), T.E[an], T.E[bn],
                                     nb, lowest);
            }
        }
        near_share(nb, met, lowest);
    }
    for (uint32_t base = warp * 32; base < n; base += NT) {  // whole warps
        const uint32_t j = base + lane;
        bool take = false;
        if (j < n) {
            const uint32_t jn = T.wrap(j + 1);
            const int ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
            const int m = max(ej, en);
            take = 2 * m + 8 >= -nb.B && (float)(m + (nb.B >> 1) + 1) >=
                                             __uint_as_float((uint32_t)T.near1[T.id[j]] << 16);
        }
        const uint32_t votes = __ballot_sync(0xffffffffu, take);
        if (votes == 0) continue;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&S.queued[parity], (uint32_t)__popc(votes));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (take) T.queue[at + __popc(votes & ((1u << lane) - 1u))] = (uint16_t)j;
    }
    __syncthreads();
    const uint32_t queued = S.queued[parity];
    uint16_t* scr = S.scratch[warp];
    for (uint32_t t = warp * 8; t < queued; t += NW * 8) {
        uint32_t open = near_lists<0, 2>(T, T.queue + t, min(8u, queued - t), scr, z, nb);
        if (open) open = near_lists<1, 1>(T, scr, open, scr, z, nb);
        if (open && !T.whole) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&S.far[parity], open);
            at = __shfl_sync(0xffffffffu, at, 0);
            for (uint32_t o = 0; o < open; ++o) {
                if (at + o < n / 2) {
                    if (lane == 0) T.far[at + o] = scr[o];
                } else {
                    near_far(T, scr[o], z, ~0u, nb);  // no room to wait
                }
            }
            __syncwarp();
        }
        // the bound of the CTA's other warps
        const int shared = *(volatile int*)&S.bound[parity];
        if (lane == 0 && nb.B < shared) atomicMin(&S.bound[parity], nb.B);
        nb.B = __shfl_sync(0xffffffffu, min(nb.B, shared), 0);
    }
    uint64_t best = warp_min_u64(nb.key);
    if (lane == 0) S.wbest[parity][warp] = best;
    __syncthreads();
    const uint32_t far = min(S.far[parity], n / 2);  // the same for every thread
    if (far) {
        nb.B = min(nb.B, S.bound[parity]);
        // entry t goes to warp t % NW; a lane each to see which are still open
        uint32_t put_off = 0;
        for (uint32_t t0 = 0; t0 < far; t0 += NT) {
            const uint32_t t = t0 + lane * NW + warp;
            uint32_t j = 0;
            bool open = false;
            if (t < far) {
                j = T.far[t];
                const uint32_t jn = T.wrap(j + 1);
                const int ej = j == z ? kNoEdge : T.E[j], en = jn == z ? kNoEdge : T.E[jn];
                const int m = max(ej, en);
                open = 2 * m + 8 >= -nb.B &&
                       near_sq(T.xy[j], T.xy[T.pos[T.nbr[T.id[j] * kNearK + kNearK - 1]]]) <=
                           near_limit(m + (nb.B >> 1));
            }
            for (uint32_t o = __ballot_sync(0xffffffffu, open); o; o &= o - 1) {
                const uint32_t jo = __shfl_sync(0xffffffffu, j, __ffs(o) - 1);
                if (near_far(T, jo, z, put_off < 32 ? 0u : ~0u, nb)) {
                    if (lane == 0) scr[put_off] = (uint16_t)jo;
                    ++put_off;
                }
            }
        }
        if (lane == 0) {
            if (nb.B < *(volatile int*)&S.bound[parity]) atomicMin(&S.bound[parity], nb.B);
            if (put_off) atomicAdd(&S.big[parity], put_off);
        }
        __syncthreads();
        if (S.big[parity]) {
            nb.B = min(nb.B, S.bound[parity]);
            for (uint32_t base = warp * 32; base < n; base += NT) {
                const uint32_t j = base + lane;
                const bool take = j < n && j != z && 2 * T.E[j] + 8 >= -nb.B;
                const uint32_t votes = __ballot_sync(0xffffffffu, take);
                if (votes == 0) continue;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&S.active[parity], (uint32_t)__popc(votes));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (take) T.queue[at + __popc(votes & ((1u << lane) - 1u))] = (uint16_t)j;
            }
            __syncthreads();
            // no edge listed: no edge can take part, and V < 0 for all of these
            const uint32_t active = max(S.active[parity], 1u);
            for (uint32_t o = 0; o < put_off; ++o) near_far(T, scr[o], z, active, nb);
        }
        best = warp_min_u64(nb.key);
        if (lane == 0) S.wbest[parity][warp] = best;
    }
    if (lane == 0) {
        uint32_t seed = kNoSeed;
        if (best != kNoMove) {
            const uint32_t i = T.slot(key_i(best)), c = T.slot(key_j(best));
            seed = (uint32_t)T.id[i] | (uint32_t)T.id[c] << 16;
        }
        S.seed[warp] = seed;
    }
    if (threadIdx.x == 0) near_reset<NT>(S, parity ^ 1);  // the next sweep's
    __syncthreads();
    unsigned long long k = S.wbest[parity][0];
#pragma unroll
    for (int w = 1; w < NW; ++w) k = S.wbest[parity][w] < k ? S.wbest[parity][w] : k;
    return k;
}

}  // namespace logo
