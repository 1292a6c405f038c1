// Verlet pair list by a counting-sort cell list, with the pair criterion of
// scipy's cKDTree.query_pairs as the reference calls it (Sim.py:85-92,
// :192-198): FP64 periodic distances of float32(pos + L/2) in a box of edge
// float32(L + 1e-4), folded once per axis, squared components summed in x, y,
// z order without FMA, compared inclusively with r*r. Pairs (i, j), i < j,
// are written sorted by i then j.
//
// Steps: (1) cell of every body (cells of edge >= r, so every pair within r
// lies in neighbouring cells), (2) count per cell, exclusive scan, (3) the bodies'
// positions and indices in cell order, (4) per body i the count of the j > i
// within r over the 27 neighbouring cells, (5) scan of the counts, (6) the same
// traversal collects the j into shared memory, ranks them and writes them in order.
//
// The traversal runs in cell order, a warp per four consecutive bodies, so that a
// candidate is loaded once (16 bytes, coalesced) for all four when they share a
// cell, and the nine neighbouring columns of three cells are contiguous. A candidate
// is tested in FP32 with a margin that covers its rounding; only one within the
// margin of r takes the FP64 test above, which decides it. At 131,072 cubes (11.3 M
// pairs) counting takes 138 us and writing 349 us, bound by instruction issue; a warp
// per body that gathered three FP64 coordinates per candidate and tested in FP64
// took 570 and 912 us, and a scan for long lists 198 us more.
//
// Gated builds (displacement-triggered rebuilds): every kernel of the pass
// takes gate (null = always build); with gate[0] == 0 they return at once, so
// a CUDA graph can hold the pass in every step and only the flagged steps pay
// for it. A gated build also stores the positions it was built from, counts
// itself in gate[1] and sets gate[2] when the list did not fit its capacity.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "common.cuh"
#include "scan.cuh"

namespace amlp {
namespace {

constexpr int kWarpsPerBlock = 8;
// Bodies per warp: four share a traversal where that leaves every scheduler four
// warps, one below (3,000 dense tetrahedra: k_write 560 us with four, 86 us with one
// and the bitonic network below).
constexpr int kBodies = 4;
constexpr int kBodiesFrom = kNumSM * 4 * 4 * kBodies;
constexpr int kSortCap = 1024;   // neighbours of a warp's bodies ranked in its shared buffer
constexpr int kBigCap = 8192;    // up to this many: written unordered, then ranked by one block (k_sort_big)

struct Grid {
    int n, nc;        // bodies, cells per side (1 = one cell holding all bodies)
    double fb, hb;    // periodic box edge and half edge (FP64)
    double r2;        // r * r
    double inv_cs;    // nc / fb
    float halfL;      // float32(L * 0.5)
    float fbf;        // fb, a float
    float lo, hi;     // FP32 squared distances below lo are within r, above hi are not
};

__global__ void k_cells(const float *pos, Grid g, int *cell_of, int *cell_count, int *cell_last, int *outside,
                        const int *gate,
                        float *ref) {
    if (gate && !*gate) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    if (ref) {
        ref[3 * i] = pos[3 * i];
        ref[3 * i + 1] = pos[3 * i + 1];
        ref[3 * i + 2] = pos[3 * i + 2];
    }
    int c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float xf = __fadd_rn(pos[3 * i + k], g.halfL);
        if (!(xf >= 0.0f && xf <= g.fbf)) *outside = 1;
        double x = (double)xf;
        int ci = (int)(x * g.inv_cs);
        c[k] = ci < 0 ? 0 : (ci >= g.nc ? g.nc - 1 : ci);
    }
    int cid = (c[0] * g.nc + c[1]) * g.nc + c[2];
    cell_of[i] = cid;
    atomicAdd(&cell_count[cid], 1);
    atomicMax(&cell_last[cid], i + 1);
}

// float32(pos + L/2) and the index (as bits) of every body, in cell order.
__global__ void k_fill(const float *pos, Grid g, const int *cell_of, const long long *cell_start, int *cell_fill,
                       float4 *sorted, const int *gate) {
    if (gate && !*gate) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    int cid = cell_of[i];
    int slot = atomicAdd(&cell_fill[cid], 1);
    sorted[cell_start[cid] + slot] =
        make_float4(__fadd_rn(pos[3 * i], g.halfL), __fadd_rn(pos[3 * i + 1], g.halfL),
                    __fadd_rn(pos[3 * i + 2], g.halfL), __int_as_float(i));
}

// What the traversals read: bodies in cell order, the cells' first slots and
// largest body index plus one, whether a body lies outside the box.
struct Cells {
    const float4 *sorted;
    const long long *start;
    const int *last, *of, *outside;
};

// The pair test: FP64 distance, folded once per axis, x, y, z order, no FMA. The
// difference is i's minus j's as in the reference's call (its sign does not matter).
__device__ __forceinline__ bool within(const float4 &a, const float4 &b, const Grid &g) {
    const float av[3] = {a.x, a.y, a.z}, bv[3] = {b.x, b.y, b.z};
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double d = __dsub_rn((double)av[k], (double)bv[k]);
        if (d < -g.hb) d = __dadd_rn(g.fb, d);
        else if (d > g.hb) d = __dsub_rn(d, g.fb);
        r = __dadd_rn(r, __dmul_rn(d, d));
    }
    return r <= g.r2;
}

// Calls f(j, ok) for every body j of the cells around `cell` (a warp's lanes on
// consecutive ones; j = -1 past a range's end), ok[b] telling whether j > i and j
// is within r of the warp's body b, whose position and index i are in p[b]. All
// lanes of the warp call it with the same arguments, and f is called by all of them
// together, so that warp collectives inside f are safe.
// Lanes 0..26 look up the neighbouring cells at once; a cell whose largest index is
// not above the warp's smallest i holds no such j and is skipped (half of them
// when the indices follow the positions), and what is left of a column of three
// cells is one range. FOLD = false: the periodic image comes from the wrapped
// columns (the bodies are shifted once per range), for three cells per side or more
// and every body in the box. FOLD = true: each component is folded, min(|d|, fb - |d|)
// having the folded distance's magnitude.
template <bool FOLD, int NB, class F>
__device__ __forceinline__ void for_candidates(const float4 (&p)[NB], int cell, const Grid &g, const Cells &cl, F &&f) {
    const int lane = threadIdx.x & 31;
    auto range = [&](int s, int count, float sx, float sy, float sz) {
        const float4 *q = cl.sorted + s;
        const float4 none = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
        float x[NB], y[NB], z[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) x[b] = p[b].x + sx, y[b] = p[b].y + sy, z[b] = p[b].z + sz;
        float4 nxt = lane < count ? q[lane] : none;
        for (int base = 0; base < count; base += 32) {
            const float4 c = nxt;
            nxt = base + 32 + lane < count ? q[base + 32 + lane] : none;  // in flight during the tests
            const int j = __float_as_int(c.w);
            bool ok[NB], near = false;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                float dx = x[b] - c.x, dy = y[b] - c.y, dz = z[b] - c.z;
                if (FOLD) {
                    dx = fminf(fabsf(dx), g.fbf - fabsf(dx));
                    dy = fminf(fabsf(dy), g.fbf - fabsf(dy));
                    dz = fminf(fabsf(dz), g.fbf - fabsf(dz));
                }
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                ok[b] = j > __float_as_int(p[b].w) && d2 <= g.hi;
                near = near || (ok[b] && d2 >= g.lo);
            }
            if (near) {
#pragma unroll
                for (int b = 0; b < NB; ++b) ok[b] = ok[b] && within(p[b], c, g);
            }
            __syncwarp();
            f(j, ok);
        }
    };
    if (g.nc < 3) {
        range(0, g.n, 0.f, 0.f, 0.f);
        return;
    }
    const int cz = cell % g.nc, cxy = cell / g.nc, cy = cxy % g.nc, cx = cxy / g.nc;
    int first = __float_as_int(p[0].w);
#pragma unroll
    for (int b = 1; b < NB; ++b) first = min(first, __float_as_int(p[b].w));
    int s = 0, e = 0;
    bool any = false;
    if (lane < 27) {  // lane 9 (dx + 1) + 3 (dy + 1) + dz + 1
        int x = cx + lane / 9 - 1, y = cy + lane / 3 % 3 - 1, z = cz + lane % 3 - 1;
        x = x < 0 ? g.nc - 1 : (x == g.nc ? 0 : x);
        y = y < 0 ? g.nc - 1 : (y == g.nc ? 0 : y);
        z = z < 0 ? g.nc - 1 : (z == g.nc ? 0 : z);
        const long long c = ((long long)x * g.nc + y) * g.nc + z;
        s = (int)cl.start[c];
        e = (int)cl.start[c + 1];
        any = e > s && cl.last[c] > first + 1;
    }
    const unsigned live = __ballot_sync(0xffffffffu, any);
    const float fb = FOLD ? 0.0f : g.fbf;
    const bool wrapped = cz == 0 || cz == g.nc - 1;  // the column's three cells are not consecutive
    for (int col = 0; col < 9; ++col) {
        const unsigned bits = (live >> (3 * col)) & 7u;
        if (!bits) continue;
        const int x = cx + col / 3 - 1, y = cy + col % 3 - 1;
        const float sx = x < 0 ? fb : (x == g.nc ? -fb : 0.0f), sy = y < 0 ? fb : (y == g.nc ? -fb : 0.0f);
        if (!wrapped) {
            const int s0 = __shfl_sync(0xffffffffu, s, 3 * col + __ffs(bits) - 1);
            const int e0 = __shfl_sync(0xffffffffu, e, 3 * col + 31 - __clz(bits));
            range(s0, e0 - s0, sx, sy, 0.f);
        } else {
            for (int k = 0; k < 3; ++k) {
                if (!(bits >> k & 1u)) continue;
                const int s0 = __shfl_sync(0xffffffffu, s, 3 * col + k), e0 = __shfl_sync(0xffffffffu, e, 3 * col + k);
                const int z = cz + k - 1;
                range(s0, e0 - s0, sx, sy, z < 0 ? fb : (z == g.nc ? -fb : 0.0f));
            }
        }
    }
}

// Bodies of this warp: four consecutive ones of the cell order (position and index
// in p, cell in cell), fewer at the end; true when there are four in one cell.
__device__ __forceinline__ bool warp_bodies(const Grid &g, const Cells &cl, int s0, float4 (&p)[kBodies],
                                            int (&cell)[kBodies]) {
    bool same = s0 + kBodies <= g.n;
#pragma unroll
    for (int b = 0; b < kBodies; ++b) {
        p[b] = cl.sorted[min(s0 + b, g.n - 1)];
        cell[b] = cl.of[__float_as_int(p[b].w)];
        same = same && cell[b] == cell[0];
    }
    return same;
}

__device__ __forceinline__ int warp_sum(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <bool FOLD, int NBW>
__device__ __forceinline__ void count_bodies(const Grid &g, const Cells &cl, long long *counts) {
    const int s0 = (blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5)) * NBW;
    if (s0 >= g.n) return;
    const int lane = threadIdx.x & 31;
    float4 p[kBodies];
    int cell[kBodies];
    if (NBW == kBodies && warp_bodies(g, cl, s0, p, cell)) {
        int cnt[kBodies] = {0, 0, 0, 0};
        for_candidates<FOLD>(p, cell[0], g, cl, [&](int, const bool (&ok)[kBodies]) {
#pragma unroll
            for (int b = 0; b < kBodies; ++b) cnt[b] += ok[b];
        });
#pragma unroll
        for (int b = 0; b < kBodies; ++b) {
            const int c = warp_sum(cnt[b]);
            if (lane == 0) counts[__float_as_int(p[b].w)] = c;
        }
        return;
    }
    for (int b = 0; b < NBW && s0 + b < g.n; ++b) {
        const float4 q[1] = {cl.sorted[s0 + b]};
        const int i = __float_as_int(q[0].w);
        int cnt = 0;
        for_candidates<FOLD>(q, cl.of[i], g, cl, [&](int, const bool (&ok)[1]) { cnt += ok[0]; });
        cnt = warp_sum(cnt);
        if (lane == 0) counts[i] = cnt;
    }
}

template <int NBW>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_count(Grid g, Cells cl, long long *counts, const int *gate) {
    if (gate && !*gate) return;
    if (g.nc < 3 || *cl.outside) count_bodies<true, NBW>(g, cl, counts);
    else count_bodies<false, NBW>(g, cl, counts);
}

// The cnt <= 32 NR distinct j in the warp's buffer b, sorted in place: each lane
// ranks NR of them by counting the smaller ones (padded to a multiple of 4).
template <int NR>
__device__ __forceinline__ void sort_small(int *b, int cnt, int padded) {
    const int lane = threadIdx.x & 31;
    int j[NR], rank[NR];
#pragma unroll
    for (int u = 0; u < NR; ++u) {
        j[u] = lane + 32 * u < cnt ? b[lane + 32 * u] : 0;
        rank[u] = 0;
    }
    for (int k = 0; k < padded; k += 4) {
        const int4 v = *reinterpret_cast<const int4 *>(b + k);
#pragma unroll
        for (int u = 0; u < NR; ++u) rank[u] += (v.x < j[u]) + (v.y < j[u]) + (v.z < j[u]) + (v.w < j[u]);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < NR; ++u)
        if (lane + 32 * u < cnt) b[rank[u]] = j[u];
    __syncwarp();
}

// The cnt distinct j in the warp's buffer b sorted by a bitonic network over the
// next power of two (padded; the buffer has room for it).
__device__ __forceinline__ void sort_bitonic(int *b, int cnt) {
    const int lane = threadIdx.x & 31;
    int n2 = 256;
    while (n2 < cnt) n2 <<= 1;
    for (int e = cnt + lane; e < n2; e += 32) b[e] = 0x7fffffff;
    __syncwarp();
    for (int k = 2; k <= n2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int t = lane; t < n2 / 2; t += 32) {
                const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo + j;
                const int x = b[lo], y = b[hi];
                if ((x > y) == ((lo & k) == 0)) b[lo] = y, b[hi] = x;
            }
            __syncwarp();
        }
}

// The cnt distinct j of body i, gathered in the warp's buffer b (16-byte aligned,
// `room` ints, at least cnt rounded up to 4), sorted and written as the segment at
// `off` (what fits below cap). Up to 128 are ranked by counting; more take the
// bitonic network (10 k against 30 k instructions for 700) when there is room.
__device__ __forceinline__ void rank_and_write(int *b, int cnt, int room, int i, long long off, int *pairs,
                                               long long cap) {
    const int lane = threadIdx.x & 31, padded = (cnt + 3) / 4 * 4;
    bool sorted = true;
    if (cnt > 128 && room == kSortCap) {
        sort_bitonic(b, cnt);
    } else {
        if (lane < padded - cnt) b[cnt + lane] = 0x7fffffff;
        __syncwarp();
        if (cnt <= 32) sort_small<1>(b, cnt, padded);
        else if (cnt <= 64) sort_small<2>(b, cnt, padded);
        else if (cnt <= 96) sort_small<3>(b, cnt, padded);
        else if (cnt <= 128) sort_small<4>(b, cnt, padded);
        else sorted = false;
    }
    if (sorted) {
        for (int e = lane; e < cnt; e += 32)
            if (off + e < cap) {
                pairs[2 * (off + e)] = i;
                pairs[2 * (off + e) + 1] = b[e];
            }
    } else {
        for (int e = lane; e < cnt; e += 32) {
            const int j = b[e];
            int rank = 0;
            for (int k = 0; k < padded; k += 4) {
                const int4 v = *reinterpret_cast<const int4 *>(b + k);
                rank += (v.x < j) + (v.y < j) + (v.z < j) + (v.w < j);
            }
            const long long o = off + rank;
            if (o < cap) {
                pairs[2 * o] = i;
                pairs[2 * o + 1] = j;
            }
        }
    }
    __syncwarp();  // the buffer may be reused
}

template <bool FOLD, int NBW>
__device__ __forceinline__ void write_bodies(const Grid &g, const Cells &cl, const long long *offsets, int *pairs,
                                             long long cap, int *bw) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s0 = (blockIdx.x * kWarpsPerBlock + w) * NBW;
    if (s0 >= g.n) return;
    const unsigned below = (1u << lane) - 1u;
    float4 p[kBodies];
    int cell[kBodies];
    if (NBW == kBodies && warp_bodies(g, cl, s0, p, cell)) {
        // all four bodies in one traversal when their lists fit the buffer together
        int cnt[kBodies], at[kBodies], total = 0;
        long long off[kBodies];
        bool fits = true;
#pragma unroll
        for (int b = 0; b < kBodies; ++b) {
            const int i = __float_as_int(p[b].w);
            off[b] = offsets[i];
            const long long c = offsets[i + 1] - off[b];
            fits = fits && c <= kSortCap;
            cnt[b] = (int)min(c, (long long)kSortCap);
            at[b] = total;
            total += (cnt[b] + 3) / 4 * 4;
        }
        if (fits && total <= kSortCap) {
            if (total == 0) return;
            int fill[kBodies] = {at[0], at[1], at[2], at[3]};
            for_candidates<FOLD>(p, cell[0], g, cl, [&](int j, const bool (&ok)[kBodies]) {
#pragma unroll
                for (int b = 0; b < kBodies; ++b) {
                    const unsigned m = __ballot_sync(0xffffffffu, ok[b]);
                    if (ok[b]) bw[fill[b] + __popc(m & below)] = j;
                    fill[b] += __popc(m);
                }
            });
            __syncwarp();
#pragma unroll
            for (int b = 0; b < kBodies; ++b)
                if (cnt[b] > 0 && off[b] < cap) rank_and_write(bw + at[b], cnt[b], (cnt[b] + 3) / 4 * 4, __float_as_int(p[b].w), off[b], pairs, cap);
            return;
        }
    }
    for (int b = 0; b < NBW && s0 + b < g.n; ++b) {
        const float4 q[1] = {cl.sorted[s0 + b]};
        const int i = __float_as_int(q[0].w), ci = cl.of[i];
        const long long off = offsets[i];
        const int cnt = (int)(offsets[i + 1] - off);
        if (cnt == 0 || off >= cap) continue;  // nothing of this body's list fits
        if (cnt <= kSortCap) {
            int fill = 0;
            for_candidates<FOLD>(q, ci, g, cl, [&](int j, const bool (&ok)[1]) {
                const unsigned m = __ballot_sync(0xffffffffu, ok[0]);
                if (ok[0]) bw[fill + __popc(m & below)] = j;
                fill += __popc(m);
            });
            __syncwarp();
            rank_and_write(bw, cnt, kSortCap, i, off, pairs, cap);
            continue;
        }
        if (cnt <= kBigCap && off + cnt > cap) continue;  // crossing cap: k_sort_big writes the part that fits
        if (cnt <= kBigCap) {
            // written in candidate order here; k_sort_big ranks the segment afterwards
            int fill = 0;
            for_candidates<FOLD>(q, ci, g, cl, [&](int j, const bool (&ok)[1]) {
                const unsigned m = __ballot_sync(0xffffffffu, ok[0]);
                const long long o = off + fill + __popc(m & below);
                if (ok[0] && o < cap) pairs[2 * o + 1] = j;
                fill += __popc(m);
            });
            continue;
        }
        // More neighbours than one block ranks: emit them in increasing order by
        // repeated warp-wide minimum (slow, only for pathological inputs).
        int prev = i;
        for (int k = 0; k < cnt; ++k) {
            int best = 0x7fffffff;
            for_candidates<FOLD>(q, ci, g, cl, [&](int j, const bool (&ok)[1]) {
                if (ok[0] && j > prev && j < best) best = j;
            });
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0 && off + k < cap) {
                pairs[2 * (off + k)] = i;
                pairs[2 * (off + k) + 1] = best;
            }
            prev = best;
        }
    }
}

template <int NBW>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, 3) k_write(Grid g, Cells cl, const long long *offsets, int *pairs,
                                                                  long long cap, const int *gate) {
    if (gate && !*gate) return;
    __shared__ __align__(16) int buf[kWarpsPerBlock][kSortCap];
    int *bw = buf[threadIdx.x >> 5];
    if (g.nc < 3 || *cl.outside) write_bodies<true, NBW>(g, cl, offsets, pairs, cap, bw);
    else write_bodies<false, NBW>(g, cl, offsets, pairs, cap, bw);
}

// Sorts the segments of bodies with kSortCap < count <= kBigCap: one block per
// body, every j ranked by counting the smaller ones (the j of a body are
// distinct), written back with i. k_write left such a segment in candidate
// order when it fits below cap; the one segment that crosses cap is gathered
// here (warp 0 walks the neighbouring cells) and only its first cap - off
// pairs are written, so the pairs that fit are always the head of the list.
// A block looks for such bodies 256 at a time, a thread each (most lists have none),
// every gridDim.x-th body: the long lists are those of the lowest indices.
constexpr int kBigThreads = 256;
__global__ void __launch_bounds__(kBigThreads) k_sort_big(const float *pos, Grid g, Cells cl, const long long *offsets,
                                                          int *pairs, long long cap, const int *gate) {
    if (gate && !*gate) return;
    const bool fold = g.nc < 3 || *cl.outside;
    __shared__ __align__(16) int buf[kBigCap];
    __shared__ int todo[kBigThreads], ntodo;
    for (long long base = blockIdx.x; base < g.n; base += (long long)gridDim.x * kBigThreads) {
        if (threadIdx.x == 0) ntodo = 0;
        __syncthreads();
        const long long mine = base + (long long)gridDim.x * threadIdx.x;
        if (mine < g.n) {
            const long long off = offsets[mine], c = offsets[mine + 1] - off;
            if (c > kSortCap && c <= kBigCap && off < cap) todo[atomicAdd(&ntodo, 1)] = (int)mine;
        }
        __syncthreads();
        const int count = ntodo;
        for (int t = 0; t < count; ++t) {
            const int i = todo[t];
            const long long off = offsets[i];
            const int cnt = (int)(offsets[i + 1] - off);
            const bool crossing = off + cnt > cap;
            if (!crossing) {
                for (int e = threadIdx.x; e < cnt; e += blockDim.x) buf[e] = pairs[2 * (off + e) + 1];
            } else if (threadIdx.x < 32) {
                const int lane = threadIdx.x;
                const float4 q[1] = {make_float4(__fadd_rn(pos[3 * i], g.halfL), __fadd_rn(pos[3 * i + 1], g.halfL),
                                                 __fadd_rn(pos[3 * i + 2], g.halfL), __int_as_float(i))};
                int fill = 0;
                auto take = [&](int j, const bool (&ok)[1]) {
                    const unsigned m = __ballot_sync(0xffffffffu, ok[0]);
                    if (ok[0]) buf[fill + __popc(m & ((1u << lane) - 1u))] = j;
                    fill += __popc(m);
                };
                if (fold) for_candidates<true>(q, cl.of[i], g, cl, take);
                else for_candidates<false>(q, cl.of[i], g, cl, take);
            }
            const int padded = (cnt + 3) / 4 * 4;
            if ((int)threadIdx.x < padded - cnt) buf[cnt + threadIdx.x] = 0x7fffffff;
            __syncthreads();
            for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
                const int j = buf[e];
                int rank = 0;
                for (int k = 0; k < padded; k += 4) {
                    const int4 v = *reinterpret_cast<const int4 *>(buf + k);
                    rank += (v.x < j) + (v.y < j) + (v.z < j) + (v.w < j);
                }
                if (off + rank < cap) {
                    pairs[2 * (off + rank)] = i;
                    pairs[2 * (off + rank) + 1] = j;
                }
            }
            __syncthreads();
        }
        __syncthreads();  // todo is rewritten
    }
}

__global__ void k_total(const long long *offsets, int n, long long *d_count, int *gate, long long cap) {
    if (gate && !gate[0]) return;
    *d_count = offsets[n];
    if (gate) {
        gate[1] += 1;
        if (offsets[n] > cap) gate[2] = 1;
    }
}

// gate[0] = 1 when some body has moved more than sqrt(max_d2) from ref
// (minimum image in the cubic box), else 0 (gate[0] is cleared before).
__global__ void k_displacement(const float *pos, const float *ref, int n, float box, float max_d2, int *gate) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float d2 = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float d = pos[3 * i + k] - ref[3 * i + k];
        d -= box * rintf(d / box);
        d2 = fmaf(d, d, d2);
    }
    if (d2 > max_d2) gate[0] = 1;
}

Grid make_grid(int n, float box, double r) {
    Grid g;
    g.n = n;
    float bs = box + 0.0001f;  // float32(L + 1e-4), as numpy evaluates Lx + 0.0001
    g.fb = (double)bs;
    g.hb = 0.5 * g.fb;
    g.r2 = r * r;
    g.halfL = box * 0.5f;
    long long nc = (long long)floor(g.fb / (r * (1.0 + 1e-6)));
    if (nc > 160) nc = 160;
    if (nc < 3) nc = 1;
    g.nc = (int)nc;
    g.inv_cs = (double)g.nc / g.fb;
    // FP32 squared distances of float32 coordinates: each folded component is off by at
    // most 2^-23 of the box edge (two roundings), the sum of squares near r2 by less than
    // 2 sqrt(3) r times that plus 2^-22 r2. The margin is more than twice as wide.
    g.fbf = bs;
    const double margin = (r * g.fb + g.r2) * 0x1p-20;
    g.lo = (float)(g.r2 - margin);
    g.hi = nextafterf((float)(g.r2 + margin), INFINITY);
    return g;
}

struct NlistWs {
    float4 *sorted;
    int *cell_of, *cell_count, *cell_last, *cell_fill, *outside;
    long long *cell_start, *counts, *scan_tmp;
};

amlp_status launch_build(const float *d_pos, const Grid &g, const NlistWs &w, int *d_pairs, long long cap,
                         long long *d_count, int *gate, float *ref, cudaStream_t s);

size_t carve(Carver &c, const Grid &g, NlistWs *w) {
    size_t ncell = (size_t)g.nc * g.nc * g.nc;
    w->sorted = c.take<float4>(g.n);
    w->cell_of = c.take<int>(g.n);
    // what starts at zero side by side, for one fill: a gated build that does not run pays
    // for its fills and launches all the same (1,000 bodies: 22.5 us with three fills, 18.6 with one)
    w->cell_count = c.take<int>(3 * ncell + 1);
    w->cell_last = w->cell_count + ncell;
    w->cell_fill = w->cell_last + ncell;
    w->outside = w->cell_fill + ncell;  // the flag "a body lies outside the box"
    w->cell_start = c.take<long long>(ncell + 1);
    w->counts = c.take<long long>((size_t)g.n + 1);
    w->scan_tmp = c.take<long long>(scan_tmp_elems(std::max<size_t>(ncell, g.n) + 1));
    return c.used;
}

// A caller's workspace, from its first 16-byte boundary on (the size query has 256
// bytes to spare for that).
bool carve_caller(void *d_ws, size_t ws_bytes, const Grid &g, NlistWs *w) {
    const size_t skip = (16 - (reinterpret_cast<uintptr_t>(d_ws) & 15)) & 15;
    if (!d_ws || ws_bytes < skip) return false;
    Carver c(static_cast<char *>(d_ws) + skip, ws_bytes - skip);
    carve(c, g, w);
    return c.ok();
}

}  // namespace
}  // namespace amlp

using namespace amlp;

extern "C" amlp_status amlp_nlist_workspace_bytes(int n, float box, double r, size_t *bytes) {
    if (n <= 0 || !(box > 0.f) || !(r > 0.0) || !bytes) return AMLP_ERR_INVALID_ARG;
    Grid g = make_grid(n, box, r);
    Carver c(nullptr, 0);
    NlistWs w;
    *bytes = carve(c, g, &w) + 256;
    return AMLP_OK;
}

extern "C" amlp_status amlp_nlist_build(const float *d_pos, int n, float box, double r, int *d_pairs,
                                        long long cap, long long *d_count, void *d_ws, size_t ws_bytes,
                                        void *stream) {
    if (n <= 0 || !(box > 0.f) || !(r > 0.0) || !d_pos || !d_count || cap < 0 || (cap > 0 && !d_pairs))
        return AMLP_ERR_INVALID_ARG;
    cudaStream_t s = as_stream(stream);
    Grid g = make_grid(n, box, r);
    NlistWs w;
    if (!carve_caller(d_ws, ws_bytes, g, &w)) return AMLP_ERR_WORKSPACE;
    return launch_build(d_pos, g, w, d_pairs, cap, d_count, nullptr, nullptr, s);
}

namespace amlp {
namespace {

amlp_status launch_build(const float *d_pos, const Grid &g, const NlistWs &w, int *d_pairs, long long cap,
                         long long *d_count, int *gate, float *ref, cudaStream_t s) {
    const int n = g.n;
    size_t ncell = (size_t)g.nc * g.nc * g.nc;
    AMLP_CHECK_CUDA(cudaMemsetAsync(w.cell_count, 0, (3 * ncell + 1) * sizeof(int), s));
    int tb = 256;
    k_cells<<<(n + tb - 1) / tb, tb, 0, s>>>(d_pos, g, w.cell_of, w.cell_count, w.cell_last, w.outside, gate,
                                            ref);
    amlp_status st = exclusive_scan_int(w.cell_count, w.cell_start, (long long)ncell, w.scan_tmp, s, gate);
    if (st) return st;
    k_fill<<<(n + tb - 1) / tb, tb, 0, s>>>(d_pos, g, w.cell_of, w.cell_start, w.cell_fill, w.sorted, gate);
    const Cells cl{w.sorted, w.cell_start, w.cell_last, w.cell_of, w.outside};
    const bool four = n >= kBodiesFrom;
    const int per = kWarpsPerBlock * (four ? kBodies : 1), nb = (n + per - 1) / per;
    (four ? k_count<kBodies> : k_count<1>)<<<nb, 32 * kWarpsPerBlock, 0, s>>>(g, cl, w.counts, gate);
    st = exclusive_scan_ll(w.counts, w.counts, n, w.scan_tmp, s, gate);
    if (st) return st;
    (four ? k_write<kBodies> : k_write<1>)<<<nb, 32 * kWarpsPerBlock, 0, s>>>(g, cl, w.counts, d_pairs, cap, gate);
    k_sort_big<<<4 * kNumSM, kBigThreads, 0, s>>>(d_pos, g, cl, w.counts, d_pairs, cap, gate);
    k_total<<<1, 1, 0, s>>>(w.counts, n, d_count, gate, cap);
    return check_launch();
}

}  // namespace
}  // namespace amlp

extern "C" amlp_status amlp_nlist_check_displacement(const float *d_pos, const float *d_ref, int n, float box,
                                                     float max_disp, int *d_gate, void *stream) {
    if (n <= 0 || !(box > 0.f) || !(max_disp >= 0.f) || !d_pos || !d_ref || !d_gate) return AMLP_ERR_INVALID_ARG;
    cudaStream_t s = as_stream(stream);
    AMLP_CHECK_CUDA(cudaMemsetAsync(d_gate, 0, sizeof(int), s));
    k_displacement<<<(n + 255) / 256, 256, 0, s>>>(d_pos, d_ref, n, box, max_disp * max_disp, d_gate);
    return check_launch();
}

extern "C" amlp_status amlp_nlist_build_gated(const float *d_pos, int n, float box, double r, int *d_pairs,
                                              long long cap, long long *d_count, void *d_ws, size_t ws_bytes,
                                              int *d_gate, float *d_ref, void *stream) {
    if (n <= 0 || !(box > 0.f) || !(r > 0.0) || !d_pos || !d_count || !d_gate || !d_ref || cap < 0 ||
        (cap > 0 && !d_pairs))
        return AMLP_ERR_INVALID_ARG;
    Grid g = make_grid(n, box, r);
    NlistWs w;
    if (!carve_caller(d_ws, ws_bytes, g, &w)) return AMLP_ERR_WORKSPACE;
    return launch_build(d_pos, g, w, d_pairs, cap, d_count, d_gate, d_ref, as_stream(stream));
}

// ---------------------------------------------------------------------------
// Allocation-free variant of amlp_nlist_build.
//
// Some callers cannot allocate device memory at all, not even a workspace:
// for example a host program (an MD engine or a serving process) that hands
// this library only the buffers it owns, under a fixed GPU-memory budget, and
// does not let plug-ins call cudaMalloc or cudaFree. This entry point needs
// nothing beyond its inputs and outputs. Its scratch is the file-scope
// device array below: every GPU that loads the library holds it (13
// MiB) until the process exits.
//
// Limits: at most kNoAllocMaxBodies bodies, and at most kNoAllocMaxCells cells
// per box edge. Larger boxes simply use larger cells, which gives the same
// list. Every call shares the one array: calls that overlap on the GPU (on
// different streams, or from different host threads without ordering) race
// and must not be issued. The counters that must start at zero are cleared
// on the stream at the start of every call.
// ---------------------------------------------------------------------------
namespace amlp {
namespace {

constexpr int kNoAllocMaxBodies = 262144;
constexpr int kNoAllocMaxCells = 48;
constexpr size_t kNoAllocScratchBytes = 13u << 20;

__device__ __align__(256) unsigned char g_nlist_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[kMaxDevices] = {};

// Device address of the scratch array on the current device, looked up once
// per device (the host-side name is only a stand-in, not a device address).
amlp_status noalloc_scratch(void **out) {
    int dev = 0;
    AMLP_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return AMLP_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        AMLP_CHECK_CUDA(cudaGetSymbolAddress(&p, g_nlist_noalloc_scratch));
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return AMLP_OK;
}

}  // namespace
}  // namespace amlp

extern "C" amlp_status amlp_nlist_build_noalloc(const float *d_pos, int n, float box, double r, int *d_pairs,
                                                long long cap, long long *d_count, void *stream) {
    if (n <= 0 || !(box > 0.f) || !(r > 0.0) || !d_pos || !d_count || cap < 0 || (cap > 0 && !d_pairs))
        return AMLP_ERR_INVALID_ARG;
    if (n > kNoAllocMaxBodies) return AMLP_ERR_TOO_LARGE;
    Grid g = make_grid(n, box, r);
    if (g.nc > kNoAllocMaxCells) {
        g.nc = kNoAllocMaxCells;
        g.inv_cs = (double)g.nc / g.fb;
    }
    Carver probe(nullptr, kNoAllocScratchBytes);
    NlistWs w;
    carve(probe, g, &w);
    if (!probe.ok()) return AMLP_ERR_TOO_LARGE;
    void *scratch = nullptr;
    amlp_status st = noalloc_scratch(&scratch);
    if (st) return st;
    Carver c(scratch, kNoAllocScratchBytes);
    carve(c, g, &w);
    return launch_build(d_pos, g, w, d_pairs, cap, d_count, nullptr, nullptr, as_stream(stream));
}
