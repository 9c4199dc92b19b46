// The photon hash grid's k-capped radius query for one point, shared by the batched query
// kernel (hashgrid.cu) and the vertex-merging step of the VCM camera pass (vcm.cu).
// HashGrid::query (src/imbatracer/rangesearch/rangesearch.h:77-129): outside the grid's box
// nothing is found; otherwise the home cell and, per axis, the neighbour on the side of the
// nearer face are scanned (8 buckets in the reference's order; a bucket reached twice is
// scanned twice, and lists its photons twice), photons with squared distance <= r^2 are kept, at
// most the k nearest. The list is ordered by (distance, photon index); of photons at exactly the
// k-th distance those with the smallest indices stay (the reference keeps a choice that depends
// on the scan order within a bucket, which its parallel scatter leaves open). Every float
// operation is explicitly rounded, so cells and distances equal the reference's bit for bit.
//
// Those eight cells hold every photon within r only while the cell size is at least 2r (the
// reference's grid: cell = 2r). Grids with smaller cells (r <= cell < 2r, e.g. cell = r) are
// queried over every cell the box [q - r, q + r] touches instead — up to 4 per axis, bounds
// rounded outward and mapped to cells with the build's own rounding, so no photon within r
// is missed — in x-major order, each bucket once.
#pragma once

#include <stdint.h>

namespace imbart {

constexpr int kGridMaxK = 64;

__device__ __forceinline__ int hash_cell(uint32_t x, uint32_t y, uint32_t z, uint32_t table) {
    const uint32_t h = (x * 73856093u) ^ (y * 19349663u) ^ (z * 83492791u);
    return (int)((table & (table - 1u)) == 0u ? h & (table - 1u) : h % table);
}

// The cells a query scans. Reference mode (cell >= 2r): cell j of 8 is (j&4 ? xo : x0,
// j&2 ? yo : y0, j&1 ? zo : z0) with (x0, y0, z0) the home cell and (xo, yo, zo) the nearer
// neighbours. Range mode: cell j is (x0 + j / (ny nz), y0 + (j / nz) % ny, z0 + j % nz).
struct GridCells {
    bool ref_mode;
    int n;                       // cells to visit
    int x0, y0, z0;              // home cell / range start
    int xo, yo, zo;              // reference mode: neighbours
    int ny, nz;                  // range mode: extent in y and z
};

// Cell coordinate of a coordinate value, rounded as the build rounds it.
__device__ __forceinline__ int grid_coord(float v, float lo, float inv) {
    return (int)floorf(__fmul_rn(inv, __fsub_rn(v, lo)));
}

// prm: lo xyz, hi xyz, radius, r^2, cell size, 1 / cell size. False outside the grid's box.
__device__ __forceinline__ bool grid_cells(const float* prm, float qx, float qy, float qz, GridCells& g) {
    const bool inside = qx >= prm[0] && qy >= prm[1] && qz >= prm[2] && qx <= prm[3] && qy <= prm[4] && qz <= prm[5];
    if (!inside) return false;
    const float inv = prm[9], r = prm[6];
    g.ref_mode = prm[8] >= __fmul_rn(2.0f, r);
    if (g.ref_mode) {
        const float cx = __fmul_rn(inv, __fsub_rn(qx, prm[0]));
        const float cy = __fmul_rn(inv, __fsub_rn(qy, prm[1]));
        const float cz = __fmul_rn(inv, __fsub_rn(qz, prm[2]));
        const float fx = floorf(cx), fy = floorf(cy), fz = floorf(cz);
        g.x0 = (int)fx; g.y0 = (int)fy; g.z0 = (int)fz;
        g.xo = g.x0 + (__fsub_rn(cx, fx) < 0.5f ? -1 : 1);
        g.yo = g.y0 + (__fsub_rn(cy, fy) < 0.5f ? -1 : 1);
        g.zo = g.z0 + (__fsub_rn(cz, fz) < 0.5f ? -1 : 1);
        g.n = 8;
    } else {
        // A photon within r has each coordinate in [q - r, q + r]; the bounds are rounded
        // outward and mapped like photon coordinates (a monotone map), so its cell is inside.
        g.x0 = grid_coord(__fsub_rd(qx, r), prm[0], inv);
        g.y0 = grid_coord(__fsub_rd(qy, r), prm[1], inv);
        g.z0 = grid_coord(__fsub_rd(qz, r), prm[2], inv);
        const int nx = min(grid_coord(__fadd_ru(qx, r), prm[0], inv) - g.x0 + 1, 4);
        g.ny = min(grid_coord(__fadd_ru(qy, r), prm[1], inv) - g.y0 + 1, 4);
        g.nz = min(grid_coord(__fadd_ru(qz, r), prm[2], inv) - g.z0 + 1, 4);
        g.n = nx * g.ny * g.nz;
    }
    return true;
}

// j / d for 0 <= j < 64 and d in 1..4, as floor(j * m / 512): exact over that whole range.
__device__ __forceinline__ int div_small(int j, int d) {
    const int m = d == 1 ? 512 : d == 2 ? 256 : d == 3 ? 171 : 128;
    return (j * m) >> 9;
}

__device__ __forceinline__ void grid_cell(const GridCells& g, int j, int& x, int& y, int& z) {
    if (g.ref_mode) {
        x = (j & 4) ? g.xo : g.x0;
        y = (j & 2) ? g.yo : g.y0;
        z = (j & 1) ? g.zo : g.z0;
    } else {
        // j / nz and (j / nz) / ny by exact small multiplications: j < 64, extents 1..4.
        const int jz = div_small(j, g.nz), jy = div_small(jz, g.ny);
        x = g.x0 + jy;
        y = g.y0 + jz - jy * g.ny;
        z = g.z0 + j - jz * g.nz;
    }
}

// A lower bound of the squared distance from the query to any photon of cell (x, y, z): the
// distance to the cell's box, less a margin for the rounding of the photons' cell coordinates
// (a few ulps of the coordinate, 2^-24 relative each; the margin is 2^-20) and of their computed
// distances.
__device__ __forceinline__ float grid_cell_min_d2(const float* prm, float qx, float qy, float qz, int x, int y, int z) {
    const float inv = prm[9], cell = prm[8];
    float d2 = 0.0f;
    const float q[3] = {qx, qy, qz};
    const int c[3] = {x, y, z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float u = inv * (q[a] - prm[a]), f = (float)c[a];
        const float gap = fmaxf(f - u, u - f - 1.0f) - (fabsf(u) + 2.0f) * 9.5367431640625e-07f;
        const float d = fmaxf(gap, 0.0f) * cell;
        d2 += d * d;
    }
    return d2 * 0.99999f;
}

// Per-warp scratch of the search: the photons found so far (squared distance bits, index) and the
// offsets of the photon segments being read. kCap >= k + 32.
template <int kCap>
struct KnnScratch {
    alignas(16) uint32_t d2[kCap];
    int id[kCap];
    int delta[32];
};
constexpr int kKnnCapSmall = 64;             // k <= 32
constexpr int kKnnCapLarge = kGridMaxK + 32;

// Orders the n photons by (distance, index) and keeps the first k: every lane ranks its entries
// against all of them by distance (squared distances are >= 0, so their bits compare as
// integers). The ranks add up to n (n - 1) / 2 unless two distances are equal (light paths of
// equal random streams leave photons at equal positions: a quarter of the lists of 64 photons in
// a 1M-path light pass); then the indices decide, and of a photon met twice (two of the query's
// cells in one bucket) one entry stays if `unique`, both if not.
template <int kCap>
__device__ __forceinline__ int knn_keep(KnnScratch<kCap>& s, int n, int k, bool unique) {
    constexpr int kPer = kCap / 32;
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int per = (n + 31) >> 5;
    if (lane < (-n & 3)) s.d2[n + lane] = 0xffffffffu;    // to a multiple of four
    __syncwarp();
    uint32_t d[kPer];
    int id[kPer], rank[kPer];
    int sum = 0;
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        if (t > 0 && t >= per) { d[t] = 0u; id[t] = 0; rank[t] = kCap; continue; }
        const int i = 32 * t + lane;
        d[t] = s.d2[i];        // beyond n: left over, not used
        id[t] = s.id[i];
        int r = -1;
#pragma unroll 2
        for (int j = 0; j < n; j += 4) {
            const uint4 o = *reinterpret_cast<const uint4*>(s.d2 + j);
            r += (o.x <= d[t]) + (o.y <= d[t]) + (o.z <= d[t]) + (o.w <= d[t]);
        }
        rank[t] = r;
        if (i < n) sum += r;
    }
    int kept = n;
    const bool ties = __reduce_add_sync(kFull, sum) != n * (n - 1) / 2;
    if (ties) {
        // Equal distances by index, equal entries by position.
#pragma unroll
        for (int t = 0; t < kPer; ++t) {
            rank[t] = 0;
            if (t >= per) continue;
            const unsigned long long key = ((unsigned long long)d[t] << 32) | (uint32_t)id[t];
            for (int j = 0; j < n; ++j) {
                const unsigned long long o = ((unsigned long long)s.d2[j] << 32) | (uint32_t)s.id[j];
                rank[t] += o < key || (o == key && j < 32 * t + lane) ? 1 : 0;
            }
        }
    }
    const int keep = ties && unique ? n : k;   // photons met twice go before the list is cut
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kPer; ++t)
        if (32 * t + lane < n && rank[t] < keep) { s.d2[rank[t]] = d[t]; s.id[rank[t]] = id[t]; }
    __syncwarp();
    if (ties && unique) {
        unsigned twins = 0u;
#pragma unroll
        for (int t = 0; t < kPer; ++t) {
            const int i = 32 * t + lane;
            d[t] = i < n ? s.d2[i] : 0u;
            id[t] = i < n ? s.id[i] : 0;
            const bool twin = i < n && i > 0 && s.d2[i - 1] == d[t] && s.id[i - 1] == id[t];
            if (twin) rank[t] = -1;
            else rank[t] = i;
            twins |= __ballot_sync(kFull, twin);
        }
        if (twins != 0u) {
            kept = 0;
            __syncwarp();
#pragma unroll
            for (int t = 0; t < kPer; ++t) {
                const bool stays = 32 * t + lane < n && rank[t] >= 0;
                const unsigned m = __ballot_sync(kFull, stays);
                const int to = kept + __popc(m & ((1u << lane) - 1u));
                if (stays) { s.d2[to] = d[t]; s.id[to] = id[t]; }
                kept += __popc(m);
            }
            __syncwarp();
        }
    }
    return min(kept, k);
}

// The query by one warp (every lane calls it with the same point); returns the count, the list
// is s.d2 / s.id [0, count).
//
// A warp's instructions and its dependent loads (bucket bounds, then photons) bind this search,
// so it does as much as it can at once: lane j takes cell j, all bucket bounds come with one
// pair of loads, and the photons of all buckets are read as one sequence, 32 per step across
// bucket boundaries, instead of bucket after bucket (27 cells of mostly 0-5 photons where the
// cell size is r). Where the buckets hold more than two steps' photons, the cells within a
// quarter radius of the point go first; once k photons are known the others are scanned only if
// they can hold a nearer one, which in dense grids skips most of the photons. Measured (B200):
// 1.74 M queries of k = 10 among 1.74 M photons, cell = r, about 11 photons in reach: 3.43 ms with
// bucket after bucket and an insertion per photon, 1.3 ms; the merges of a 720p VCM iteration
// with about 100 in reach 10.9 against 2.3 ms. It issues at 85 % of the SMs' rate, so what is left
// is its instruction count. sorted: photons in bucket order (xyz + original index bits), ends:
// inclusive bucket ends.
template <int kCap>
__device__ __forceinline__ int grid_query_knn_warp(const float4* __restrict__ sorted, const int* __restrict__ ends,
                                                   const float* prm, uint32_t table, float qx, float qy, float qz,
                                                   int k, KnnScratch<kCap>& s) {
    const unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    GridCells gc;
    if (!grid_cells(prm, qx, qy, qz, gc)) return 0;
    const bool unique = !gc.ref_mode;    // range mode lists each photon once
    const float r2 = prm[7];
    float limit = r2;                    // photons farther than this are not wanted
    bool full = false;                   // k photons are kept, the last at distance^2 `limit`
    int n = 0;
    for (int c0 = 0; c0 < gc.n; c0 += 32) {
        const int jj = c0 + lane;
        const bool cell = jj < gc.n;
        int x = 0, y = 0, z = 0;
        grid_cell(gc, cell ? jj : 0, x, y, z);
        const int bucket = hash_cell((uint32_t)x, (uint32_t)y, (uint32_t)z, table);
        int b = 0, cnt = 0;
        if (cell) {
            b = bucket == 0 ? 0 : __ldg(ends + bucket - 1);
            cnt = __ldg(ends + bucket) - b;
        }
        float min_d2 = 0.0f;
        float near2 = r2;
        if (__reduce_add_sync(kFull, cnt) > 64) {
            near2 = 0.0625f * r2;
            min_d2 = grid_cell_min_d2(prm, qx, qy, qz, x, y, z);
            if (gc.ref_mode) {
                // A bucket that several of the cells share is scanned for each of them.
                const unsigned same = __match_any_sync(kFull, cell ? bucket : -2 - lane);
                if ((same & (same - 1u)) != 0u) min_d2 = 0.0f;
            }
        }
#pragma unroll 1
        for (int phase = 0; phase < 2; ++phase) {
            const bool mine = cnt > 0 && (phase == 0 ? !(min_d2 > near2) : !full || !(min_d2 > limit));
            const unsigned segs = __ballot_sync(kFull, mine);
            if (segs == 0u) continue;
            const int len = mine ? cnt : 0;
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += up;
            }
            const int total = __shfl_sync(kFull, incl, 31);
            int first = incl - len;
            if (mine) {
                s.delta[__popc(segs & lt)] = b - first;
                cnt = 0;
            } else {
                first = -1;
            }
            __syncwarp();
            const bool left = __ballot_sync(kFull, cnt > 0) != 0u;
            int seg = -1;     // segment of the photon before this step's first
            for (int at = 0; at < total; at += 32) {
                const unsigned start = (unsigned)(first - at) < 32u && first >= 0 ? 1u << (first - at) : 0u;
                const unsigned starts = __reduce_or_sync(kFull, start);
                const int i = at + lane;
                float d2 = 0.0f;
                int id = 0;
                bool in = false;
                if (i < total) {
                    const float4 ph = __ldg(sorted + (s.delta[seg + __popc(starts & (lt | (1u << lane)))] + i));
                    const float dx = __fsub_rn(qx, ph.x), dy = __fsub_rn(qy, ph.y), dz = __fsub_rn(qz, ph.z);
                    d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                    id = __float_as_int(ph.w);
                    in = d2 <= limit;
                }
                seg += __popc(starts);
                const unsigned found = __ballot_sync(kFull, in);
                if (in) {
                    const int to = n + __popc(found & lt);
                    s.d2[to] = __float_as_uint(d2);
                    s.id[to] = id;
                }
                n += __popc(found);
                // Order the list when the scratch could overflow, when it settles which cells are
                // left to scan, and at the end (with cells left and fewer than k photons, the
                // other phase scans them and orders the list).
                if (n > kCap - 32 || (at + 32 >= total && (n >= k || !left))) {
                    n = knn_keep(s, n, k, unique);
                    full = n == k;
                    if (full) limit = __uint_as_float(s.d2[k - 1]);
                }
            }
            __syncwarp();
        }
    }
    return n;
}

}  // namespace imbart
