// GPU BVH builder: builds a whole scene (one BVH per mesh, a top-level BVH over the
// instances) on the device, directly in the compressed 8-wide layout the traversal kernels
// read, so that admitting a scene does not wait for a CPU build and a host-side conversion.
//
// The reference builds its mesh BVHs on the CPU, serially, with SBVH (sbvh_builder.h:29-165)
// and its top level with binned SAH (fast_bvh_builder.h); here all trees of a scene are built
// together as one forest: the primitives of every mesh, and the instances as one more segment,
// stand segment after segment in one array, and no step looks across a segment's ends.
//   1. primitive boxes and, per segment, the box of their centroids (instances: the bound of
//      their mesh's transformed vertices);
//   2. keys (segment, Morton code of the centroid), radix-sorted (CUB);
//   3. PLOC clustering (Meister and Bittner, "Parallel Locally-Ordered Clustering for
//      Bounding Volume Hierarchy Construction", TVCG 2018): every cluster finds its nearest
//      neighbour (smallest union surface area) among the 16 clusters on either side in Morton
//      order, mutual nearest neighbours merge, the cluster array is compacted; repeated until
//      one cluster per segment is left. Merged nodes are numbered by prefix sums, so the tree
//      does not depend on thread timing. A merge also computes the node's surface-area cost
//      (traversal cost 1, one unit per primitive) and turns subtrees of at most three triangles
//      into leaves where that is cheaper (one instance per leaf at the top level);
//      It also chooses the collapse below it: the wide nodes of smallest summed surface area, by
//      the dynamic programme of the host converter (convert.cpp, Collapse);
//   4. a top-down collapse into 8-wide nodes, level by level over all meshes, then over the
//      instances: a wide node takes the chosen descendants of its binary node as children,
//      assigns slots by direction octant, quantizes the child boxes conservatively (the same
//      arithmetic as the host converter) and writes the leaves' triangle or instance records.
// Hits do not depend on the tree: traversal over this layout finds the same closest hit
// as over any other BVH of the same triangles.
//
// What bounds a build is not the work but its dependent steps: about 35 clustering rounds and
// 10 collapse levels, most of them over few clusters. So steps 3 and 4 are one cooperative
// kernel each, whose blocks meet at a barrier between dependent phases, instead of a dozen
// launches, two scans and a read-back by the host per round, mesh after mesh. Measured (B200): 9
// meshes of 104 k triangles and 201 instances, up to the hits of a first ray batch, 28 -> 3.3 ms.
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "imbart_internal.h"

namespace imbart {
namespace {

constexpr int kRadius = 16;          // PLOC search radius
constexpr int kBlock = 256;
constexpr int kMaxLeafTris = 3;

// BuildState::error
constexpr int kErrIndex = 1, kErrProgress = 2, kErrBarrier = 3;

struct Box6 {
    float lo[3], hi[3];
};

__device__ __forceinline__ float half_area(const Box6& b) {
    const float dx = fmaxf(b.hi[0] - b.lo[0], 0.0f), dy = fmaxf(b.hi[1] - b.lo[1], 0.0f),
                dz = fmaxf(b.hi[2] - b.lo[2], 0.0f);
    return dx * (dy + dz) + dy * dz;
}

__device__ __forceinline__ Box6 merge(const Box6& a, const Box6& b) {
    Box6 r;
    for (int k = 0; k < 3; ++k) { r.lo[k] = fminf(a.lo[k], b.lo[k]); r.hi[k] = fmaxf(a.hi[k], b.hi[k]); }
    return r;
}

// Order-preserving int encoding of floats for atomicMin / atomicMax.
__device__ __forceinline__ int f2ord(float f) { const int i = __float_as_int(f); return i >= 0 ? i : i ^ 0x7fffffff; }
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// ---------------------------------------------------------------------------------------
// 1-2. Boxes, centroid bounds, Morton codes
// ---------------------------------------------------------------------------------------
// Segment of primitive i: the last one that starts at or before it.
__device__ __forceinline__ int segment_of(const int* __restrict__ first, int n_seg, int i) {
    int lo = 0, hi = n_seg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(first + mid) <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void bounds_init_kernel(int* cb, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) cb[i] = i % 6 < 3 ? 0x7fffffff : (int)0x80000000;   // the extreme encodings of f2ord
}

// Adds centroids to their segments' bounds (ordered-int atomics). A warp whose primitives all
// belong to one segment reduces first. NaN coordinates stay out: their encoding lies beyond every
// float's, and bounds that hold one order the segment's primitives along no curve.
__device__ __forceinline__ void add_centroid(const Box6& b, bool valid, int seg, int* cb) {
    const unsigned full = 0xffffffffu;
    const int s0 = __shfl_sync(full, seg, 0);
    const bool uniform = __all_sync(full, !valid || seg == s0);
    for (int k = 0; k < 3; ++k) {
        const float c = 0.5f * (b.lo[k] + b.hi[k]);
        const bool in = valid && c == c;
        if (uniform) {
            const int lo = __reduce_min_sync(full, in ? f2ord(c) : 0x7fffffff);
            const int hi = __reduce_max_sync(full, in ? f2ord(c) : (int)0x80000000);
            if ((threadIdx.x & 31) == 0 && lo <= hi) {
                int* q = cb + 6 * s0 + k;
                if (lo < __ldcg(q)) atomicMin(q, lo);
                if (hi > __ldcg(q + 3)) atomicMax(q + 3, hi);
            }
        } else if (in) {
            atomicMin(cb + 6 * seg + k, f2ord(c));
            atomicMax(cb + 6 * seg + 3 + k, f2ord(c));
        }
    }
}

// Triangle boxes and centroid bounds; a vertex index outside its mesh sets *error.
__global__ void tri_boxes_kernel(const float* __restrict__ verts, const int4* __restrict__ idx, int n,
                                 const int* __restrict__ seg_first, int n_seg,
                                 const long long* __restrict__ vert_first, const int* __restrict__ vert_count,
                                 Box6* boxes, int* cb, int* error) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    Box6 b;
    for (int k = 0; k < 3; ++k) b.lo[k] = b.hi[k] = 0.0f;
    int seg = 0;
    if (valid) {
        seg = segment_of(seg_first, n_seg, i);
        const int4 t = idx[i];
        const int nv = vert_count[seg];
        if ((unsigned)t.x >= (unsigned)nv || (unsigned)t.y >= (unsigned)nv || (unsigned)t.z >= (unsigned)nv) {
            atomicExch(error, kErrIndex);
        } else {
            const float* v = verts + 3 * vert_first[seg];
            for (int k = 0; k < 3; ++k) {
                const float a = v[3ll * t.x + k], c = v[3ll * t.y + k], d = v[3ll * t.z + k];
                b.lo[k] = fminf(a, fminf(c, d));
                b.hi[k] = fmaxf(a, fmaxf(c, d));
            }
        }
        boxes[i] = b;
    }
    add_centroid(b, valid, seg, cb);
}

// World boxes of instances: the bound of the instanced mesh's vertices through the 3x4
// object-to-world matrix in double precision (tighter than transforming the mesh box for rotated
// instances). Block (i, c) takes chunks c, c + gridDim.y, ... of instance i's vertices and adds its
// bound with 64-bit ordered atomics: one block per instance left a single large mesh to one SM. With
// many instances there are fewer blocks for each (kInstBlocks in all): blocks for the largest mesh's
// chunks that most instances do not have took 25 of 36 ms (200,000 instances, 655,362 vertices).
constexpr int kVertChunk = 16 * kBlock;
constexpr int kInstBlocks = 1 << 14;

__device__ __forceinline__ long long d2ord(double d) {
    const long long i = __double_as_longlong(d);
    return i >= 0 ? i : i ^ 0x7fffffffffffffffll;
}
__device__ __forceinline__ double ord2d(long long i) {
    return __longlong_as_double(i >= 0 ? i : i ^ 0x7fffffffffffffffll);
}

__global__ void inst_bounds_init_kernel(long long* ob, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ob[i] = d2ord(i % 6 < 3 ? DBL_MAX : -DBL_MAX);
}

__global__ void __launch_bounds__(kBlock) inst_bounds_kernel(const imbart_instance_desc* __restrict__ insts,
                                                             const float* __restrict__ verts,
                                                             const long long* __restrict__ vert_first,
                                                             const int* __restrict__ vert_count, long long* ob) {
    const int i = blockIdx.x, mesh = insts[i].mesh;
    const int nv = vert_count[mesh];
    if ((long long)blockIdx.y * kVertChunk >= nv) return;
    float m[12];
    for (int k = 0; k < 12; ++k) m[k] = insts[i].obj_to_world[k];
    const float* v = verts + 3 * vert_first[mesh];
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (long long c = (long long)blockIdx.y * kVertChunk; c < nv; c += (long long)gridDim.y * kVertChunk)
        for (long long k = c + threadIdx.x; k < nv && k < c + kVertChunk; k += kBlock) {
            const double p[3] = {v[3 * k], v[3 * k + 1], v[3 * k + 2]};
            for (int r = 0; r < 3; ++r) {
                const double w = (double)m[4 * r] * p[0] + (double)m[4 * r + 1] * p[1] + (double)m[4 * r + 2] * p[2] +
                                 (double)m[4 * r + 3];
                lo[r] = fmin(lo[r], w);
                hi[r] = fmax(hi[r], w);
            }
        }
    for (int r = 0; r < 3; ++r)
        for (int o = 16; o > 0; o >>= 1) {
            lo[r] = fmin(lo[r], __shfl_xor_sync(0xffffffffu, lo[r], o));
            hi[r] = fmax(hi[r], __shfl_xor_sync(0xffffffffu, hi[r], o));
        }
    if ((threadIdx.x & 31) != 0) return;
    for (int r = 0; r < 3; ++r) {
        if (lo[r] > hi[r]) continue;
        atomicMin(ob + 6ll * i + r, d2ord(lo[r]));
        atomicMax(ob + 6ll * i + 3 + r, d2ord(hi[r]));
    }
}

// Rounded outward and widened by 2^-20 of the magnitude; box and centroid of each instance.
__global__ void inst_boxes_kernel(const long long* __restrict__ ob, int n, Box6* boxes, int seg, int* cb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    Box6 b;
    for (int k = 0; k < 3; ++k) b.lo[k] = b.hi[k] = 0.0f;
    if (i < n) {
        double lo[3], hi[3], mag = 0.0;
        for (int r = 0; r < 3; ++r) {
            lo[r] = ord2d(ob[6ll * i + r]);
            hi[r] = ord2d(ob[6ll * i + 3 + r]);
            mag = fmax(mag, fmax(fabs(lo[r]), fabs(hi[r])));
        }
        const double pad = mag * 9.5367431640625e-07 + 1e-30;
        for (int r = 0; r < 3; ++r) { b.lo[r] = __double2float_rd(lo[r] - pad); b.hi[r] = __double2float_ru(hi[r] + pad); }
        boxes[i] = b;
    }
    add_centroid(b, i < n, seg, cb);
}

__device__ __forceinline__ uint64_t spread21(uint32_t x) {
    uint64_t v = x & 0x1fffffu;
    v = (v | (v << 32)) & 0x001f00000000ffffull;
    v = (v | (v << 16)) & 0x001f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// Key: segment above `bits` Morton bits per axis (as many as 64 bits leave, at most 21).
__global__ void morton_kernel(const Box6* __restrict__ boxes, int n, const int* __restrict__ seg_first, int n_seg,
                              int bits, const int* __restrict__ cb, uint64_t* keys, int* vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Box6 b = boxes[i];
    const int seg = segment_of(seg_first, n_seg, i);
    uint32_t q[3];
    for (int k = 0; k < 3; ++k) {
        const float lo = ord2f(cb[6 * seg + k]), hi = ord2f(cb[6 * seg + 3 + k]);
        const float ext = hi - lo;
        const float c = 0.5f * (b.lo[k] + b.hi[k]);
        const float t = ext > 0.0f ? (c - lo) / ext : 0.0f;
        q[k] = (uint32_t)fminf(fmaxf(t * 2097152.0f, 0.0f), 2097151.0f) >> (21 - bits);
    }
    const uint64_t code = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
    keys[i] = ((uint64_t)seg << (3 * bits)) | code;
    vals[i] = i;
}

// ---------------------------------------------------------------------------------------
// Barrier of a cooperative launch's blocks. Every block passes the same barriers in the same
// order; thread 0's fences order the block's accesses before and after it. The last block to
// arrive opens the barrier for the others, which poll a word of its own, so that their polls do
// not hold up the arrivals. A wait gives up after kSpinLimit polls and sets *error, which every
// block reads after the barrier and then leaves by.
// ---------------------------------------------------------------------------------------
constexpr int kSpinLimit = 1 << 22;

struct BuildState {
    unsigned arrived;       // barrier: blocks arrived so far
    unsigned pad0[31];
    unsigned open;          // arrivals of the barriers passed so far
    unsigned pad1[31];
    int error;
    int wide_count;         // wide nodes written
    int bottom_nodes;       // of these, mesh trees
    int tri_count;          // triangle records written
    int inst_count;
};

__device__ __forceinline__ bool grid_barrier(BuildState* st, unsigned& target) {
    __shared__ int s_error;
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        __threadfence();
        if (atomicAdd(&st->arrived, 1u) + 1u == target) {
            atomicExch(&st->open, target);
        } else {
            int polls = 0;
            while ((int)(*(volatile unsigned*)&st->open - target) < 0) {
                if (++polls > kSpinLimit) { atomicExch(&st->error, kErrBarrier); break; }
                __nanosleep(20);
            }
        }
        __threadfence();
        s_error = *(volatile int*)&st->error;
    }
    __syncthreads();
    return s_error == 0;
}

// Sums of (x, y) over the block's threads, in every thread.
__device__ __forceinline__ int2 block_sum(int x, int y) {
    __shared__ int sx[kBlock / 32], sy[kBlock / 32];
    x = __reduce_add_sync(0xffffffffu, x);
    y = __reduce_add_sync(0xffffffffu, y);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) { sx[threadIdx.x >> 5] = x; sy[threadIdx.x >> 5] = y; }
    __syncthreads();
    int2 r = make_int2(0, 0);
    for (int w = 0; w < kBlock / 32; ++w) { r.x += sx[w]; r.y += sy[w]; }
    return r;
}

// Sums of the blocks' pairs before this one (before) and of all (total).
__device__ __forceinline__ void block_prefix(const int2* sums, int blocks, int me, int2& before, int2& total) {
    int2 a = make_int2(0, 0), t = make_int2(0, 0);
    for (int i = threadIdx.x; i < blocks; i += kBlock) {
        const int2 v = __ldcg(sums + i);
        t.x += v.x; t.y += v.y;
        if (i < me) { a.x += v.x; a.y += v.y; }
    }
    before = block_sum(a.x, a.y);
    total = block_sum(t.x, t.y);
}

// The binary forest: leaves are primitives [0, n), inner nodes n + k.
struct Forest {
    int n;                  // primitives
    int n_seg;
    int top_seg;            // the instances' segment (-1: none in this batch)
    const int* seg_first;
    Box6* nbox;             // 2n: boxes of leaves and inner nodes
    int *left, *right;      // per inner node k: children
    int* cnt;               //   primitives
    float* cost;            //   surface-area cost
    uint8_t* leafy;         //   becomes a leaf
    float* area;            //   7 each: smallest sum of wide-node areas below with up to m entries
    uint8_t* split;         //   8 each: entries of the left child with m entries (0: one entry)
    int* roots;             // per segment
};

__device__ __forceinline__ bool is_leafy(const Forest& f, int node) { return node < f.n || f.leafy[node - f.n] != 0; }
__device__ __forceinline__ int prim_count(const Forest& f, int node) { return node < f.n ? 1 : f.cnt[node - f.n]; }

// The collapse below new inner node k (children l, r, half area a): area[7 k + m - 1] and
// split[8 k + m - 1] for m entries, as convert.cpp's Collapse.
__device__ __forceinline__ void choose_collapse(const Forest& f, int k, int l, int r, bool leaf, float a) {
    float* out = f.area + 7ll * k;
    uint8_t split[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float cost[8];
    for (int m = 0; m < 8; ++m) cost[m] = 0.0f;
    if (!leaf) {
        float lc[7], rc[7];
        const bool li = !is_leafy(f, l), ri = !is_leafy(f, r);
        for (int m = 0; m < 7; ++m) {
            lc[m] = li ? f.area[7ll * (l - f.n) + m] : 0.0f;
            rc[m] = ri ? f.area[7ll * (r - f.n) + m] : 0.0f;
        }
#pragma unroll
        for (int m = 2; m <= 8; ++m) {
            float best = lc[0] + rc[m - 2];
            int s = 1;
#pragma unroll
            for (int j = 2; j < m; ++j) {
                const float v = lc[j - 1] + rc[m - j - 1];
                if (v < best) { best = v; s = j; }
            }
            cost[m - 1] = best;
            split[m - 1] = (uint8_t)s;
        }
        cost[0] = a + cost[7];
#pragma unroll
        for (int m = 2; m < 8; ++m)
            if (cost[0] < cost[m - 1]) { cost[m - 1] = cost[0]; split[m - 1] = 0; }
    }
    for (int m = 0; m < 7; ++m) out[m] = cost[m];
    uint32_t w[2] = {0u, 0u};
    for (int m = 0; m < 8; ++m) w[m >> 2] |= (uint32_t)split[m] << (8 * (m & 3));
    *reinterpret_cast<uint2*>(f.split + 8ll * k) = make_uint2(w[0], w[1]);
}

struct PlocArrays {
    const int* sorted;      // primitives by (segment, Morton code)
    const Box6* boxes;      // their boxes, by primitive
    int *cl[2], *sg[2];     // clusters: node, segment
    Box6* box[2];           // and box
    int* link;              // >= 0: merges with that position; kKeep, kGone
    int2* sums;             // per block
};
constexpr int kKeep = -1, kGone = -2;
constexpr int kPlainRounds = 128;   // rounds by nearest neighbours; ordinary scenes take about 35
constexpr int kSolo = 1024; // clusters from which one block goes on alone (no barriers)
constexpr int kOwn = kBlock - 2 * kRadius;   // clusters of a tile: its neighbours within kRadius fill the block

// 3. PLOC. Each block owns a contiguous run of clusters and takes it in tiles of kOwn: boxes of the
// tile and 32 positions on either side in shared memory, nearest neighbours of the tile and 16
// positions on either side, one per thread (so that a merge is known to be mutual without another
// barrier), then after a barrier the compaction into the other buffers at the blocks' scanned
// offsets. Two barriers a round; below kSolo clusters one block goes on alone.
//
// Rounds are few as long as many clusters merge in each. Of equally near neighbours a cluster takes
// the one it shares an even-odd pair of positions with, then the smallest position: coinciding or
// evenly spaced primitives then pair up and halve every round (the smallest position alone made all
// but the first cluster point at ever smaller ones, one merge and one more level a round). Distances
// that grow along the order do the same without ties, so after kPlainRounds the pairs of positions
// merge as they stand, even-odd and odd-even in turn. Measured (B200): 30,000 triangles at growing
// spacings 84 -> 3 ms; the kernel over the instanced scene's 104 k triangles 394 -> 388 us, over 8
// and 100 spheres of 5,120 297 -> 307 and 676 -> 687 us.
__global__ void __launch_bounds__(kBlock) ploc_kernel(Forest f, PlocArrays p, BuildState* st) {
    constexpr int kHalo = 2 * kRadius;
    __shared__ float4 sb4[kOwn + 2 * kHalo];     // staged boxes: low corner, high x
    __shared__ float2 sb2[kOwn + 2 * kHalo];     // high y, z
    __shared__ int ss[kOwn + 2 * kHalo];
    __shared__ int snn[kBlock];
    __shared__ int wk[kBlock / 32], wm[kBlock / 32];
    if (*(volatile int*)&st->error != 0) return;
    unsigned target = 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = blockIdx.x * kBlock + tid; i < f.n; i += gridDim.x * kBlock) {
        const int v = p.sorted[i];
        const Box6 b = p.boxes[v];
        p.cl[0][i] = v;
        p.sg[0][i] = segment_of(f.seg_first, f.n_seg, v);
        p.box[0][i] = b;
        f.nbox[v] = b;
    }
    if (!grid_barrier(st, target)) return;
    int m = f.n, made = 0, cur = 0;
    bool solo = gridDim.x == 1;
    for (int round = 0; m > f.n_seg; ++round) {
        const bool plain = round >= kPlainRounds;
        if (!solo && m <= kSolo) {
            if (blockIdx.x != 0) return;
            solo = true;
        }
        const int blocks = solo ? 1 : gridDim.x;
        const int chunk = ((m + blocks - 1) / blocks + kOwn - 1) / kOwn * kOwn;
        const int lo = min((solo ? 0 : blockIdx.x) * chunk, m), hi = min(lo + chunk, m);
        const int* cl = p.cl[cur];
        const int* sg = p.sg[cur];
        const Box6* box = p.box[cur];
        int kept = 0, merged = 0;
        for (int tile = lo; tile < hi; tile += kOwn) {
            const int first = tile - kHalo;
            __syncthreads();
            for (int t = tid; t < kOwn + 2 * kHalo; t += kBlock) {
                const int j = first + t;
                ss[t] = -1;
                if (j >= 0 && j < m) {
                    const Box6 b = box[j];
                    sb4[t] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.hi[0]);
                    sb2[t] = make_float2(b.hi[1], b.hi[2]);
                    ss[t] = sg[j];
                }
            }
            __syncthreads();
            // Thread t finds the nearest neighbour of staged position t + kRadius.
            const int c = tid + kRadius;
            const int seg = ss[c];
            int bj = -1;
            if (seg >= 0) {
                const float4 a4 = sb4[c];
                const float2 a2 = sb2[c];
                float best = FLT_MAX;
                auto consider = [&](int j) {
                    const float4 b4 = sb4[j];
                    const float2 b2 = sb2[j];
                    // half_area of the union
                    const float dx = fmaxf(fmaxf(a4.w, b4.w) - fminf(a4.x, b4.x), 0.0f);
                    const float dy = fmaxf(fmaxf(a2.x, b2.x) - fminf(a4.y, b4.y), 0.0f);
                    const float dz = fmaxf(fmaxf(a2.y, b2.y) - fminf(a4.z, b4.z), 0.0f);
                    const float d = ss[j] == seg ? dx * (dy + dz) + dy * dz : FLT_MAX;
                    if (d < best) { best = d; bj = j; }   // of equal ones the first considered
                };
                // Tiles start at even positions: c has its position's parity, its pair is c ^ 1.
                const int pair = c ^ 1;
                if (plain) {
                    consider((round & 1) ? 2 * c - pair : pair);
                } else {
                    consider(pair);
                    consider(2 * c - pair);
#pragma unroll 10
                    for (int o = 0; o < 2 * kRadius - 2; ++o)
                        consider(c + (o < kRadius - 1 ? o - kRadius : o - kRadius + 3));
                }
            }
            snn[tid] = bj;
            __syncthreads();
            const int i = tile + tid - kRadius;
            if (tid >= kRadius && tid < kRadius + kOwn && i < hi) {
                const bool mutual = bj >= 0 && snn[bj - kRadius] == c;
                p.link[i] = !mutual ? kKeep : c < bj ? first + bj : kGone;
                merged += mutual && c < bj ? 1 : 0;
                kept += mutual && c > bj ? 0 : 1;
            }
        }
        __syncthreads();    // the links below are read by other threads of the block
        const int2 mine = block_sum(kept, merged);
        int2 before = make_int2(0, 0), total = mine;
        if (!solo) {
            if (tid == 0) p.sums[blockIdx.x] = mine;
            if (!grid_barrier(st, target)) return;
            block_prefix(p.sums, blocks, blockIdx.x, before, total);
        }
        // Pairs of one parity may all cross segments, so a plain round may pass without a merge; two
        // of them at least halve every segment that is longer than two.
        if (plain ? round >= kPlainRounds + 2 * 40 : total.y <= 0) {
            if (tid == 0) atomicExch(&st->error, kErrProgress);
            return;   // every block sees the same total
        }
        int* cl2 = p.cl[1 - cur];
        int* sg2 = p.sg[1 - cur];
        Box6* box2 = p.box[1 - cur];
        int kbase = before.x, mbase = made + before.y;
        for (int tile = lo; tile < hi; tile += kBlock) {
            const int i = tile + tid;
            const int link = i < hi ? p.link[i] : kGone;
            const unsigned km = __ballot_sync(0xffffffffu, link != kGone), mm = __ballot_sync(0xffffffffu, link >= 0);
            __syncthreads();
            if (lane == 0) { wk[warp] = __popc(km); wm[warp] = __popc(mm); }
            __syncthreads();
            int ko = kbase, mo = mbase;
            for (int w = 0; w < kBlock / 32; ++w) {
                if (w < warp) { ko += wk[w]; mo += wm[w]; }
                kbase += wk[w];
                mbase += wm[w];
            }
            if (link == kGone) continue;
            const unsigned lt = (1u << lane) - 1u;
            const int to = ko + __popc(km & lt);
            const int l = cl[i], seg = sg[i];
            sg2[to] = seg;
            if (link < 0) {
                cl2[to] = l;
                box2[to] = box[i];
                continue;
            }
            const int k = mo + __popc(mm & lt), r = cl[link];
            const Box6 bl = box[i], br = box[link], b = merge(bl, br);
            const int c = prim_count(f, l) + prim_count(f, r);
            const float a = half_area(b);
            const float inner = a + (l < f.n ? half_area(bl) : f.cost[l - f.n]) +
                                (r < f.n ? half_area(br) : f.cost[r - f.n]);
            const float leaf = a * (float)c;
            const bool lf = c <= (seg == f.top_seg ? 1 : kMaxLeafTris) && leaf <= inner;
            f.nbox[f.n + k] = b;
            f.left[k] = l;
            f.right[k] = r;
            f.cnt[k] = c;
            f.cost[k] = lf ? leaf : inner;
            f.leafy[k] = lf ? 1 : 0;
            choose_collapse(f, k, l, r, lf, a);
            cl2[to] = f.n + k;
            box2[to] = b;
        }
        made += total.y;
        m = total.x;
        cur = 1 - cur;
        if (solo) {
            __syncthreads();   // one block: its writes are ordered by the block barrier
        } else if (!grid_barrier(st, target)) {
            return;
        }
    }
    // One cluster per segment, in segment order.
    if (solo || blockIdx.x == 0)
        for (int i = tid; i < f.n_seg; i += kBlock) f.roots[i] = p.cl[cur][i];
}

// ---------------------------------------------------------------------------------------
// 4. Collapse into 8-wide nodes
// ---------------------------------------------------------------------------------------

// Eight lanes work on one wide node, a lane per child (then per slot).
__device__ __forceinline__ unsigned octet_ballot(bool b) {
    return (__ballot_sync(0xffffffffu, b) >> (threadIdx.x & 24u)) & 0xffu;
}

__device__ __forceinline__ double exp2_int(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// Conservative 8-bit quantization of one axis over an octet's lanes (convert.cpp quantize_axis,
// same arithmetic: divisions by a power of two as exact multiplications). Lanes of empty slots
// get the inverted bytes 1, 0.
__device__ __forceinline__ void quantize_axis_octet(float lo, float hi, bool valid, float pad, float& p_out,
                                                    int& bexp_out, uint32_t& qlo, uint32_t& qhi) {
    const unsigned full = 0xffffffffu;
    double nlo = valid ? (double)lo - pad : DBL_MAX, nhi = valid ? (double)hi + pad : -DBL_MAX;
    for (int o = 4; o > 0; o >>= 1) {
        nlo = fmin(nlo, __shfl_xor_sync(full, nlo, o));
        nhi = fmax(nhi, __shfl_xor_sync(full, nhi, o));
    }
    if (nlo > nhi) { nlo = 0.0; nhi = 0.0; }
    const double ext = nhi - nlo;
    int e = -126;
    if (ext > 0.0) {
        int ex;
        frexp(ext / 252.0, &ex);
        e = max(ex - 1, -126);
        while (e < 127 && 252.0 * exp2_int(e) < ext) ++e;
    }
    float P = 0.0f;
    bool done = false;
    qlo = 1u;
    qhi = 0u;
    while (__ballot_sync(full, !done) != 0u) {
        const double s = exp2_int(e), inv = exp2_int(-e);
        const double margin = s / 128.0;
        const double origin = nlo - margin - 32768.0 * s;
        float Pn = (float)origin;
        if ((double)Pn > origin) Pn = nextafterf(Pn, -FLT_MAX);
        bool ok = true;
        if (valid) {
            const double L = (double)lo - pad - margin, H = (double)hi + pad + margin;
            double ql = floor((L - (double)Pn) * inv) - 32768.0;
            double qh = ceil((H - (double)Pn) * inv) - 32768.0;
            for (int g = 0; g < 64 && (double)Pn + (32768.0 + ql) * s > L; ++g) ql -= 1;
            for (int g = 0; g < 64 && (double)Pn + (32768.0 + qh) * s < H; ++g) qh += 1;
            ok = ql >= 0 && qh <= 255;
            if (!done && ok) { qlo = (uint32_t)ql; qhi = (uint32_t)qh; }
        }
        const bool all = octet_ballot(!ok) == 0u;
        if (!done) {
            P = Pn;
            done = all || e >= 127;
            if (!done) ++e;
        }
    }
    p_out = P;
    bexp_out = e + 127;
}

// The child boxes of one node (lane s: slot s, zero where not valid) padded and quantized into
// its byte planes, words 8 to 19 of the record w (written if active); returns origin and exponents.
__device__ __forceinline__ void quantize_octet(bool active, const Box6& b, bool valid, uint32_t* w, float p[3],
                                               int bexp[3]) {
    const unsigned full = 0xffffffffu;
    const int lane8 = threadIdx.x & 7;
    float mag = 0.0f;
    if (valid)
        for (int a = 0; a < 3; ++a) {
            mag = fmaxf(mag, fmaxf(fabsf(b.lo[a]), fabsf(b.hi[a])));
            mag = fmaxf(mag, b.hi[a] - b.lo[a]);
        }
    for (int o = 4; o > 0; o >>= 1) mag = fmaxf(mag, __shfl_xor_sync(full, mag, o));
    const float pad = mag * 9.5367431640625e-07f + 1e-30f;
    // Lanes 0-3 make the first word of each byte row, lanes 4-7 the second.
    const int half = lane8 >> 2;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        uint32_t ql, qh;
        quantize_axis_octet(b.lo[a], b.hi[a], valid, pad, p[a], bexp[a], ql, qh);
        ql <<= 8 * (lane8 & 3);
        qh <<= 8 * (lane8 & 3);
        for (int o = 2; o > 0; o >>= 1) {
            ql |= __shfl_xor_sync(full, ql, o);
            qh |= __shfl_xor_sync(full, qh, o);
        }
        if (active && (lane8 & 3) == 0) { w[8 + 4 * a + half] = ql; w[10 + 4 * a + half] = qh; }
    }
}

// Where the leaves' records go.
struct LeafOut {
    int n_tris;                       // primitives below are triangles, the rest instances
    const float* verts;
    const int4* idx;
    const int* seg_first;
    int n_seg;
    const long long* vert_first;
    const int* tri_offset;            // per mesh: global id of its first triangle
    WideTri* tris;
    const imbart_instance_desc* inst;
    const int* mesh_root;             // wide root per mesh of the scene
    WideInst* insts;
};

__device__ __forceinline__ void emit_prim(const LeafOut& o, int prim, long long at) {
    if (prim < o.n_tris) {
        const int4 t = o.idx[prim];
        const int seg = segment_of(o.seg_first, o.n_seg, prim);
        const float* v = o.verts + 3 * o.vert_first[seg];
        float4* r = reinterpret_cast<float4*>(o.tris + at);
        r[0] = make_float4(v[3ll * t.x], v[3ll * t.x + 1], v[3ll * t.x + 2],
                           __int_as_float(o.tri_offset[seg] + (prim - o.seg_first[seg])));
        r[1] = make_float4(v[3ll * t.y], v[3ll * t.y + 1], v[3ll * t.y + 2], 0.0f);
        r[2] = make_float4(v[3ll * t.z], v[3ll * t.z + 1], v[3ll * t.z + 2], 0.0f);
    } else {
        const imbart_instance_desc& d = o.inst[prim - o.n_tris];
        WideInst r;
        for (int k = 0; k < 12; ++k) r.m[k] = d.world_to_obj[k];
        r.id = d.id;
        r.root = __ldcg(o.mesh_root + d.mesh);
        r.pad[0] = 0;
        r.pad[1] = 0;
        o.insts[at] = r;
    }
}

struct CollapseArrays {
    int *queue[2];          // binary nodes of a level's wide nodes
    int* kids;              // 8 per queue entry
    int *n_int, *n_prims;   // per entry: internal children, leaf primitives
    int2* sums;             // per block
    int* mesh_root;         // wide root per mesh of the scene (this batch's meshes are written)
};

// The children of a top-level wide node (whole warp, eight lanes per node, node < 0: none): lane i
// returns child i or -1. The internal child of largest area is opened until there are eight (as
// the host converter does at the top level).
__device__ __forceinline__ int gather_largest(const Forest& f, int node) {
    const unsigned full = 0xffffffffu;
    const int i = threadIdx.x & 7;
    int kid = -1, nk = 0;
    if (node >= 0) {
        if (is_leafy(f, node)) {
            kid = i == 0 ? node : -1;
            nk = 1;
        } else {
            kid = i == 0 ? f.left[node - f.n] : i == 1 ? f.right[node - f.n] : -1;
            nk = 2;
        }
    }
    float area = kid >= 0 && !is_leafy(f, kid) ? half_area(f.nbox[kid]) : -1.0f;
    for (int round = 0; round < 6; ++round) {
        float ba = area;
        int bi = i;
        for (int o = 4; o > 0; o >>= 1) {
            const float oa = __shfl_xor_sync(full, ba, o);
            const int oi = __shfl_xor_sync(full, bi, o);
            if (oa > ba || (oa == ba && oi < bi)) { ba = oa; bi = oi; }
        }
        const bool open = ba >= 0.0f && nk < 8 && nk >= 2;
        if (__ballot_sync(full, open) == 0u) break;
        const int c = __shfl_sync(full, kid, bi, 8);
        const int next_kid = __shfl_down_sync(full, kid, 1, 8);
        const float next_area = __shfl_down_sync(full, area, 1, 8);
        if (!open) continue;
        if (i >= bi) { kid = next_kid; area = next_area; }
        if (i == nk - 1 || i == nk) {
            kid = i == nk - 1 ? f.left[c - f.n] : f.right[c - f.n];
            area = is_leafy(f, kid) ? -1.0f : half_area(f.nbox[kid]);
        }
        ++nk;
        if (i >= nk) { kid = -1; area = -1.0f; }
    }
    return kid;
}

// The children of wide node `node` (whole warp, eight lanes per node, node < 0: none): a lane
// returns a child or -1. An entry (binary node, m) stands at the first of the m lanes it may
// fill and hands the right child's share to the lane where that begins.
__device__ __forceinline__ int gather_children(const Forest& f, int node) {
    const unsigned full = 0xffffffffu;
    const int i = threadIdx.x & 7;
    int kid = i == 0 ? node : -1, m = i == 0 && node >= 0 ? 8 : 0;
    bool open = m > 0 && !is_leafy(f, node);     // the wide node itself is opened in any case
    while (__ballot_sync(full, open) != 0u) {
        int k = 0, right = -1;
        if (open) {
            k = f.split[8ll * (kid - f.n) + m - 1];
            right = f.right[kid - f.n];
            kid = f.left[kid - f.n];
        }
        const int take = open ? i + k : -1, share = m - k;
        // Each lane looks for the opened entry that hands over to it.
        int from = -1;
        for (int s = 0; s < 8; ++s)
            if (__shfl_sync(full, take, s, 8) == i) from = s;
        const int r = __shfl_sync(full, right, from & 7, 8), rm = __shfl_sync(full, share, from & 7, 8);
        if (open) m = k;
        if (from >= 0) { kid = r; m = rm; }
        open = (open || from >= 0) && !is_leafy(f, kid) && m > 1 && f.split[8ll * (kid - f.n) + m - 1] != 0;
    }
    return kid;
}

// Writes one wide node (eight lanes; `active` is the octet's), its leaves' records and its
// internal children's queue entries. kid: lane i holds child i or -1.
__device__ __forceinline__ void write_wide(const Forest& f, bool active, int kid, int child_base, int prim_base,
                                           int* next_queue, WideNode* out, const LeafOut& lo) {
    const unsigned full = 0xffffffffu;
    const int lane8 = threadIdx.x & 7;
    Box6 b;
    for (int a = 0; a < 3; ++a) { b.lo[a] = FLT_MAX; b.hi[a] = -FLT_MAX; }
    if (kid >= 0) b = f.nbox[kid];
    Box6 all = b;
    for (int o = 4; o > 0; o >>= 1)
        for (int a = 0; a < 3; ++a) {
            all.lo[a] = fminf(all.lo[a], __shfl_xor_sync(full, all.lo[a], o));
            all.hi[a] = fmaxf(all.hi[a], __shfl_xor_sync(full, all.hi[a], o));
        }
    float d[3];
    for (int a = 0; a < 3; ++a) d[a] = 0.5f * (b.lo[a] + b.hi[a]) - 0.5f * (all.lo[a] + all.hi[a]);
    // Slot assignment: slot s prefers children towards (s&1 ? +x : -x, s&2 ? +y : -y,
    // s&4 ? +z : -z); greedy over (score, kid, slot) in decreasing score, ties in kid/slot order.
    unsigned used = 0u, owner = 0u;     // slots taken; nibble s: the child in slot s
    bool placed = kid < 0;
    for (int round = 0; round < 8; ++round) {
        float best = -FLT_MAX;
        int bs = -1;
        if (!placed) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (used & (1u << s)) continue;
                const float score = (s & 1 ? d[0] : -d[0]) + (s & 2 ? d[1] : -d[1]) + (s & 4 ? d[2] : -d[2]);
                if (score > best || bs < 0) { best = score; bs = s; }
            }
            if (!(best >= -FLT_MAX)) best = -FLT_MAX;   // a NaN score ranks last
        }
        int who = placed ? 8 : lane8;    // 8: nothing to place
        int slot = bs;
        for (int o = 4; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(full, best, o);
            const int ow = __shfl_xor_sync(full, who, o), os = __shfl_xor_sync(full, slot, o);
            if (ow < 8 && (who == 8 || ob > best || (ob == best && ow < who))) { best = ob; who = ow; slot = os; }
        }
        if (__ballot_sync(full, who < 8) == 0u) break;
        if (who < 8) {
            used |= 1u << slot;
            owner |= (unsigned)who << (4 * slot);
            if (who == lane8) placed = true;
        }
    }
    // From here lane s holds slot s.
    const bool valid = (used >> lane8) & 1u;
    const int src = (owner >> (4 * lane8)) & 7;
    const int k = __shfl_sync(full, kid, src, 8);
    for (int a = 0; a < 3; ++a) {
        const float l = __shfl_sync(full, b.lo[a], src, 8), h = __shfl_sync(full, b.hi[a], src, 8);
        b.lo[a] = valid ? l : 0.0f;
        b.hi[a] = valid ? h : 0.0f;
    }
    const bool internal = valid && !is_leafy(f, k);
    const int count = valid && !internal ? prim_count(f, k) : 0;
    const unsigned imask = octet_ballot(internal);
    if (active && internal) next_queue[__popc(imask & ((1u << lane8) - 1u))] = k;
    int poff = count;
    for (int o = 1; o < 8; o <<= 1) {
        const int up = __shfl_up_sync(full, poff, o, 8);
        if (lane8 >= o) poff += up;
    }
    poff -= count;
    if (active && count > 0) {
        // The leaf's primitives, left to right (at most kMaxLeafTris).
        int stack[4], sp = 0, n = 0;
        stack[sp++] = k;
        while (sp > 0) {
            const int x = stack[--sp];
            if (x < f.n) {
                emit_prim(lo, x, (long long)prim_base + poff + n);
                ++n;
            } else {
                stack[sp++] = f.right[x - f.n];
                stack[sp++] = f.left[x - f.n];
            }
        }
    }
    uint32_t* w = reinterpret_cast<uint32_t*>(out);
    uint32_t meta = (uint32_t)((count << 5) | (count > 0 ? poff : 0)) << (8 * (lane8 & 3));
    for (int o = 2; o > 0; o >>= 1) meta |= __shfl_xor_sync(full, meta, o);
    if (active && (lane8 & 3) == 0) w[6 + (lane8 >> 2)] = meta;
    float p[3];
    int bexp[3];
    quantize_octet(active, b, valid, w, p, bexp);
    if (active && lane8 == 0) {
        w[0] = __float_as_uint(p[0]);
        w[1] = __float_as_uint(p[1]);
        w[2] = __float_as_uint(p[2]);
        w[3] = (uint32_t)bexp[0] | ((uint32_t)bexp[1] << 8) | ((uint32_t)bexp[2] << 16) | (imask << 24);
        w[4] = (uint32_t)child_base;
        w[5] = (uint32_t)prim_base;
    }
}

// All meshes' trees level by level (their roots first, in mesh order), then the instances'.
// Per level: children and counts of the block's queue entries, a barrier, the blocks' scanned
// offsets and the nodes, a barrier. wide_first / tri_first: nodes and triangle records written
// by earlier batches.
__global__ void __launch_bounds__(kBlock) collapse_kernel(Forest f, CollapseArrays c, WideNode* nodes, int wide_first,
                                                          int tri_first, int first_mesh, LeafOut lo, BuildState* st) {
    constexpr int kGroup = kBlock / 8;    // queue entries a block takes at once
    __shared__ int s_int[kGroup], s_prim[kGroup];
    if (*(volatile int*)&st->error != 0) return;   // no trees to collapse
    unsigned target = 0;
    const int tid = threadIdx.x;
    const int oct = tid >> 3;
    const int meshes = f.top_seg >= 0 ? f.n_seg - 1 : f.n_seg;
    int wide = wide_first;
    int prims = tri_first;
    for (int part = 0; part < (f.top_seg >= 0 ? 2 : 1); ++part) {
        int q = part == 0 ? meshes : 1;
        if (part == 1) prims = 0;
        const int* queue = part == 0 ? f.roots : f.roots + f.top_seg;
        int level_first = wide, free_at = wide + q, buf = 0;
        if (part == 0)
            for (int i = blockIdx.x * kBlock + tid; i < q; i += gridDim.x * kBlock) c.mesh_root[first_mesh + i] = wide + i;
        // A level is at least a primitive shorter than the one above: the loop ends.
        while (q > 0) {
            const int chunk = max(kGroup, ((q + (int)gridDim.x - 1) / (int)gridDim.x + kGroup - 1) / kGroup * kGroup);
            const int e0 = (int)min((long long)blockIdx.x * chunk, (long long)q), e1 = min(e0 + chunk, q);
            int sum_int = 0, sum_prim = 0;
            for (int g = e0; g < e1; g += kGroup) {
                const int e = g + oct;
                const bool has = e < e1;
                const int node = has ? queue[e] : -1;
                const int kid = part == 0 ? gather_children(f, node) : gather_largest(f, node);
                const bool lf = kid >= 0 && is_leafy(f, kid);
                const int ni = __popc(octet_ballot(kid >= 0 && !lf));
                int np = lf ? prim_count(f, kid) : 0;
                for (int o = 4; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
                if (!has) continue;
                c.kids[8ll * e + (tid & 7)] = kid;
                if ((tid & 7) == 0) {
                    c.n_int[e] = ni;
                    c.n_prims[e] = np;
                    sum_int += ni;
                    sum_prim += np;
                }
            }
            const int2 mine = block_sum(sum_int, sum_prim);
            if (tid == 0) c.sums[blockIdx.x] = mine;
            if (!grid_barrier(st, target)) return;
            int2 before, total;
            block_prefix(c.sums, gridDim.x, blockIdx.x, before, total);
            int* next = c.queue[buf];
            for (int g = e0; g < e1; g += kGroup) {
                const int e = g + oct;
                const bool has = e < e1;
                __syncthreads();
                if (tid < kGroup) {      // exclusive scan of the group's counts by the first warp
                    const int x = g + tid < e1 ? c.n_int[g + tid] : 0, y = g + tid < e1 ? c.n_prims[g + tid] : 0;
                    int ix = x, iy = y;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int ux = __shfl_up_sync(0xffffffffu, ix, o), uy = __shfl_up_sync(0xffffffffu, iy, o);
                        if (tid >= o) { ix += ux; iy += uy; }
                    }
                    s_int[tid] = before.x + ix - x;
                    s_prim[tid] = before.y + iy - y;
                    before.x += __shfl_sync(0xffffffffu, ix, 31);
                    before.y += __shfl_sync(0xffffffffu, iy, 31);
                }
                __syncthreads();
                const int kid = has ? c.kids[8ll * e + (tid & 7)] : -1;
                write_wide(f, has, kid, free_at + s_int[oct], prims + s_prim[oct], next + s_int[oct],
                           nodes + (level_first + (has ? e : 0)), lo);
            }
            prims += total.y;
            level_first = free_at;
            free_at += total.x;
            q = total.x;
            queue = next;
            buf = 1 - buf;
            if (!grid_barrier(st, target)) return;
        }
        wide = free_at;
        if (blockIdx.x == 0 && tid == 0) {
            if (part == 0) { st->bottom_nodes = wide; st->tri_count = prims; }
            else st->inst_count = prims;
            st->wide_count = wide;
        }
    }
}

// ---------------------------------------------------------------------------------------
// Host driver
// ---------------------------------------------------------------------------------------
bool ck(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    set_error(e == cudaErrorMemoryAllocation ? IMBART_ERR_OUT_OF_MEMORY : IMBART_ERR_CUDA,
              std::string("imbart_scene_build_gpu: ") + what + ": " + cudaGetErrorString(e));
    return false;
}

template <typename T>
bool dmalloc(T** p, size_t n) { *p = nullptr; return ck(cudaMalloc((void**)p, sizeof(T) * std::max<size_t>(n, 1)), "cudaMalloc"); }

int grid(long long n) { return (int)std::max<long long>(1, (n + kBlock - 1) / kBlock); }

// One device allocation carved into arrays: measured first (base null), then laid out.
struct Slab {
    char* base = nullptr;
    size_t used = 0;
    template <typename T>
    void take(T*& p, size_t n) {
        used = (used + 255) & ~(size_t)255;
        p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += sizeof(T) * std::max<size_t>(n, 1);
    }
};

// The builds' scratch is kept between them, one allocation per device and at most kKeptScratch
// bytes of it; a scene's records share one allocation too. An allocation and its release cost
// 0.6 ms here whatever the size: the instanced scene's build took 2.8 ms with five of them (and
// with PLOC tiles of two passes and barriers polled where they count arrivals), 1.6 ms. A build
// takes the kept one, so concurrent builds have their own, and hands it back after its stream is
// done; imbart_invalidate_scenes frees it.
constexpr size_t kKeptScratch = 256ull << 20;
struct KeptScratch {
    char* base = nullptr;
    size_t bytes = 0;
};
std::mutex g_scratch_mutex;
KeptScratch g_scratch[64];

char* take_scratch(int device, size_t& bytes) {
    if (device >= 0 && device < 64) {
        std::lock_guard<std::mutex> lk(g_scratch_mutex);
        KeptScratch& k = g_scratch[device];
        if (k.base && k.bytes >= bytes) {
            char* p = k.base;
            bytes = k.bytes;
            k = KeptScratch{};
            return p;
        }
    }
    char* p = nullptr;
    if (cudaMalloc((void**)&p, bytes) == cudaSuccess) return p;
    (void)cudaGetLastError();
    release_build_scratch();
    return dmalloc(&p, bytes) ? p : nullptr;
}

void give_scratch(int device, char* base, size_t bytes) {
    if (base && device >= 0 && device < 64 && bytes <= kKeptScratch) {
        std::lock_guard<std::mutex> lk(g_scratch_mutex);
        KeptScratch& k = g_scratch[device];
        if (k.bytes < bytes) {
            std::swap(k.base, base);
            k.bytes = bytes;
        }
    }
    cudaFree(base);
}

// Meshes are built together up to this many primitives (IMBART_BUILD_BATCH).
long long batch_prims() {
    const char* v = getenv("IMBART_BUILD_BATCH");
    const long long n = v ? atoll(v) : 0;
    return n > 0 ? n : 32ll << 20;
}
constexpr int kMaxBuildBlocks = 2048;

// Device arrays of a scene build.
struct BuildArrays {
    // inputs of the whole scene
    float* verts;
    long long* vert_first;
    int *vert_count, *tri_offset, *mesh_root;
    imbart_instance_desc* insts;
    long long* inst_bounds;
    BuildState* state;
    // one batch of meshes
    int4* idx;
    int* seg_first;
    int* cb;
    Box6 *boxes, *nbox, *clbox[2];
    uint64_t* keys[2];
    int *vals[2], *cl[2], *sg[2], *link, *left, *right, *cnt;
    float *cost, *area;
    uint8_t *leafy, *split;
    int *roots, *queue[2], *kids, *n_int, *n_prims;
    int2* sums;
    void* temp;
    // the scene's records when there is one batch: they move to an allocation of their size
    WideNode* nodes;
    WideTri* tris;
    WideInst* winsts;

    void layout(Slab& s, long long verts_n, int n_meshes, int n_insts, size_t n, int max_seg, size_t temp_bytes,
                size_t nodes_n, size_t tris_n, size_t insts_n) {
        s.take(verts, 3 * (size_t)verts_n);
        s.take(vert_first, n_meshes); s.take(vert_count, n_meshes); s.take(tri_offset, n_meshes);
        s.take(mesh_root, n_meshes);
        s.take(insts, n_insts); s.take(inst_bounds, 6 * (size_t)n_insts);
        s.take(state, 1);
        s.take(idx, n); s.take(seg_first, (size_t)max_seg + 1); s.take(cb, 6 * (size_t)max_seg);
        s.take(boxes, n); s.take(nbox, 2 * n);
        for (int k = 0; k < 2; ++k) {
            s.take(clbox[k], n); s.take(keys[k], n); s.take(vals[k], n); s.take(cl[k], n); s.take(sg[k], n);
            s.take(queue[k], n);
        }
        s.take(link, n); s.take(left, n); s.take(right, n); s.take(cnt, n); s.take(cost, n); s.take(leafy, n);
        s.take(area, 7 * n); s.take(split, 8 * n);
        s.take(roots, max_seg);
        s.take(kids, 8 * n); s.take(n_int, n); s.take(n_prims, n);
        s.take(sums, kMaxBuildBlocks);
        char* t = nullptr;
        s.take(t, temp_bytes);
        temp = t;
        s.take(nodes, nodes_n); s.take(tris, tris_n); s.take(winsts, insts_n);
    }
};

// Blocks of a cooperative launch of `kernel` for `items` work items of which a block takes
// `per` at once: all can be resident together, at most four per SM (more only make the barriers
// slower).
int coop_blocks(const void* kernel, int device, long long items, int per) {
    int sms = 1, occ = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kBlock, 0);
    const long long cap = std::min<long long>((long long)sms * std::max(1, std::min(occ, 4)), kMaxBuildBlocks);
    return (int)std::max<long long>(1, std::min<long long>(cap, (items + per - 1) / per));
}

int build_error(int code) {
    switch (code) {
        case kErrIndex:
            set_error(IMBART_ERR_BAD_SCENE, "imbart_scene_build_gpu: vertex index out of range");
            return IMBART_ERR_BAD_SCENE;
        case kErrProgress:
            set_error(IMBART_ERR_CUDA, "imbart_scene_build_gpu: clustering made no progress");
            return IMBART_ERR_CUDA;
        default:
            set_error(IMBART_ERR_CUDA, "imbart_scene_build_gpu: the build's blocks did not meet");
            return IMBART_ERR_CUDA;
    }
}

// What a build is given, with the meshes' places in the scene.
struct SceneInput {
    const imbart_mesh_desc* meshes;
    int n_meshes;
    const imbart_instance_desc* insts;
    int n_insts;
    long long total_tris = 0, total_verts = 0;
    std::vector<long long> vert_first;
    std::vector<int> vert_count, tri_offset;
};

int build_batches(const SceneInput& in, long long limit, int device, cudaStream_t st, imbart_scene** out);

int build_scene_gpu(const imbart_mesh_desc* meshes, int n_meshes, const imbart_instance_desc* insts, int n_insts,
                    int device, void* stream, imbart_scene** out, float* build_ms) {
    *out = nullptr;
    if (!meshes || n_meshes <= 0 || !insts || n_insts <= 0) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_scene_build_gpu: invalid argument");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    SceneInput in{meshes, n_meshes, insts, n_insts};
    in.vert_first.resize(n_meshes);
    in.vert_count.resize(n_meshes);
    in.tri_offset.resize(n_meshes);
    long long max_n = n_insts;
    for (int k = 0; k < n_meshes; ++k) {
        const imbart_mesh_desc& m = meshes[k];
        if (!m.vertices || !m.indices || m.n_vertices <= 0 || m.n_tris <= 0) {
            set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_scene_build_gpu: empty mesh");
            return IMBART_ERR_INVALID_ARGUMENT;
        }
        in.vert_first[k] = in.total_verts;
        in.vert_count[k] = m.n_vertices;
        in.tri_offset[k] = m.tri_offset;
        in.total_verts += m.n_vertices;
        in.total_tris += m.n_tris;
        max_n = std::max<long long>(max_n, m.n_tris);
    }
    for (int i = 0; i < n_insts; ++i)
        if (insts[i].mesh < 0 || insts[i].mesh >= n_meshes) {
            set_error(IMBART_ERR_BAD_SCENE, "imbart_scene_build_gpu: instance of an unknown mesh");
            return IMBART_ERR_BAD_SCENE;
        }
    if (in.total_tris >= (1ll << 30) || max_n >= (1ll << 29)) {
        set_error(IMBART_ERR_LIMIT, "imbart_scene_build_gpu: scene too large");
        return IMBART_ERR_LIMIT;
    }
    int prev = 0;
    cudaGetDevice(&prev);
    if (!ck(cudaSetDevice(device), "cudaSetDevice")) return IMBART_ERR_CUDA;
    const auto t0 = std::chrono::steady_clock::now();
    const int code = imbart_last_error();
    const std::string msg = imbart_last_error_string();
    int rc = build_batches(in, batch_prims(), device, (cudaStream_t)stream, out);
    if (rc == IMBART_ERR_OUT_OF_MEMORY) {
        // Building the meshes together takes up to 540 B a triangle; one after another they take the
        // records (128 B) and the scratch of the largest (281 B).
        (void)cudaGetLastError();
        release_build_scratch();
        rc = build_batches(in, 0, device, (cudaStream_t)stream, out);
        if (rc == 0) set_error(code, msg);
    }
    if (rc == 0 && build_ms)
        *build_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
    cudaSetDevice(prev);
    return rc;
}

// Builds the scene in batches of consecutive meshes of at most `limit` primitives (or one mesh); the
// last one takes the instances too where they fit. A scene of one batch goes into one allocation.
int build_batches(const SceneInput& in, long long limit, int device, cudaStream_t st, imbart_scene** out) {
    const imbart_mesh_desc* meshes = in.meshes;
    const imbart_instance_desc* insts = in.insts;
    const int n_meshes = in.n_meshes, n_insts = in.n_insts;
    const long long total_tris = in.total_tris, total_verts = in.total_verts;
    const std::vector<long long>& vert_first = in.vert_first;
    const std::vector<int>&vert_count = in.vert_count, &tri_offset = in.tri_offset;
    std::vector<int> batch_end;
    long long cap = 0, in_batch = 0;
    int max_seg = 1, batch_first = 0;
    auto close_batch = [&](int k) {
        batch_end.push_back(k);
        cap = std::max(cap, in_batch);
        max_seg = std::max(max_seg, k - batch_first);
        batch_first = k;
        in_batch = 0;
    };
    for (int k = 0; k < n_meshes; ++k) {
        if (in_batch > 0 && in_batch + meshes[k].n_tris > limit) close_batch(k);
        in_batch += meshes[k].n_tris;
    }
    if (in_batch + n_insts > limit) close_batch(n_meshes);
    batch_end.push_back(n_meshes);
    cap = std::max(cap, in_batch + n_insts);
    max_seg = std::max(max_seg, n_meshes - batch_first + 1);
    const bool single = batch_end.size() == 1;
    // Wide nodes: at most one per binary internal node, plus one per mesh (and the top).
    const long long node_cap = total_tris + n_insts + n_meshes + 2;
    size_t temp_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (const int*)nullptr, (int*)nullptr, (int)cap, 0, 64);
    Slab slab;
    BuildArrays A{};
    auto layout = [&] {
        slab.used = 0;
        A.layout(slab, total_verts, n_meshes, n_insts, (size_t)cap, max_seg, temp_bytes, single ? node_cap : 0,
                 single ? (size_t)total_tris : 0, single ? (size_t)n_insts : 0);
    };
    layout();
    size_t scratch_bytes = slab.used;
    char* base = take_scratch(device, scratch_bytes);
    WideNode* nodes = nullptr;
    WideTri* tris = nullptr;
    WideInst* winsts = nullptr;
    int* error_flags = nullptr;
    char* block = nullptr;
    bool good = base && (single || (dmalloc(&nodes, node_cap) && dmalloc(&tris, total_tris) &&
                                    dmalloc(&winsts, n_insts) && dmalloc(&error_flags, 4)));
    auto copy = [&](void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
        return ck(cudaMemcpyAsync(dst, src, bytes, kind, st), "cudaMemcpyAsync");
    };
    BuildState hs{};
    if (good) {
        slab.base = base;
        layout();
        if (single) { nodes = A.nodes; tris = A.tris; winsts = A.winsts; }
        good = copy(A.vert_first, vert_first.data(), sizeof(long long) * n_meshes, cudaMemcpyHostToDevice) &&
               copy(A.vert_count, vert_count.data(), sizeof(int) * n_meshes, cudaMemcpyHostToDevice) &&
               copy(A.tri_offset, tri_offset.data(), sizeof(int) * n_meshes, cudaMemcpyHostToDevice) &&
               copy(A.insts, insts, sizeof(imbart_instance_desc) * (size_t)n_insts, cudaMemcpyDefault);
    }
    int rc = 0;
    std::vector<int> seg_first;
    for (size_t b = 0; b < batch_end.size() && good; ++b) {
        const int k0 = b == 0 ? 0 : batch_end[b - 1], k1 = batch_end[b];
        const bool last = b + 1 == batch_end.size();
        const int n_seg = k1 - k0 + (last ? 1 : 0), top_seg = last ? k1 - k0 : -1;
        seg_first.assign(n_seg + 1, 0);
        for (int k = k0; k < k1 && good; ++k) {
            const imbart_mesh_desc& m = meshes[k];
            seg_first[k - k0 + 1] = seg_first[k - k0] + m.n_tris;
            good = copy(A.verts + 3 * vert_first[k], m.vertices, sizeof(float) * 3 * (size_t)m.n_vertices,
                        cudaMemcpyDefault) &&
                   copy(A.idx + seg_first[k - k0], m.indices, sizeof(int4) * (size_t)m.n_tris, cudaMemcpyDefault);
        }
        const int n_tris = seg_first[k1 - k0];
        if (last) seg_first[n_seg] = n_tris + n_insts;
        const int n = seg_first[n_seg];
        int seg_bits = 0;
        while ((1ll << seg_bits) < n_seg) ++seg_bits;
        const int bits = std::min(21, (64 - seg_bits) / 3);
        hs.arrived = hs.open = 0;
        hs.error = 0;
        good = good && copy(A.seg_first, seg_first.data(), sizeof(int) * (n_seg + 1), cudaMemcpyHostToDevice) &&
               copy(A.state, &hs, sizeof(hs), cudaMemcpyHostToDevice);
        if (!good) break;
        bounds_init_kernel<<<grid(6ll * n_seg), kBlock, 0, st>>>(A.cb, 6 * n_seg);
        tri_boxes_kernel<<<grid(n_tris), kBlock, 0, st>>>(A.verts, A.idx, n_tris, A.seg_first, n_seg, A.vert_first + k0,
                                                          A.vert_count + k0, A.boxes, A.cb, &A.state->error);
        if (last) {
            int max_verts = 0;
            for (int i = 0; i < n_insts; ++i) max_verts = std::max(max_verts, vert_count[insts[i].mesh]);
            const unsigned chunks = (unsigned)std::max(1, std::min((max_verts + kVertChunk - 1) / kVertChunk,
                                                                   kInstBlocks / n_insts));
            inst_bounds_init_kernel<<<grid(6ll * n_insts), kBlock, 0, st>>>(A.inst_bounds, 6 * n_insts);
            inst_bounds_kernel<<<dim3(n_insts, chunks), kBlock, 0, st>>>(A.insts, A.verts, A.vert_first, A.vert_count,
                                                                        A.inst_bounds);
            inst_boxes_kernel<<<grid(n_insts), kBlock, 0, st>>>(A.inst_bounds, n_insts, A.boxes + n_tris, top_seg, A.cb);
        }
        morton_kernel<<<grid(n), kBlock, 0, st>>>(A.boxes, n, A.seg_first, n_seg, bits, A.cb, A.keys[0], A.vals[0]);
        good = ck(cudaGetLastError(), "build kernels") &&
               ck(cub::DeviceRadixSort::SortPairs(A.temp, temp_bytes, A.keys[0], A.keys[1], A.vals[0], A.vals[1], n, 0,
                                                  3 * bits + seg_bits, st), "SortPairs");
        if (!good) break;
        Forest f{n, n_seg, top_seg, A.seg_first, A.nbox, A.left, A.right, A.cnt, A.cost, A.leafy, A.area, A.split,
                 A.roots};
        PlocArrays p{};
        p.sorted = A.vals[1];
        p.boxes = A.boxes;
        for (int k = 0; k < 2; ++k) { p.cl[k] = A.cl[k]; p.sg[k] = A.sg[k]; p.box[k] = A.clbox[k]; }
        p.link = A.link;
        p.sums = A.sums;
        BuildState* state = A.state;
        void* pargs[] = {&f, &p, &state};
        good = ck(cudaLaunchCooperativeKernel((const void*)ploc_kernel,
                                              dim3(coop_blocks((const void*)ploc_kernel, device, n, kOwn)),
                                              dim3(kBlock), pargs, 0, st), "clustering launch") &&
               ck(cudaMemsetAsync(A.state, 0, offsetof(BuildState, error), st), "cudaMemsetAsync");
        if (!good) break;
        CollapseArrays c{{A.queue[0], A.queue[1]}, A.kids, A.n_int, A.n_prims, A.sums, A.mesh_root};
        LeafOut lo{n_tris, A.verts, A.idx, A.seg_first, n_seg, A.vert_first + k0, A.tri_offset + k0, tris, A.insts,
                   A.mesh_root, winsts};
        WideNode* wn = nodes;
        int wide_first = hs.wide_count, tri_first = hs.tri_count, first_mesh = k0;
        void* cargs[] = {&f, &c, &wn, &wide_first, &tri_first, &first_mesh, &lo, &state};
        good = ck(cudaLaunchCooperativeKernel((const void*)collapse_kernel,
                                              dim3(coop_blocks((const void*)collapse_kernel, device, n / 8, kBlock / 8)),
                                              dim3(kBlock), cargs, 0, st), "collapse launch") &&
               copy(&hs, A.state, sizeof(hs), cudaMemcpyDeviceToHost) &&
               ck(cudaStreamSynchronize(st), "cudaStreamSynchronize");
        note_launches(last ? 8 : 5);
        if (good && hs.error) {
            rc = build_error(hs.error);
            good = false;
        }
    }
    if (good && single) {
        // The records into one allocation of their size, error flags last.
        Slab out;
        auto place = [&] {
            out.used = 0;
            out.take(nodes, hs.wide_count);
            out.take(tris, hs.tri_count);
            out.take(winsts, n_insts);
            out.take(error_flags, 4);
        };
        place();
        good = dmalloc(&block, out.used);
        if (good) {
            out.base = block;
            place();
            good = copy(nodes, A.nodes, sizeof(WideNode) * (size_t)hs.wide_count, cudaMemcpyDeviceToDevice) &&
                   copy(tris, A.tris, sizeof(WideTri) * (size_t)hs.tri_count, cudaMemcpyDeviceToDevice) &&
                   copy(winsts, A.winsts, sizeof(WideInst) * (size_t)n_insts, cudaMemcpyDeviceToDevice);
        }
    }
    if (good)
        good = ck(cudaMemsetAsync(error_flags, 0, 4 * sizeof(int), st), "cudaMemsetAsync") &&
               ck(cudaStreamSynchronize(st), "cudaStreamSynchronize");
    if (!good) cudaStreamSynchronize(st);   // nothing of a failed build still runs on the scratch
    give_scratch(device, base, scratch_bytes);
    if (good) {
        int direct_inst = -1;
        WideInst w{};
        std::memcpy(w.m, insts[0].world_to_obj, sizeof(w.m));
        if (n_insts == 1 && identity_instance(w)) direct_inst = insts[0].id;
        // The meshes' roots are the first nodes of their batch.
        int direct_root = -1;
        if (direct_inst >= 0 && n_meshes == 1) direct_root = 0;
        *out = scene_adopt_device_arrays(device, block, nodes, hs.wide_count, hs.wide_count - hs.bottom_nodes, tris,
                                         hs.tri_count, winsts, n_insts, error_flags, hs.bottom_nodes, direct_root,
                                         direct_inst);
    } else {
        cudaFree(block);
        if (!single) { cudaFree(nodes); cudaFree(tris); cudaFree(winsts); cudaFree(error_flags); }
        if (!rc) rc = imbart_last_error() ? imbart_last_error() : IMBART_ERR_CUDA;
    }
    return rc;
}

// ---------------------------------------------------------------------------------------
// Refit: the vertices moved, the topology did not. Triangle records take their triangle's
// new vertices; node boxes are recomputed bottom-up (bottom levels, then the instances'
// world boxes, then the top level) and requantized with the build's conservative
// arithmetic. Eight lanes start at each node without internal children, a lane per slot, and
// climb: the last child of a parent to finish refits the parent (a counter per node, back at
// its start value afterwards, so that it serves every refit of the scene). The chain of a leaf's
// ancestors bounds a refit, hence eight lanes for a node's children, boxes and bytes. Measured
// (B200), 512 k triangles, with 65,536 rays traced after it: 960 us with a thread per node and
// scratch allocated by every refit, 276 us.
// ---------------------------------------------------------------------------------------

// Parent of every internal child (-1: none) and the count of internal children of each node.
__global__ void refit_links_kernel(const WideNode* __restrict__ nodes, int n_nodes, int* parent, int* pending) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n_nodes) return;
    const WideNode nd = nodes[n];
    pending[n] = __popc(nd.imask);
    int rank = 0;
    for (int s = 0; s < 8; ++s)
        if (nd.imask & (1u << s)) parent[nd.child_base + rank++] = n;
}

__device__ __forceinline__ Box6 empty_box() {
    Box6 b;
    for (int a = 0; a < 3; ++a) { b.lo[a] = FLT_MAX; b.hi[a] = -FLT_MAX; }
    return b;
}

// Another thread's finished box, read past the L1 cache.
__device__ __forceinline__ Box6 load_box_cg(const Box6* p) {
    const float* f = reinterpret_cast<const float*>(p);
    Box6 b;
    for (int a = 0; a < 3; ++a) { b.lo[a] = __ldcg(f + a); b.hi[a] = __ldcg(f + 3 + a); }
    return b;
}

// The moved vertices of a bottom-level refit.
struct MovedVerts {
    const float* verts;
    long long n_verts;
    const int4* tri_verts;
    int n_tri_ids;
    int* error;
};

// Moves triangle record t to its new vertices and returns its box; a bad id or index sets
// *error and leaves the record.
__device__ __forceinline__ Box6 move_triangle(WideTri* t, const MovedVerts& m) {
    float4* r = reinterpret_cast<float4*>(t);
    float4 v0 = r[0], v1 = r[1], v2 = r[2];
    const int id = __float_as_int(v0.w);
    if (id < 0 || id >= m.n_tri_ids) {
        atomicExch(m.error, 1);
    } else {
        const int4 i = __ldg(m.tri_verts + id);
        if (i.x < 0 || i.y < 0 || i.z < 0 || i.x >= m.n_verts || i.y >= m.n_verts || i.z >= m.n_verts) {
            atomicExch(m.error, 2);
        } else {
            const float *a = m.verts + 3ll * i.x, *b = m.verts + 3ll * i.y, *c = m.verts + 3ll * i.z;
            v0.x = __ldg(a); v0.y = __ldg(a + 1); v0.z = __ldg(a + 2);
            v1.x = __ldg(b); v1.y = __ldg(b + 1); v1.z = __ldg(b + 2);
            v2.x = __ldg(c); v2.y = __ldg(c + 1); v2.z = __ldg(c + 2);
            r[0] = v0; r[1] = v1; r[2] = v2;
        }
    }
    Box6 x;
    x.lo[0] = fminf(v0.x, fminf(v1.x, v2.x)); x.hi[0] = fmaxf(v0.x, fmaxf(v1.x, v2.x));
    x.lo[1] = fminf(v0.y, fminf(v1.y, v2.y)); x.hi[1] = fmaxf(v0.y, fmaxf(v1.y, v2.y));
    x.lo[2] = fminf(v0.z, fminf(v1.z, v2.z)); x.hi[2] = fmaxf(v0.z, fmaxf(v1.z, v2.z));
    return x;
}

// Refits node n of an active octet: lane s takes slot s (leaf slots: their triangles, moved, or
// instances; internal slots: the boxes their refits stored); the node's own box goes to exact.
__device__ __forceinline__ void refit_node(bool active, WideNode* nodes, int n, WideTri* tris, const MovedVerts& mv,
                                           const Box6* inst_boxes, Box6* exact) {
    const unsigned full = 0xffffffffu;
    const int lane8 = threadIdx.x & 7;
    uint32_t* w = reinterpret_cast<uint32_t*>(nodes + n);
    Box6 b = empty_box();
    bool valid = false;
    uint32_t imask = 0u;
    if (active) {
        imask = w[3] >> 24;
        if ((imask >> lane8) & 1u) {
            valid = true;
            b = load_box_cg(exact + w[4] + __popc(imask & ((1u << lane8) - 1u)));
        } else {
            const uint32_t meta = (w[6 + (lane8 >> 2)] >> (8 * (lane8 & 3))) & 0xffu;
            const int count = (int)(meta >> 5);
            const long long first = (long long)w[5] + (meta & 31u);
            valid = count > 0;
            for (int k = 0; k < count; ++k)
                b = merge(b, inst_boxes ? inst_boxes[first + k] : move_triangle(tris + first + k, mv));
        }
    }
    Box6 all = b;
    for (int o = 4; o > 0; o >>= 1)
        for (int a = 0; a < 3; ++a) {
            all.lo[a] = fminf(all.lo[a], __shfl_xor_sync(full, all.lo[a], o));
            all.hi[a] = fmaxf(all.hi[a], __shfl_xor_sync(full, all.hi[a], o));
        }
    if (!valid)
        for (int a = 0; a < 3; ++a) b.lo[a] = b.hi[a] = 0.0f;
    float p[3];
    int bexp[3];
    quantize_octet(active, b, valid, w, p, bexp);
    if (active && lane8 == 0) {
        w[0] = __float_as_uint(p[0]);
        w[1] = __float_as_uint(p[1]);
        w[2] = __float_as_uint(p[2]);
        w[3] = (uint32_t)bexp[0] | ((uint32_t)bexp[1] << 8) | ((uint32_t)bexp[2] << 16) | (imask << 24);
        float* e = reinterpret_cast<float*>(exact + n);
        for (int a = 0; a < 3; ++a) { e[a] = all.lo[a]; e[3 + a] = all.hi[a]; }
    }
}

__global__ void __launch_bounds__(kBlock) refit_up_kernel(WideNode* nodes, int first, int last,
                                                          const int* __restrict__ parent, int* pending, WideTri* tris,
                                                          MovedVerts mv, const Box6* inst_boxes, Box6* exact) {
    const unsigned full = 0xffffffffu;
    const int lane8 = threadIdx.x & 7;
    int n = first + (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 3);
    bool active = n < last && nodes[n].imask == 0;
    while (__ballot_sync(full, active) != 0u) {
        refit_node(active, nodes, n, tris, mv, inst_boxes, exact);
        int up = -1;
        if (active && lane8 == 0) {
            __threadfence();
            const int p = parent[n];
            if (p >= 0 && atomicSub(pending + p, 1) == 1) {   // the parent's last child to finish goes on
                __threadfence();
                pending[p] = __popc(nodes[p].imask);
                up = p;
            }
        }
        __syncwarp();    // the shuffle alone would not order the other lanes' reads behind lane 0's fence
        n = __shfl_sync(full, up, 0, 8);
        active = n >= 0;
    }
}

// World box of each instance record: its mesh root's box through the object-to-world
// transform (the inverse of the stored world-to-object rows, in double precision), corners
// rounded outward and widened by 2^-20 of their magnitude.
__global__ void refit_inst_boxes_kernel(const WideInst* __restrict__ insts, int n, const Box6* exact, Box6* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const WideInst w = insts[i];
    const Box6 b = load_box_cg(exact + w.root);
    double a[3][3], t[3];
    for (int r = 0; r < 3; ++r) {
        for (int c = 0; c < 3; ++c) a[r][c] = w.m[4 * r + c];
        t[r] = w.m[4 * r + 3];
    }
    const double det = a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[2][1]) -
                       a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0]) +
                       a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0]);
    double inv[3][3];
    inv[0][0] = (a[1][1] * a[2][2] - a[1][2] * a[2][1]) / det;
    inv[0][1] = (a[0][2] * a[2][1] - a[0][1] * a[2][2]) / det;
    inv[0][2] = (a[0][1] * a[1][2] - a[0][2] * a[1][1]) / det;
    inv[1][0] = (a[1][2] * a[2][0] - a[1][0] * a[2][2]) / det;
    inv[1][1] = (a[0][0] * a[2][2] - a[0][2] * a[2][0]) / det;
    inv[1][2] = (a[0][2] * a[1][0] - a[0][0] * a[1][2]) / det;
    inv[2][0] = (a[1][0] * a[2][1] - a[1][1] * a[2][0]) / det;
    inv[2][1] = (a[0][1] * a[2][0] - a[0][0] * a[2][1]) / det;
    inv[2][2] = (a[0][0] * a[1][1] - a[0][1] * a[1][0]) / det;
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (int c = 0; c < 8; ++c) {
        const double x = (c & 1) ? b.hi[0] : b.lo[0], y = (c & 2) ? b.hi[1] : b.lo[1], z = (c & 4) ? b.hi[2] : b.lo[2];
        const double px = x - t[0], py = y - t[1], pz = z - t[2];   // object = A world + t  =>  world = A^-1 (object - t)
        for (int r = 0; r < 3; ++r) {
            const double v = inv[r][0] * px + inv[r][1] * py + inv[r][2] * pz;
            lo[r] = fmin(lo[r], v);
            hi[r] = fmax(hi[r], v);
        }
    }
    Box6 o;
    double m = 0.0;
    for (int r = 0; r < 3; ++r) m = fmax(m, fmax(fabs(lo[r]), fabs(hi[r])));
    const double pad = m * 9.5367431640625e-07 + 1e-30;
    for (int r = 0; r < 3; ++r) {
        o.lo[r] = __double2float_rd(lo[r] - pad);
        o.hi[r] = __double2float_ru(hi[r] + pad);
    }
    out[i] = o;
}

int refit_scene(imbart_scene* scene, const float* verts, long long n_verts, const int* tri_verts, int n_tri_ids,
                cudaStream_t st) {
    imbart_scene_info info;
    const void *vn = nullptr, *vt = nullptr, *vi = nullptr;
    if (imbart_scene_get_info(scene, &info) != 0 || imbart_scene_get_device_arrays(scene, &vn, &vt, &vi) != 0)
        return imbart_last_error() ? imbart_last_error() : IMBART_ERR_INVALID_ARGUMENT;
    if (!vn || info.wide_nodes <= 0 || info.wide_nodes > INT_MAX || info.top_nodes <= 0 ||
        info.top_nodes > info.wide_nodes) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_scene_refit: scene without its own node array");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    WideNode* nodes = static_cast<WideNode*>(const_cast<void*>(vn));
    WideTri* tris = static_cast<WideTri*>(const_cast<void*>(vt));
    const WideInst* insts = static_cast<const WideInst*>(vi);
    const int n_nodes = (int)info.wide_nodes, first_top = (int)(info.wide_nodes - info.top_nodes);
    // Scratch of the scene's refits, kept with the scene: parents and child counters (filled by the
    // first refit, the topology never changes), node and instance boxes, the error word.
    Slab slab;
    Box6 *exact = nullptr, *inst_boxes = nullptr;
    int *parent = nullptr, *pending = nullptr, *error = nullptr;
    auto layout = [&] {
        slab.used = 0;
        slab.take(exact, n_nodes);
        slab.take(inst_boxes, info.instances);
        slab.take(parent, n_nodes);
        slab.take(pending, n_nodes);
        slab.take(error, 1);
    };
    layout();
    bool fresh = false;
    slab.base = static_cast<char*>(scene_refit_scratch(scene, slab.used, &fresh));
    if (!slab.base) return imbart_last_error() ? imbart_last_error() : IMBART_ERR_OUT_OF_MEMORY;
    layout();
    bool good = ck(cudaMemsetAsync(error, 0, sizeof(int), st), "cudaMemsetAsync");
    if (good && fresh) {
        good = ck(cudaMemsetAsync(parent, 0xff, sizeof(int) * (size_t)n_nodes, st), "cudaMemsetAsync");
        if (good) refit_links_kernel<<<grid(n_nodes), kBlock, 0, st>>>(nodes, n_nodes, parent, pending);
        note_launches(1);
    }
    if (good) {
        const MovedVerts mv{verts, n_verts, reinterpret_cast<const int4*>(tri_verts), n_tri_ids, error};
        if (first_top > 0)
            refit_up_kernel<<<grid(8ll * first_top), kBlock, 0, st>>>(nodes, 0, first_top, parent, pending, tris, mv,
                                                                     nullptr, exact);
        refit_inst_boxes_kernel<<<grid(info.instances), kBlock, 0, st>>>(insts, (int)info.instances, exact,
                                                                        inst_boxes);
        refit_up_kernel<<<grid(8ll * info.top_nodes), kBlock, 0, st>>>(nodes, first_top, n_nodes, parent, pending, tris,
                                                                      mv, inst_boxes, exact);
        note_launches(first_top > 0 ? 3 : 2);
        int h_error = 0;
        good = ck(cudaGetLastError(), "refit launch") &&
               ck(cudaMemcpyAsync(&h_error, error, sizeof(int), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync") &&
               ck(cudaStreamSynchronize(st), "cudaStreamSynchronize");
        if (good && h_error) {
            set_error(IMBART_ERR_INVALID_ARGUMENT, h_error == 1 ? "imbart_scene_refit: a triangle id beyond n_tri_ids"
                                                                : "imbart_scene_refit: a vertex index out of range");
            good = false;
        }
    }
    if (!good && fresh) scene_refit_scratch(scene, 0, &fresh);   // links may be missing: start over next time
    return good ? 0 : (imbart_last_error() ? imbart_last_error() : IMBART_ERR_CUDA);
}

}  // namespace

void release_build_scratch() {
    std::lock_guard<std::mutex> lk(g_scratch_mutex);
    int prev = 0;
    cudaGetDevice(&prev);
    for (int d = 0; d < 64; ++d) {
        if (!g_scratch[d].base) continue;
        cudaSetDevice(d);
        cudaFree(g_scratch[d].base);
        g_scratch[d] = KeptScratch{};
    }
    cudaSetDevice(prev);
}

}  // namespace imbart

extern "C" int imbart_scene_refit(imbart_scene* scene, const float* vertices, long long n_vertices,
                                  const int* tri_vertices, int n_tri_ids, void* stream) {
    if (!scene || !vertices || !tri_vertices || n_vertices <= 0 || n_tri_ids <= 0) {
        imbart::set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_scene_refit: invalid argument");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    imbart_scene_info info;
    if (imbart_scene_get_info(scene, &info) != 0) return imbart_last_error();
    int prev = 0;
    cudaGetDevice(&prev);
    int dev = prev;
    // The scene's device: the one its arrays live on (pointer attributes).
    const void* vn = nullptr;
    const void* vt = nullptr;
    const void* vi = nullptr;
    imbart_scene_get_device_arrays(scene, &vn, &vt, &vi);
    cudaPointerAttributes attr;
    if (vn && cudaPointerGetAttributes(&attr, vn) == cudaSuccess && attr.type == cudaMemoryTypeDevice) dev = attr.device;
    cudaSetDevice(dev);
    const int rc = imbart::refit_scene(scene, vertices, n_vertices, tri_vertices, n_tri_ids, (cudaStream_t)stream);
    cudaSetDevice(prev);
    return rc;
}

extern "C" imbart_scene* imbart_scene_build_gpu(const imbart_mesh_desc* meshes, int n_meshes,
                                                const imbart_instance_desc* instances, int n_instances, int device,
                                                void* stream, float* build_ms) {
    imbart_scene* s = nullptr;
    imbart::build_scene_gpu(meshes, n_meshes, instances, n_instances, device, stream, &s, build_ms);
    return s;
}
