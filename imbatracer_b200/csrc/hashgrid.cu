// Photon hash grid on the GPU: build (bounding box, hashed counting sort) and batched
// k-capped radius queries, with the semantics of the reference's HashGrid
// (src/imbatracer/rangesearch/rangesearch.h):
//   build  :25-75   r^2, cell size (2r in the reference, a parameter here), bbox of the
//                   photon positions inflated by 0.1 % of its extent per side, counting sort
//                   into `table_size` buckets (2 * photon count in the reference)
//   hash   :137-148 ((x*73856093) ^ (y*19349663) ^ (z*83492791)) mod table_size on unsigned
//                   coordinates, coordinates = floor((p - bbox.min) / cell size)
//   query  :77-129  outside the bbox -> nothing; home cell plus the nearer neighbour per
//                   axis (8 buckets in the reference's order, a bucket hit twice is scanned
//                   twice), squared distance <= r^2, k nearest kept by insertion sort
// Every float operation is explicitly rounded (no contraction) so that cell indices and
// distances equal the reference's bit for bit. Within a bucket photons are placed in the order
// an atomic counter met them, as in the reference's parallel scatter (rangesearch.h:68-74); the
// query returns its k photons ordered by (distance, photon index).
//
// A build is five launches: small grids are bound by the launches and their gaps, large ones by
// memory (the photons twice, the table three times, the sorted photons once). The bounding box's
// and the tile sums' finishing steps run in the last block of the launch that produces them, and
// a photon's place in its bucket is the count it got when it was counted, so the scatter needs no
// cursors. Measured (B200): 20,011 photons with 2,000 queries 44.0 us in nine launches, 34.9 us;
// 1.74 M photons into 2^22 buckets 80 us less.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cfloat>
#include <mutex>
#include <string>

#include "hashgrid_query.cuh"
#include "imbart_internal.h"

struct imbart_hashgrid {
    int device = 0;
    int n = 0;              // photons in the current build
    int table = 0;          // buckets in the current build
    int sorted_cap = 0, place_cap = 0, ends_cap = 0;
    float4* sorted = nullptr;   // position xyz + original index (int bits) in bucket order
    int* cell_ends = nullptr;   // inclusive end of each bucket
    int2* place = nullptr;      // bucket of each photon and its place there (scratch)
    int* block_sums = nullptr;  // scan scratch
    int block_sums_cap = 0;
    unsigned* state = nullptr;  // 8 words, zero between builds (GridState)
    bool state_zeroed = false;  // by an earlier build
    float* params = nullptr;    // device: lo[3], hi[3], radius, r^2, cell, inv_cell
    float host_params[10] = {};
    float cell_factor = 2.0f;   // cell size / radius of the current build
};

namespace imbart {
namespace {

constexpr int kBlock = 256;
constexpr int kScanItems = 8;                 // items per thread in the scan kernels
constexpr int kScanTile = kBlock * kScanItems;
constexpr int kMaxK = kGridMaxK;

bool ok(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    set_error(e == cudaErrorMemoryAllocation ? IMBART_ERR_OUT_OF_MEMORY : IMBART_ERR_CUDA,
              std::string(what) + ": " + cudaGetErrorString(e));
    return false;
}

// Order-preserving float -> unsigned mapping; every float maps above 0, so 0 stands for "none".
__device__ __forceinline__ unsigned float_to_ordered(float f) {
    const unsigned i = __float_as_uint(f);
    return (i & 0x80000000u) ? ~i : i | 0x80000000u;
}
__device__ __forceinline__ float ordered_to_float(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? u & 0x7fffffffu : ~u);
}

// Words of a build's running state: the box as maxima (of ~ordered for the low side), then the
// counts of finished blocks of the two launches whose last block goes on. All zero between
// builds: the last block that reads a word clears it.
enum GridState { kStateLo = 0, kStateHi = 3, kStateBoxDone = 6, kStateScanDone = 7, kStateWords = 8 };

// True in the block of the launch that finishes last (its threads then see the other blocks'
// writes); clears the count.
__device__ __forceinline__ bool last_block(unsigned* done) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
        if (last) *done = 0u;
        __threadfence();
    }
    __syncthreads();
    return last;
}

// Zeroes the bucket counts and finds the exact min / max of the positions (order-independent, so
// bit-identical to a serial pass). The last block inflates the box (rangesearch.h:44-46) and
// derives the cell parameters (:27-30).
__global__ void __launch_bounds__(kBlock) bounds_kernel(const float* __restrict__ pos, int stride, int n,
                                                        int* __restrict__ counts, int table, float radius,
                                                        float cell_factor, float* __restrict__ prm, unsigned* state) {
    __shared__ unsigned s_box[6];
    const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    if (threadIdx.x < 6) s_box[threadIdx.x] = 0u;
    if (((size_t)counts & 15) == 0) {
        int4* c4 = reinterpret_cast<int4*>(counts);
        for (int i = first; i < table / 4; i += step) c4[i] = make_int4(0, 0, 0, 0);
        if (first < (table & 3)) counts[(table & ~3) + first] = 0;
    } else {
        for (int i = first; i < table; i += step) counts[i] = 0;
    }
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int i = first; i < n; i += step) {
        const float* p = pos + (size_t)i * stride;
        for (int a = 0; a < 3; ++a) {
            const float v = p[a];    // a NaN is no position: it is kept out of both
            lo[a] = v < lo[a] ? v : lo[a];
            hi[a] = v > hi[a] ? v : hi[a];
        }
    }
    __syncthreads();
    for (int a = 0; a < 3; ++a) {
        const unsigned l = __reduce_max_sync(0xffffffffu, ~float_to_ordered(lo[a]));
        const unsigned h = __reduce_max_sync(0xffffffffu, float_to_ordered(hi[a]));
        if ((threadIdx.x & 31) == 0) { atomicMax(s_box + a, l); atomicMax(s_box + 3 + a, h); }
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(state + threadIdx.x, s_box[threadIdx.x]);
    if (!last_block(state + kStateBoxDone) || threadIdx.x != 0) return;
    float blo[3], bhi[3], ext[3];
    for (int a = 0; a < 3; ++a) {
        blo[a] = ordered_to_float(~__ldcg(state + kStateLo + a));
        bhi[a] = ordered_to_float(__ldcg(state + kStateHi + a));
        state[kStateLo + a] = 0u;
        state[kStateHi + a] = 0u;
    }
    for (int a = 0; a < 3; ++a) ext[a] = __fsub_rn(bhi[a], blo[a]);
    for (int a = 0; a < 3; ++a) bhi[a] = __fadd_rn(bhi[a], __fmul_rn(ext[a], 0.001f));
    for (int a = 0; a < 3; ++a) blo[a] = __fsub_rn(blo[a], __fmul_rn(ext[a], 0.001f));
    const float cell = __fmul_rn(radius, cell_factor);
    for (int a = 0; a < 3; ++a) { prm[a] = blo[a]; prm[3 + a] = bhi[a]; }
    prm[6] = radius;
    prm[7] = __fmul_rn(radius, radius);
    prm[8] = cell;
    prm[9] = __fdiv_rn(1.0f, cell);
}

__device__ __forceinline__ int cell_of_point(const float* prm, float px, float py, float pz, uint32_t table) {
    const float inv = prm[9];
    const int cx = (int)floorf(__fmul_rn(inv, __fsub_rn(px, prm[0])));
    const int cy = (int)floorf(__fmul_rn(inv, __fsub_rn(py, prm[1])));
    const int cz = (int)floorf(__fmul_rn(inv, __fsub_rn(pz, prm[2])));
    return hash_cell((uint32_t)cx, (uint32_t)cy, (uint32_t)cz, table);
}

// Counts the photons of every bucket; the count a photon gets is its place in the bucket.
__global__ void count_kernel(const float* __restrict__ pos, int stride, int n, const float* __restrict__ prm,
                             uint32_t table, int* __restrict__ counts, int2* __restrict__ place) {
    __shared__ float sp[10];
    if (threadIdx.x < 10) sp[threadIdx.x] = prm[threadIdx.x];
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* p = pos + (size_t)i * stride;
        const int c = cell_of_point(sp, p[0], p[1], p[2], table);
        place[i] = make_int2(c, atomicAdd(counts + c, 1));
    }
}

// A thread's kScanItems consecutive counts, as 16-byte loads where the array allows it.
__device__ __forceinline__ void load_items(const int* in, int base, int n, int v[kScanItems]) {
    if (base + kScanItems <= n && ((size_t)in & 15) == 0) {
        for (int k = 0; k < kScanItems; k += 4) {
            const int4 q = *reinterpret_cast<const int4*>(in + base + k);
            v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
        }
    } else {
        for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0;
    }
}

// Inclusive scan of one value per thread over the block (kBlock threads).
__device__ __forceinline__ int block_scan(int v) {
    __shared__ int warp_sums[kBlock / 32];
    int incl = v;
    for (int off = 1; off < 32; off <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, off);
        if ((int)(threadIdx.x & 31) >= off) incl += t;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = incl;
    __syncthreads();
    for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) incl += warp_sums[w];
    return incl;
}

// Sums of the tiles of kScanTile counts; the last block turns them into exclusive offsets.
__global__ void __launch_bounds__(kBlock) scan_tiles_kernel(const int* __restrict__ in, int n, int* tile_sums,
                                                            unsigned* state) {
    __shared__ int carry;
    int v[kScanItems], s = 0;
    load_items(in, blockIdx.x * kScanTile + threadIdx.x * kScanItems, n, v);
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    s = block_scan(s);
    if (threadIdx.x == kBlock - 1) tile_sums[blockIdx.x] = s;
    if (!last_block(state + kStateScanDone)) return;
    const int n_tiles = gridDim.x;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < n_tiles; base += kScanTile) {
        const int first = base + threadIdx.x * kScanItems;
        int sum = 0;
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = first + k < n_tiles ? __ldcg(tile_sums + first + k) : 0;
            sum += v[k];
        }
        const int incl = block_scan(sum);
        int run = carry + incl - sum;
        for (int k = 0; k < kScanItems; ++k) {
            if (first + k < n_tiles) tile_sums[first + k] = run;
            run += v[k];
        }
        __syncthreads();
        if (threadIdx.x == kBlock - 1) carry = run;
        __syncthreads();
    }
}

// Turns the counts into the buckets' inclusive ends, in place. Also clears the state words, so
// that builds which overlapped on one grid (an error of the caller's) cannot spoil later ones.
__global__ void __launch_bounds__(kBlock) scan_apply_kernel(int* ends, int n, const int* __restrict__ tile_off,
                                                            unsigned* state) {
    if (blockIdx.x == 0 && threadIdx.x < kStateWords) state[threadIdx.x] = 0u;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems], s = 0;
    load_items(ends, base, n, v);
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    int run = tile_off[blockIdx.x] + block_scan(s) - s;
    for (int k = 0; k < kScanItems; ++k) { run += v[k]; v[k] = run; }
    if (base + kScanItems <= n && ((size_t)ends & 15) == 0) {
        for (int k = 0; k < kScanItems; k += 4)
            *reinterpret_cast<int4*>(ends + base + k) = make_int4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < n) ends[base + k] = v[k];
    }
}

__global__ void scatter_kernel(const float* __restrict__ pos, int stride, int n, const int2* __restrict__ place,
                               const int* __restrict__ ends, float4* __restrict__ sorted) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* p = pos + (size_t)i * stride;
        const int2 at = place[i];
        sorted[__ldg(ends + at.x) - 1 - at.y] = make_float4(p[0], p[1], p[2], __int_as_float(i));
    }
}

// One warp per query (the search is grid_query_knn_warp).
template <int kCap>
__global__ void __launch_bounds__(128, 10) query_warp_kernel(const float4* __restrict__ sorted,
                                                         const int* __restrict__ ends, const float* __restrict__ prm,
                                                         uint32_t table, const float* __restrict__ queries, int nq,
                                                         int k, int* __restrict__ out_ids, int* __restrict__ out_count,
                                                         float* __restrict__ out_d2) {
    __shared__ float sp[10];
    __shared__ KnnScratch<kCap> scratch[4];
    if (threadIdx.x < 10) sp[threadIdx.x] = prm[threadIdx.x];
    __syncthreads();
    const long long q = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (q >= nq) return;   // uniform across the warp
    const int lane = threadIdx.x & 31;
    const float qx = queries[3 * q + 0], qy = queries[3 * q + 1], qz = queries[3 * q + 2];
    KnnScratch<kCap>& s = scratch[threadIdx.x >> 5];
    const int count = grid_query_knn_warp<kCap>(sorted, ends, sp, table, qx, qy, qz, k, s);
    if (lane == 0) out_count[q] = count;
    for (int i = lane; i < k; i += 32) {
        out_ids[q * k + i] = i < count ? s.id[i] : -1;
        if (out_d2) out_d2[q * k + i] = i < count ? __uint_as_float(s.d2[i]) : 0.0f;
    }
}

// Grid-stride launches over n items: at most 8 blocks per SM of the current device (SM
// counts cached per device index).
int grid_for(int n) {
    static std::mutex mu;
    static int sms_of[64] = {};
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) {
        std::lock_guard<std::mutex> lk(mu);
        if (!sms_of[dev]) cudaDeviceGetAttribute(&sms_of[dev], cudaDevAttrMultiProcessorCount, dev);
        sms = sms_of[dev];
    } else {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    return std::max(1, std::min((n + kBlock - 1) / kBlock, std::max(sms, 1) * 8));
}

// The launches of one build (`state` all zero, as builds leave it).
void launch_build(const float* positions, int stride, int n, float radius, float cell_factor, int table, float4* sorted,
                  int* ends, float* params, int2* place, int* tile_sums, unsigned* state, cudaStream_t st) {
    const int n_tiles = (table + kScanTile - 1) / kScanTile;
    bounds_kernel<<<grid_for(std::max(n, table / 4)), kBlock, 0, st>>>(positions, stride, n, ends, table, radius,
                                                                       cell_factor, params, state);
    const int grid = grid_for(n);
    if (n > 0) count_kernel<<<grid, kBlock, 0, st>>>(positions, stride, n, params, (uint32_t)table, ends, place);
    scan_tiles_kernel<<<n_tiles, kBlock, 0, st>>>(ends, table, tile_sums, state);
    scan_apply_kernel<<<n_tiles, kBlock, 0, st>>>(ends, table, tile_sums, state);
    if (n > 0) scatter_kernel<<<grid, kBlock, 0, st>>>(positions, stride, n, place, ends, sorted);
    note_launches(n > 0 ? 5 : 3);
}

// Grows geometrically: reallocation synchronizes the device, and a grid rebuilt every
// iteration over a slowly growing photon count would otherwise reallocate every time.
template <typename T>
bool grow(T** p, int* cap, int need) {
    if (*cap >= need) return true;
    const int n = (int)std::min<long long>(std::max<long long>(need, (long long)*cap * 3 / 2), INT_MAX);
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    if (!ok(cudaMalloc((void**)p, sizeof(T) * (size_t)std::max(n, 1)), "cudaMalloc")) return false;
    *cap = n;
    return true;
}

}  // namespace

bool hashgrid_device_view(const imbart_hashgrid* g, const void** sorted, const int** cell_ends, const float** params,
                          int* table, int* n) {
    if (!g || g->table == 0) return false;
    *sorted = g->sorted;
    *cell_ends = g->cell_ends;
    *params = g->params;
    *table = g->table;
    *n = g->n;
    return true;
}

}  // namespace imbart

using namespace imbart;

extern "C" {

imbart_hashgrid* imbart_hashgrid_create(int device) {
    imbart_hashgrid* g = new imbart_hashgrid;
    g->device = device;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    // The parameters, then the builds' state words (zeroed by the first build on its stream: a wait
    // for the device here would end a graph capture in progress on another thread).
    const bool good = ok(cudaMalloc((void**)&g->params, sizeof(float) * 16 + sizeof(unsigned) * kStateWords),
                         "cudaMalloc");
    cudaSetDevice(prev);
    if (!good) { cudaFree(g->params); delete g; return nullptr; }
    g->state = reinterpret_cast<unsigned*>(g->params + 16);
    return g;
}

void imbart_hashgrid_destroy(imbart_hashgrid* g) {
    if (!g) return;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    cudaFree(g->sorted); cudaFree(g->cell_ends); cudaFree(g->place); cudaFree(g->block_sums); cudaFree(g->params);
    cudaSetDevice(prev);
    delete g;
}

int imbart_hashgrid_build(imbart_hashgrid* g, const float* positions, int stride, int n, float radius,
                          float cell_factor, int table_size, void* stream) {
    if (!g || n < 0 || (n > 0 && !positions) || stride < 3 || !(radius > 0.0f) || !(cell_factor > 0.0f)) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_build: invalid argument");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    if (table_size <= 0) table_size = std::max(2 * n, 1);   // reference: 2 * photons (rangesearch.h:26)
    cudaStream_t st = (cudaStream_t)stream;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    int rc = 0;
    const int n_tiles = (table_size + kScanTile - 1) / kScanTile;
    if (!grow(&g->sorted, &g->sorted_cap, n) || !grow(&g->place, &g->place_cap, n) ||
        !grow(&g->cell_ends, &g->ends_cap, table_size) || !grow(&g->block_sums, &g->block_sums_cap, n_tiles))
        rc = IMBART_ERR_OUT_OF_MEMORY;
    if (!rc && !g->state_zeroed) {
        // Under capture the zeroing is recorded, not done: the next build repeats it.
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        if (!ok(cudaMemsetAsync(g->state, 0, sizeof(unsigned) * kStateWords, st), "cudaMemsetAsync") ||
            !ok(cudaStreamIsCapturing(st, &capturing), "cudaStreamIsCapturing"))
            rc = IMBART_ERR_CUDA;
        g->state_zeroed = !rc && capturing == cudaStreamCaptureStatusNone;
    }
    if (!rc) {
        launch_build(positions, stride, n, radius, cell_factor, table_size, g->sorted, g->cell_ends, g->params, g->place,
                     g->block_sums, g->state, st);
        if (!ok(cudaGetLastError(), "hash grid build")) {
            rc = IMBART_ERR_CUDA;
            g->state_zeroed = false;
        }
        g->n = n;
        g->table = table_size;
        g->cell_factor = cell_factor;
    }
    cudaSetDevice(prev);
    return rc;
}

int imbart_hashgrid_query(const imbart_hashgrid* g, const float* queries, int nq, int k, int* out_ids,
                          int* out_counts, float* out_d2, void* stream) {
    if (!g || nq < 0 || k < 1 || k > kMaxK || (nq > 0 && (!queries || !out_ids || !out_counts)) || g->table == 0) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_query: invalid argument (k must be 1..64, grid built)");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    if (!(g->cell_factor >= 1.0f)) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_query: the grid's cells are smaller than the radius "
                                               "(build with cell_factor >= 1)");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    if (nq == 0) return 0;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    const auto kernel = k <= 32 ? query_warp_kernel<kKnnCapSmall> : query_warp_kernel<kKnnCapLarge>;
    const long long blocks = ((long long)nq * 32 + 127) / 128;
    kernel<<<(unsigned)blocks, 128, 0, (cudaStream_t)stream>>>(g->sorted, g->cell_ends, g->params, (uint32_t)g->table,
                                                               queries, nq, k, out_ids, out_counts, out_d2);
    note_launches(1);
    const bool good = ok(cudaGetLastError(), "hash grid query");
    cudaSetDevice(prev);
    return good ? 0 : IMBART_ERR_CUDA;
}

}  // extern "C"

namespace imbart {
namespace {
// Staging buffers and a stream of one host thread for the host-array entry points (on one
// device at a time; they move to another device when the grid does).
struct HostStaging {
    int device = -1;
    cudaStream_t stream = nullptr;
    float* in = nullptr;
    size_t in_cap = 0;
    int* ids = nullptr;
    size_t out_cap = 0;
    float* d2 = nullptr;
    size_t d2_cap = 0;
    int* counts = nullptr;
    size_t count_cap = 0;

    void release() {
        cudaFree(in); cudaFree(ids); cudaFree(d2); cudaFree(counts);
        if (stream) cudaStreamDestroy(stream);
        in = nullptr; ids = nullptr; d2 = nullptr; counts = nullptr; stream = nullptr;
        in_cap = out_cap = d2_cap = count_cap = 0;
    }
    ~HostStaging() { if (device >= 0) release(); }

    bool on(int dev) {
        if (device == dev) return true;
        if (device >= 0) {
            int prev = 0;
            cudaGetDevice(&prev);
            cudaSetDevice(device);
            release();
            cudaSetDevice(prev);
        }
        device = dev;
        return ok(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
    }
};

template <typename T>
bool stage(T** p, size_t* cap, size_t need) {
    if (*cap >= need) return true;
    const size_t n = std::max(need, *cap * 3 / 2);
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    if (!ok(cudaMalloc((void**)p, sizeof(T) * n), "cudaMalloc")) return false;
    *cap = n;
    return true;
}

thread_local HostStaging t_staging;
}  // namespace
}  // namespace imbart

extern "C" {

int imbart_hashgrid_build_host(imbart_hashgrid* g, const float* positions, int stride, int n, float radius,
                               float cell_factor, int table_size) {
    if (!g || n < 0 || (n > 0 && !positions) || stride < 3) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_build_host: invalid argument");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    HostStaging& h = t_staging;
    const size_t floats = (size_t)std::max(n, 1) * (size_t)stride;
    int rc = 0;
    if (!h.on(g->device) || !stage(&h.in, &h.in_cap, floats)) rc = IMBART_ERR_CUDA;
    if (!rc && n > 0 &&
        !ok(cudaMemcpyAsync(h.in, positions, sizeof(float) * (size_t)n * stride, cudaMemcpyHostToDevice, h.stream),
            "cudaMemcpyAsync"))
        rc = IMBART_ERR_CUDA;
    if (!rc) rc = imbart_hashgrid_build(g, h.in, stride, n, radius, cell_factor, table_size, h.stream);
    if (!rc && !ok(cudaStreamSynchronize(h.stream), "imbart_hashgrid_build_host")) rc = IMBART_ERR_CUDA;
    cudaSetDevice(prev);
    return rc;
}

int imbart_hashgrid_query_host(const imbart_hashgrid* g, const float* queries, int nq, int k, int* out_ids,
                               int* out_counts, float* out_d2) {
    if (!g || nq < 0 || k < 1 || k > kMaxK || (nq > 0 && (!queries || !out_ids || !out_counts))) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_query_host: invalid argument");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    if (nq == 0) return 0;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    HostStaging& h = t_staging;
    const size_t nk = (size_t)nq * (size_t)k;
    int rc = 0;
    if (!h.on(g->device) || !stage(&h.in, &h.in_cap, (size_t)nq * 3) || !stage(&h.ids, &h.out_cap, nk) ||
        !stage(&h.counts, &h.count_cap, (size_t)nq))
        rc = IMBART_ERR_CUDA;
    if (!rc && out_d2 && !stage(&h.d2, &h.d2_cap, nk)) rc = IMBART_ERR_CUDA;
    if (!rc && !ok(cudaMemcpyAsync(h.in, queries, sizeof(float) * 3 * (size_t)nq, cudaMemcpyHostToDevice, h.stream),
                   "cudaMemcpyAsync"))
        rc = IMBART_ERR_CUDA;
    if (!rc) rc = imbart_hashgrid_query(g, h.in, nq, k, h.ids, h.counts, out_d2 ? h.d2 : nullptr, h.stream);
    if (!rc && !(ok(cudaMemcpyAsync(out_ids, h.ids, sizeof(int) * nk, cudaMemcpyDeviceToHost, h.stream), "D2H") &&
                 ok(cudaMemcpyAsync(out_counts, h.counts, sizeof(int) * (size_t)nq, cudaMemcpyDeviceToHost, h.stream),
                    "D2H") &&
                 (!out_d2 || ok(cudaMemcpyAsync(out_d2, h.d2, sizeof(float) * nk, cudaMemcpyDeviceToHost, h.stream),
                                "D2H")) &&
                 ok(cudaStreamSynchronize(h.stream), "imbart_hashgrid_query_host")))
        rc = IMBART_ERR_CUDA;
    cudaSetDevice(prev);
    return rc;
}

int imbart_hashgrid_get_params(const imbart_hashgrid* g, float* params10, int* n, int* table_size) {
    if (!g) { set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_get_params"); return IMBART_ERR_INVALID_ARGUMENT; }
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    bool good = true;
    if (params10) good = ok(cudaMemcpy(params10, g->params, sizeof(float) * 10, cudaMemcpyDeviceToHost), "cudaMemcpy");
    cudaSetDevice(prev);
    if (n) *n = g->n;
    if (table_size) *table_size = g->table;
    return good ? 0 : IMBART_ERR_CUDA;
}

int imbart_hashgrid_get_arrays(const imbart_hashgrid* g, const void** sorted, const int** cell_ends) {
    if (!g) { set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_get_arrays"); return IMBART_ERR_INVALID_ARGUMENT; }
    if (sorted) *sorted = g->sorted;
    if (cell_ends) *cell_ends = g->cell_ends;
    return 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Hash-grid build that allocates nothing.
//
// Some callers must not allocate device memory at all: a server that admits work against a
// fixed HBM budget accounts for every byte up front, and cudaMalloc / cudaFree synchronize
// the device, stalling the other requests' streams; hosts that own all device memory
// through their own arena hand out only buffers they sized themselves. For them the build's
// scratch (bucket and place per photon, scan tile sums, state words) lives in one
// statically sized device array below, held by every GPU that loads the library until the
// process exits: 4 * (2 * 2^20 + 1024 + 8) bytes, about 8 MiB. The caller passes the
// inputs and the outputs it allocated itself.
// ---------------------------------------------------------------------------------------
namespace imbart {
namespace {
constexpr int kNoAllocMaxPhotons = 1 << 20;
constexpr int kNoAllocMaxTable = 1 << 21;
constexpr int kNoAllocTiles = (kNoAllocMaxTable + kScanTile - 1) / kScanTile;
constexpr size_t kNoAllocInts = 2 * (size_t)kNoAllocMaxPhotons + kNoAllocTiles + kStateWords;

static __device__ __align__(256) int g_noalloc_scratch[kNoAllocInts];

// Device address of the scratch array, looked up once per device with that device current.
std::mutex g_noalloc_mutex;
int* g_noalloc_addr[64] = {};
}  // namespace
}  // namespace imbart

extern "C" int imbart_hashgrid_build_noalloc(const float* positions, int stride, int n, float radius,
                                             float cell_factor, int table_size, void* sorted_out,
                                             int* cell_ends_out, float* params_out, void* stream) {
    if (n < 0 || (n > 0 && (!positions || !sorted_out)) || stride < 3 || !(radius > 0.0f) || !(cell_factor > 0.0f) ||
        !cell_ends_out || !params_out) {
        set_error(IMBART_ERR_INVALID_ARGUMENT, "imbart_hashgrid_build_noalloc: invalid argument");
        return IMBART_ERR_INVALID_ARGUMENT;
    }
    if (table_size <= 0) table_size = std::max(2 * n, 1);
    if (n > kNoAllocMaxPhotons || table_size > kNoAllocMaxTable) {
        set_error(IMBART_ERR_LIMIT, "imbart_hashgrid_build_noalloc: at most 1048576 photons and 2097152 buckets "
                                    "(the size of its static scratch); use imbart_hashgrid_build for more");
        return IMBART_ERR_LIMIT;
    }
    // A launch error left pending by earlier work on this thread is cleared here, so that
    // the status returned below describes this call's own launches.
    (void)cudaGetLastError();
    int device = 0;
    if (!ok(cudaGetDevice(&device), "cudaGetDevice")) return IMBART_ERR_CUDA;
    if (device < 0 || device >= 64) {
        set_error(IMBART_ERR_LIMIT, "imbart_hashgrid_build_noalloc: device index above 63");
        return IMBART_ERR_LIMIT;
    }
    int* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mutex);
        if (!g_noalloc_addr[device]) {
            void* addr = nullptr;
            if (!ok(cudaGetSymbolAddress(&addr, g_noalloc_scratch), "cudaGetSymbolAddress")) return IMBART_ERR_CUDA;
            g_noalloc_addr[device] = static_cast<int*>(addr);
        }
        scratch = g_noalloc_addr[device];
    }
    int2* place = reinterpret_cast<int2*>(scratch);
    int* tile_sums = scratch + 2 * kNoAllocMaxPhotons;
    unsigned* state = reinterpret_cast<unsigned*>(tile_sums + kNoAllocTiles);
    // The scratch keeps the previous call's contents: places and tile sums are fully rewritten
    // before they are read, and a build leaves the state words zero as it found them.
    launch_build(positions, stride, n, radius, cell_factor, table_size, static_cast<float4*>(sorted_out), cell_ends_out,
                 params_out, place, tile_sums, state, (cudaStream_t)stream);
    return ok(cudaGetLastError(), "imbart_hashgrid_build_noalloc") ? 0 : IMBART_ERR_CUDA;
}
