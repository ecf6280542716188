// LOR preprocessing on the GPU: the reference's host numpy pass
// src/python/srf/preprocess/function/on_tor_lors.py (recon_process :251-262,
// map_process :243-248) as three kernels.
//
// Per event (float32 arithmetic in numpy's operation order; numpy never fuses a*b+c,
// so every product and sum here is a separately rounded __fmul_rn/__fadd_rn):
//   f  = (dx^2+dy^2)^2 / (x1^2+x2^2+y1^2+y2^2) / L^2 / 2          (:137-166)
//   dominant axis with the reference tie rules                      (:70-77)
//   swap endpoints so the dominant coordinate grows, negating TOF    (:175-193)
//   recon only: TOF centre C and the cut to C -/+ 3 sigma            (:196-229)
//   column permutation that puts the dominant axis last              (:246-247, :259-260)
//
// Output order is the reference's: the x group, then y, then z; inside a group the
// events that kept their orientation (ascending index), then the swapped ones
// (ascending index) — np.intersect1d sorts, SwapPointsOrder vstacks positive/negative.
// That is a stable partition into six buckets (axis, swapped), done with a per-tile
// count, a scan over tiles and a stable scatter (ballot ranks inside each warp).

#include <mutex>

#include "lor_prep.cuh"
#include "srf_common.cuh"

namespace srf {
namespace {

constexpr int kThreads = 512;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;

struct PreParams {
    const float *events;
    int64_t n, stride;
    int recon, cut;
    float limit;
    unsigned char *bucket;   // [n]
    int *tile_counts;        // [ntiles * kBuckets]
    int64_t *tile_offsets;   // [ntiles * kBuckets]
    int64_t *bucket_base;    // [kBuckets + 1]
    int64_t *group_counts;   // [3] output
    float *out;
    int ntiles;
};

template <bool RECON>
__global__ void __launch_bounds__(kThreads) classify_kernel(const PreParams p) {
    __shared__ int counts[kBuckets];
    if (threadIdx.x < kBuckets) counts[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kTile;
    int local[kBuckets] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int64_t i = base + (int64_t)k * kThreads + threadIdx.x;
        if (i < p.n) {
            const Rec r = process<RECON>(p.events + i * p.stride, p.cut, p.limit);
            p.bucket[i] = (unsigned char)r.bucket;
#pragma unroll
            for (int b = 0; b < kBuckets; b++) local[b] += (r.bucket == b);
        }
    }
#pragma unroll
    for (int b = 0; b < kBuckets; b++) {
        int v = local[b];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(&counts[b], v);
    }
    __syncthreads();
    if (threadIdx.x < kBuckets) p.tile_counts[blockIdx.x * kBuckets + threadIdx.x] = counts[threadIdx.x];
}

// One block: exclusive scan of the tile counts of each bucket, then of the bucket
// totals; bucket_base[b] is where bucket b starts in the output. The six buckets of a tile
// are read and scanned together (one after the other, every pass touched every line of the
// counts again: 13 us for 1953 tiles, now 10).
__global__ void __launch_bounds__(1024) scan_kernel(const PreParams p) {
    __shared__ int64_t totals[kBuckets];
    __shared__ int warp_sums[kBuckets][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t carry[kBuckets] = {0, 0, 0, 0, 0, 0};
    for (int start = 0; start < p.ntiles; start += 1024) {
        const int i = start + threadIdx.x;
        int v[kBuckets], x[kBuckets];
#pragma unroll
        for (int b = 0; b < kBuckets; b++)
            x[b] = v[b] = i < p.ntiles ? p.tile_counts[(int64_t)i * kBuckets + b] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {  // inclusive scans inside the warp
#pragma unroll
            for (int b = 0; b < kBuckets; b++) {
                const int y = __shfl_up_sync(0xffffffffu, x[b], o);
                if (lane >= o) x[b] += y;
            }
        }
        if (lane == 31) {
#pragma unroll
            for (int b = 0; b < kBuckets; b++) warp_sums[b][wid] = x[b];
        }
        __syncthreads();
        if (wid < kBuckets) {
            int w = warp_sums[wid][lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            warp_sums[wid][lane] = w;  // a chunk of 1024 tiles counts at most 2^22 events
        }
        __syncthreads();
#pragma unroll
        for (int b = 0; b < kBuckets; b++) {
            if (i < p.ntiles)
                p.tile_offsets[(int64_t)i * kBuckets + b] =
                    carry[b] + (wid ? warp_sums[b][wid - 1] : 0) + x[b] - v[b];
            carry[b] += warp_sums[b][31];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int64_t acc = 0;
#pragma unroll
        for (int b = 0; b < kBuckets; b++) {
            totals[b] = carry[b];
            p.bucket_base[b] = acc;
            acc += carry[b];
        }
        p.bucket_base[kBuckets] = acc;
        for (int a = 0; a < 3; a++) p.group_counts[a] = totals[2 * a] + totals[2 * a + 1];
    }
}

// A tile's events to their places. Every event's place comes first, for the whole tile at
// once (warp ballots in index order, then one scan per bucket over the tile's 128 warp
// counts). Then, 512 events at a time: the events come in as one contiguous stretch through
// shared memory, their records go to a staging buffer compacted by bucket, and each bucket's
// run leaves as one contiguous stretch (a record is 28-40 bytes, so one thread per record
// would touch a new sector per lane and column, in and out). Bound by HBM: 8M events, 224 MB
// in and 320 MB out, 268 -> 240 us; ranking each 512 events by themselves, with one thread
// adding up the warps' counts, had six barriers per step where this has two.
template <bool RECON>
__global__ void __launch_bounds__(kThreads, 3) scatter_kernel(const PreParams p) {
    constexpr int ncols = RECON ? 10 : 7, nin = RECON ? 7 : 6;
    constexpr int kWarps = kThreads / 32;
    __shared__ int before[kBuckets][kItems * kWarps];  // counts, then events of the tile before
    __shared__ unsigned short place[kItems][kThreads];  // in the step's staging buffer
    __shared__ int start[kItems][kBuckets + 1];         // bucket runs of the staging buffer
    __shared__ int64_t shift[kItems][kBuckets];         // from there to the output, in floats
    __shared__ float stage[kThreads * ncols];
    __shared__ float events[kThreads * nin];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kTile;
    {
        int bucket[kItems], rank[kItems];
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const int64_t i = base + (int64_t)k * kThreads + threadIdx.x;
            bucket[k] = i < p.n ? (int)p.bucket[i] : kBuckets;
        }
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            rank[k] = 0;
#pragma unroll
            for (int q = 0; q < kBuckets; q++) {
                const unsigned m = __ballot_sync(0xffffffffu, bucket[k] == q);
                if (bucket[k] == q) rank[k] = __popc(m & ((1u << lane) - 1u));
                if (lane == 0) before[q][k * kWarps + wid] = __popc(m);
            }
        }
        __syncthreads();
        if (wid < kBuckets) {  // exclusive scan of this bucket's kItems x kWarps counts
            constexpr int kEach = kItems * kWarps / 32;
            int v[kEach], sum = 0;
#pragma unroll
            for (int u = 0; u < kEach; u++) {
                v[u] = before[wid][lane * kEach + u];
                sum += v[u];
            }
            int x = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            x -= sum;
#pragma unroll
            for (int u = 0; u < kEach; u++) {
                before[wid][lane * kEach + u] = x;
                x += v[u];
            }
        }
        __syncthreads();
        if (threadIdx.x < kItems) {
            const int k = threadIdx.x;
            int at = 0;
            for (int q = 0; q < kBuckets; q++) {
                const int run = before[q][k * kWarps];
                const int next = k + 1 < kItems
                                     ? before[q][(k + 1) * kWarps]
                                     : p.tile_counts[(int64_t)blockIdx.x * kBuckets + q];
                start[k][q] = at;
                shift[k][q] = (p.bucket_base[q] +
                               p.tile_offsets[(int64_t)blockIdx.x * kBuckets + q] + run - at) *
                              ncols;
                at += next - run;
            }
            start[k][kBuckets] = at;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const int q = bucket[k];
            place[k][threadIdx.x] =
                q < kBuckets ? (unsigned short)(start[k][q] + before[q][k * kWarps + wid] -
                                                before[q][k * kWarps] + rank[k])
                             : (unsigned short)kThreads;
        }
    }
    const bool packed = p.stride == nin;
    float in[nin];
    auto fetch = [&](int k) {  // this thread's share of step k's events
        const int64_t first = base + (int64_t)k * kThreads;
        const int left = (int)min((p.n - first) * nin, (int64_t)kThreads * nin);
#pragma unroll
        for (int u = 0; u < nin; u++) {
            const int e = u * kThreads + threadIdx.x;
            in[u] = e < left ? __ldg(p.events + first * nin + e) : 0.0f;
        }
    };
    if (packed) fetch(0);
#pragma unroll 1
    for (int k = 0; k < kItems; k++) {
        const int64_t i = base + (int64_t)k * kThreads + threadIdx.x;
        if (base + (int64_t)k * kThreads >= p.n) break;  // the whole block
        if (packed) {
#pragma unroll
            for (int u = 0; u < nin; u++) events[u * kThreads + threadIdx.x] = in[u];
            __syncthreads();
            if (k + 1 < kItems) fetch(k + 1);
        }
        const int pos = place[k][threadIdx.x];
        if (pos < kThreads) {
            const Rec r = packed ? process<RECON>(events + threadIdx.x * nin, p.cut, p.limit)
                                 : process<RECON>(p.events + i * p.stride, p.cut, p.limit);
#pragma unroll
            for (int c = 0; c < ncols; c++) stage[pos * ncols + c] = r.v[c];
        }
        __syncthreads();
        const int total = start[k][kBuckets] * ncols;
        int q = 0, end = start[k][1] * ncols;
        float *dst = p.out + shift[k][0];
        for (int e = threadIdx.x; e < total; e += kThreads) {
            while (e >= end) {
                q++;
                end = start[k][q + 1] * ncols;
                dst = p.out + shift[k][q];
            }
            dst[e] = stage[e];
        }
        if (!packed) __syncthreads();  // else the next step's barrier comes first
    }
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace
}  // namespace srf

using namespace srf;

extern "C" int64_t srf_preprocess_workspace_size(int64_t num_events) {
    if (num_events < 0) return -1;
    const int64_t ntiles = (num_events + kTile - 1) / kTile;
    return (int64_t)(align256((size_t)num_events) + align256(sizeof(int) * ntiles * kBuckets) +
                     align256(sizeof(int64_t) * ntiles * kBuckets) +
                     align256(sizeof(int64_t) * (kBuckets + 1)));
}

namespace {
int preprocess(const float *events, int64_t n, int64_t stride, int recon, double tof_res,
               float *out, int64_t *group_counts, void *workspace, int64_t workspace_bytes,
               cudaStream_t stream) {
    if (n < 0 || !group_counts) return SRF_ERR_INVALID_ARGUMENT;
    if (stride < (recon ? 7 : 6)) return SRF_ERR_INVALID_ARGUMENT;
    if (n > 0 && (!events || !out || !workspace)) return SRF_ERR_INVALID_ARGUMENT;
    if (workspace_bytes < srf_preprocess_workspace_size(n)) return SRF_ERR_INVALID_ARGUMENT;
    if (!(tof_res == tof_res)) return SRF_ERR_INVALID_ARGUMENT;
    PreParams p{};
    p.events = events;
    p.n = n;
    p.stride = stride;
    p.recon = recon;
    p.cut = recon && tof_res < 10000.0;
    p.limit = (float)(tof_res * 0.15 / 2.35482005 * 3);
    p.ntiles = (int)((n + kTile - 1) / kTile);
    char *w = static_cast<char *>(workspace);
    p.bucket = reinterpret_cast<unsigned char *>(w);
    w += align256((size_t)n);
    p.tile_counts = reinterpret_cast<int *>(w);
    w += align256(sizeof(int) * p.ntiles * kBuckets);
    p.tile_offsets = reinterpret_cast<int64_t *>(w);
    w += align256(sizeof(int64_t) * p.ntiles * kBuckets);
    p.bucket_base = reinterpret_cast<int64_t *>(w);
    p.group_counts = group_counts;
    p.out = out;
    if (n == 0) {
        cudaError_t e = cudaMemsetAsync(group_counts, 0, 3 * sizeof(int64_t), stream);
        if (e != cudaSuccess) {
            set_cuda_error(e);
            return SRF_ERR_CUDA;
        }
        return SRF_OK;
    }
    if (recon) {
        classify_kernel<true><<<p.ntiles, kThreads, 0, stream>>>(p);
        scan_kernel<<<1, 1024, 0, stream>>>(p);
        scatter_kernel<true><<<p.ntiles, kThreads, 0, stream>>>(p);
        count_launches(3);
    } else {
        classify_kernel<false><<<p.ntiles, kThreads, 0, stream>>>(p);
        scan_kernel<<<1, 1024, 0, stream>>>(p);
        scatter_kernel<false><<<p.ntiles, kThreads, 0, stream>>>(p);
        count_launches(3);
    }
    return check_launch();
}
}  // namespace

extern "C" int srf_recon_process(const float *events, int64_t num_events, int64_t event_stride,
                                 double tof_res, float *out, int64_t *group_counts,
                                 void *workspace, int64_t workspace_bytes, void *stream) {
    return preprocess(events, num_events, event_stride, 1, tof_res, out, group_counts, workspace,
                      workspace_bytes, (cudaStream_t)stream);
}

extern "C" int srf_map_process(const float *lors, int64_t num_lors, int64_t lor_stride,
                               float *out, int64_t *group_counts, void *workspace,
                               int64_t workspace_bytes, void *stream) {
    return preprocess(lors, num_lors, lor_stride, 0, 1.0e4, out, group_counts, workspace,
                      workspace_bytes, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------
// recon_process without any allocation.
//
// Some callers cannot allocate device memory at the time they preprocess events: an
// acquisition-side reconstruction service that owns a fixed memory budget and forbids
// allocations after start-up, or code on a latency-critical path where cudaMalloc's
// implicit device synchronisation is not acceptable. srf_recon_process needs a scratch
// workspace for its stable partition; this variant takes that scratch from a buffer
// that is part of the library itself, a file-scope __device__ array of fixed size.
//
// * The buffer holds the workspace for up to SRF_RECON_PROCESS_NOALLOC_MAX_EVENTS events
//   (8.1 MiB); every GPU that loads the library keeps it until the process exits.
//   Larger calls are rejected with SRF_ERR_UNSUPPORTED before anything is launched.
// * Host code cannot use the array's name as a device address, so the first call on
//   each device (with that device current) asks the runtime for the address with
//   cudaGetSymbolAddress and caches it; that first call should therefore happen before
//   any stream capture. The cache lives as long as the process: after cudaDeviceReset
//   the address is stale, and the library must not be called on that device again.
// * All calls on a device share the one buffer and it keeps the last call's contents.
//   Nothing in it needs to start at zero: every byte a call reads was written earlier
//   in the same call. Calls whose kernels overlap on the GPU (concurrent streams, or
//   several host threads) race on the buffer; serialise them on one stream.
// * No cudaMalloc, cudaFree or allocating library routine is called.

namespace srf {
namespace {

constexpr int64_t kNoAllocMaxEvents = SRF_RECON_PROCESS_NOALLOC_MAX_EVENTS;
constexpr size_t align256c(size_t v) { return (v + 255) & ~(size_t)255; }
constexpr int64_t kNoAllocTiles = (kNoAllocMaxEvents + kTile - 1) / kTile;
constexpr size_t kNoAllocScratchBytes =
    align256c((size_t)kNoAllocMaxEvents) + align256c(sizeof(int) * kNoAllocTiles * kBuckets) +
    align256c(sizeof(int64_t) * kNoAllocTiles * kBuckets) +
    align256c(sizeof(int64_t) * (kBuckets + 1));

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device (looked up once).
int noalloc_scratch(void **ptr) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return SRF_ERR_CUDA;
    }
    if (dev < 0 || dev >= kNoAllocMaxDevices) return SRF_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e == cudaSuccess && !p) e = cudaErrorInvalidSymbol;  // never a null address
        if (e != cudaSuccess) {
            set_cuda_error(e);
            return SRF_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = p;
    }
    *ptr = g_noalloc_ptr[dev];
    return SRF_OK;
}

}  // namespace
}  // namespace srf

extern "C" int srf_recon_process_noalloc(const float *events, int64_t num_events,
                                         int64_t event_stride, double tof_res, float *out,
                                         int64_t *group_counts, void *stream) {
    if (num_events < 0) return SRF_ERR_INVALID_ARGUMENT;
    if (num_events > kNoAllocMaxEvents) return SRF_ERR_UNSUPPORTED;
    void *scratch = nullptr;
    const int st = noalloc_scratch(&scratch);
    if (st != SRF_OK) return st;
    return preprocess(events, num_events, event_stride, 1, tof_res, out, group_counts, scratch,
                      (int64_t)kNoAllocScratchBytes, (cudaStream_t)stream);
}
