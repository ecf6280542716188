// Reordering of preprocessed LOR records by the shape of their tube's section, inside
// blocks of 4096 consecutive records (no counterpart in the reference; an optional step
// between preprocessing and the projectors).
//
// A record's section box spans sqrt((1 - uy^2)/q) by sqrt((1 - ux^2)/q), q = 1 - ux^2 - uy^2,
// with (ux, uy) the in-slice components of its unit direction. The slab kernels hand a
// warp 32 consecutive LORs of a slab and walk the largest box among them, so records of
// similar direction side by side walk fewer voxel slots. Sorting only inside blocks keeps
// every stretch of the per-slab lists a mix of directions, so the persistent grid's equal
// shares stay equal work. The class key quantises both extents to 16 levels over [1, 2)
// (dominant-axis groups have extents in [1, sqrt(3)]); inside a class, records are ordered
// by where the LOR starts along the slice axis (8 mm bins), so a warp's segments cover
// similar slice counts. Records with NaN sort last. The sort is a stable block radix sort,
// so the order is deterministic.

#include <cub/block/block_radix_sort.cuh>

#include "srf_common.cuh"

namespace srf {
namespace {

constexpr int kOrderThreads = 512;
constexpr int kOrderItems = 8;
constexpr int kOrderBlock = kOrderThreads * kOrderItems;  // 4096 records
constexpr int kIndexBits = 12;                            // of a record's place in its block
static_assert(kOrderBlock == 1 << kIndexBits, "");
constexpr int kKeyBits = 17;

__device__ __forceinline__ int direction_class(const float *r) {
    const float dx = r[3] - r[0], dy = r[4] - r[1], dz = r[5] - r[2];
    const float inv = rsqrtf(fmaxf(dx * dx + dy * dy + dz * dz, 1e-30f));
    const float ux2 = dx * dx * inv * inv, uy2 = dy * dy * inv * inv;
    const float q = fmaxf(1.0f - ux2 - uy2, 1e-6f);
    const float bx = sqrtf((1.0f - uy2) / q), by = sqrtf((1.0f - ux2) / q);
    if (!(bx == bx) || !(by == by)) return 255 << 8;
    const int kx = min(15, max(0, (int)((bx - 1.0f) * 16.0f)));
    const int ky = min(15, max(0, (int)((by - 1.0f) * 16.0f)));
    // secondary: where the LOR starts along the slice axis (8 mm bins over +-1 m)
    const float zs = fminf(r[2], r[5]);
    const int kz = (zs == zs) ? min(255, max(0, (int)((zs + 1024.0f) * 0.125f))) : 255;
    return ((kx * 16 + ky) << 8) | kz;
}

// One block per 4096 records: the keys, a stable sort of key << 12 | place (so that the place
// needs no array of its own), then every element of the output in order from the record it
// comes from. The records are read twice, the second time from L2, which leaves 27 KB of
// shared memory per block and three blocks on an SM. Passing records of up to 10 columns
// through shared memory (160 KB) left one block per SM with too few loads in flight, and
// wider ones a thread per record: 6M records of 7 columns 217 -> 202 us, 50k of 11 columns
// (13 blocks: a block's own latency) 53 -> 25 us. Blocks of 1024 threads took 261 and 28 us,
// of 256 threads 235 and 34 us.
__global__ void __launch_bounds__(kOrderThreads, 3)
order_kernel(const float *__restrict__ in, float *__restrict__ out, int64_t n, int ncols,
             int64_t stride) {
    using Sort = cub::BlockRadixSort<unsigned, kOrderThreads, kOrderItems>;
    __shared__ typename Sort::TempStorage tmp;
    __shared__ unsigned short perm[kOrderBlock];
    const int64_t base = (int64_t)blockIdx.x * kOrderBlock;
    const int cnt = (int)min((int64_t)kOrderBlock, n - base);
    const float *src = in + base * stride;
    unsigned key[kOrderItems];
#pragma unroll
    for (int k = 0; k < kOrderItems; k++) {  // any arrangement: the places break ties
        const int j = k * kOrderThreads + threadIdx.x;
        const int c = j < cnt ? direction_class(src + j * stride) : (256 << 8);  // padding last
        key[k] = (unsigned)c << kIndexBits | (unsigned)j;
    }
    Sort(tmp).Sort(key, 0, kIndexBits + kKeyBits);
#pragma unroll
    for (int k = 0; k < kOrderItems; k++)
        perm[threadIdx.x * kOrderItems + k] =
            (unsigned short)(key[k] & (unsigned)(kOrderBlock - 1));
    __syncthreads();
    float *dst = out + base * stride;
    const int64_t total = (int64_t)cnt * ncols;
    const int dr = kOrderThreads / ncols, dc = kOrderThreads - dr * ncols;
    int r = (int)threadIdx.x / ncols, c = (int)threadIdx.x - r * ncols;
#pragma unroll 4
    for (int64_t e = threadIdx.x; e < total; e += kOrderThreads) {
        dst[r * stride + c] = __ldg(src + perm[r] * stride + c);
        r += dr;
        c += dc;
        if (c >= ncols) {
            c -= ncols;
            r++;
        }
    }
}

}  // namespace
}  // namespace srf

using namespace srf;

extern "C" int srf_order_by_direction(const float *records, int64_t num_records, int ncols,
                                      int64_t record_stride, float *out, void *stream) {
    if (num_records < 0 || ncols < 6 || record_stride < ncols) return SRF_ERR_INVALID_ARGUMENT;
    if (num_records == 0) return SRF_OK;
    if (!records || !out || records == out) return SRF_ERR_INVALID_ARGUMENT;
    const int64_t blocks = (num_records + kOrderBlock - 1) / kOrderBlock;
    if (blocks > INT32_MAX) return SRF_ERR_UNSUPPORTED;
    order_kernel<<<(int)blocks, kOrderThreads, 0, (cudaStream_t)stream>>>(
        records, out, num_records, ncols, record_stride);
    count_launches(1);
    return check_launch();
}
