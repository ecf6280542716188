// Image stacks from one axis order to another, and the sum of several such stacks: the
// transposes between the [nx, ny, nz] image and the three axis groups' kernel layouts
// (split_lors.py:54-70, the sum over groups :116-133).
//
// A block moves a 16 x 16 x 16 tile: each source is read along its own fastest axis (runs of
// 64 bytes, whole sectors) into shared memory, added there in the order of the sources, and
// the sum is written along the output's. Bound by HBM or L2: every source is read once and
// the output written once, where a strided copy per source and an add each wrote and read
// the image again and touched a sector per element. One 256 x 256 x 128 image 18 us (torch's strided
// copy 39), three summed ones 19 us (a copy, two adds and a copy: 117).

#include "srf_common.cuh"

namespace srf {
namespace {

constexpr int kSide = 16;
constexpr int kTileY = kSide + 1, kTileX = kSide * kTileY + 1;  // odd strides: no bank conflicts
constexpr int kMaxSources = 3;

struct PermuteArgs {
    float *out;
    int d[3];      // output extents, d[2] fastest
    int tiles[3];  // tiles along each
    int n_src;
    const float *src[kMaxSources];
    int64_t stride[kMaxSources][3];  // element strides along the output's axes
    int fast[kMaxSources];           // the axis of stride 1
    int64_t frame;                   // elements per frame (all stacks)
};

__global__ void __launch_bounds__(kSide *kSide) permute_sum_kernel(const PermuteArgs a) {
    __shared__ float tile[kSide * kTileX];
    int64_t b = blockIdx.x;
    int at[3];
    at[2] = (int)(b % a.tiles[2]) * kSide;
    b /= a.tiles[2];
    at[1] = (int)(b % a.tiles[1]) * kSide;
    b /= a.tiles[1];
    at[0] = (int)(b % a.tiles[0]) * kSide;
    const int64_t frame = b / a.tiles[0] * a.frame;
    const int lo = threadIdx.x % kSide, hi = threadIdx.x / kSide;
    for (int s = 0; s < a.n_src; s++) {
        const int f = a.fast[s], g = f == 0 ? 1 : 0, h = 3 - f - g;
        const int word[3] = {kTileX, kTileY, 1};
        const int i = at[f] + lo, j = at[g] + hi, left = min(kSide, a.d[h] - at[h]);
        const float *q = a.src[s] + frame + (int64_t)i * a.stride[s][f] +
                         (int64_t)j * a.stride[s][g] + (int64_t)at[h] * a.stride[s][h];
        float *t = tile + lo * word[f] + hi * word[g];
        const bool in = i < a.d[f] && j < a.d[g];
        float v[kSide];
#pragma unroll
        for (int k = 0; k < kSide; k++)
            v[k] = in && k < left ? __ldg(q + (int64_t)k * a.stride[s][h]) : 0.0f;
        if (s) __syncthreads();
#pragma unroll
        for (int k = 0; k < kSide; k++) t[k * word[h]] = s ? t[k * word[h]] + v[k] : v[k];
    }
    __syncthreads();
    if (at[2] + lo < a.d[2] && at[1] + hi < a.d[1]) {
        float *o = a.out + frame + ((int64_t)at[0] * a.d[1] + at[1] + hi) * a.d[2] + at[2] + lo;
        const int left = min(kSide, a.d[0] - at[0]);
        for (int k = 0; k < left; k++)
            o[(int64_t)k * a.d[1] * a.d[2]] = tile[k * kTileX + hi * kTileY + lo];
    }
}

}  // namespace
}  // namespace srf

using namespace srf;

extern "C" int srf_permute_sum(float *out, const int *dims, int64_t n_frames, int n_sources,
                               const float *const *sources, const int64_t *strides,
                               void *stream) {
    if (!dims || n_frames < 0 || n_sources < 1 || n_sources > kMaxSources || !sources || !strides)
        return SRF_ERR_INVALID_ARGUMENT;
    PermuteArgs a{};
    a.out = out;
    a.n_src = n_sources;
    int64_t blocks = 1;
    a.frame = 1;
    for (int k = 0; k < 3; k++) {
        if (dims[k] < 0) return SRF_ERR_INVALID_ARGUMENT;
        a.d[k] = dims[k];
        a.tiles[k] = (dims[k] + kSide - 1) / kSide;
        a.frame *= dims[k];
        if (a.frame > ((int64_t)1 << 31) - 1) return SRF_ERR_UNSUPPORTED;
        blocks *= a.tiles[k];  // at most 2^31: tiles <= dims
    }
    if (blocks == 0 || n_frames == 0) return SRF_OK;
    if (n_frames > INT32_MAX / blocks) return SRF_ERR_UNSUPPORTED;
    blocks *= n_frames;
    if (!out) return SRF_ERR_INVALID_ARGUMENT;
    for (int s = 0; s < n_sources; s++) {
        if (!sources[s] || sources[s] == out) return SRF_ERR_INVALID_ARGUMENT;
        a.src[s] = sources[s];
        // each source is a dense stack in some axis order: its strides are those of one
        a.fast[s] = -1;
        for (int k = 0; k < 3; k++) {
            a.stride[s][k] = strides[3 * s + k];
            // beyond the frame the sum below could pass it by overflowing
            if (a.stride[s][k] < 1 || a.stride[s][k] > a.frame) return SRF_ERR_INVALID_ARGUMENT;
            if (a.stride[s][k] == 1 && (a.fast[s] < 0 || a.d[k] > a.d[a.fast[s]])) a.fast[s] = k;
        }
        int64_t last = 0;
        for (int k = 0; k < 3; k++) last += (int64_t)(a.d[k] - 1) * a.stride[s][k];
        if (a.fast[s] < 0 || last >= a.frame) return SRF_ERR_INVALID_ARGUMENT;
    }
    permute_sum_kernel<<<(unsigned)blocks, kSide * kSide, 0, (cudaStream_t)stream>>>(a);
    count_launches(1);
    return check_launch();
}
