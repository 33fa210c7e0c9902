// gcf_spectrum.cu -- tile-spectrum stage (CGenAvgSpectrum / GCalcSpectrum)
// and the Fourier-crop rescale (CRescaleImage / GFtResize2D).
//
// Two implementations of the averaged amplitude spectrum:
//   * the batched-cuFFT variant here: one pass extracts every tile with its
//     mean removed and the GRoundEdge taper applied, one cuFFT R2C batch,
//     one pass accumulates |F| with the DC moved to (0, tile/2);
//   * the fused hand-written tile-FFT kernel in gcf_fused.cu.
#include <cuda_runtime.h>

#include "gcf_internal.h"

namespace gcf {

namespace {

// mExtractPadTile + GCalcMoment2D + GNormalize2D + GRoundEdge
// (FindCTF/CGenAvgSpectrum.cpp:105-139): tile with its mean removed and
// the taper applied, dense tile x tile, in two passes.
//
// Bound: HBM (the image through L2, the dense tiles written once).  One CTA
// per tile left 99 of 148 SMs idle at 49 tiles and walked each tile twice
// with one load in flight: 3608 us for the 49 tiles of 1024 of a 4096 x 4096
// frame.  Slices of rows over the whole chip, one warp per row: under 80 us for
// both passes (the whole call 4445 -> 913 us).
//
// FP64 sums of the kMeanSlices row slices of each tile.
__global__ void __launch_bounds__(256) k_tile_sums(const float* __restrict__ img, int pitch, int tile, int ntx,
                                                   int offx, int offy, int stride, int first_tile,
                                                   double* __restrict__ sums)
{
    __shared__ double sh[8];
    const int t = first_tile + blockIdx.y;
    const int tx = t % ntx, ty = t / ntx;
    const float* src = img + (size_t)(offy + ty * stride) * pitch + offx + tx * stride;
    const int rows = (tile + kMeanSlices - 1) / kMeanSlices;
    const int y0 = blockIdx.x * rows, y1 = min(tile, y0 + rows);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s = 0.0;
    for (int y = y0 + warp; y < y1; y += 8) {
        const float* row = src + (size_t)y * pitch;
#pragma unroll 8
        for (int x = lane; x < tile; x += 32) s += (double)__ldg(row + x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sh[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += sh[w];
        sums[(size_t)blockIdx.y * kMeanSlices + blockIdx.x] = v;
    }
}

__global__ void __launch_bounds__(256) k_extract_tiles(const float* __restrict__ img, int pitch, int tile, int ntx,
                                                       int offx, int offy, int stride, int first_tile,
                                                       const float* __restrict__ taper,
                                                       const double* __restrict__ sums, float* __restrict__ out)
{
    const int t = first_tile + blockIdx.y;
    const int tx = t % ntx, ty = t / ntx;
    const int lane = threadIdx.x & 31, y = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (y >= tile) return;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kMeanSlices; ++k) s += __ldg(sums + (size_t)blockIdx.y * kMeanSlices + k);
    const float m = (float)(s / (double)(tile * tile));
    const float* src = img + (size_t)(offy + ty * stride + y) * pitch + offx + tx * stride;
    const float* tap = taper + (size_t)y * tile;
    float* dst = out + ((size_t)blockIdx.y * tile + y) * tile;
#pragma unroll 8
    for (int x = lane; x < tile; x += 32) dst[x] = (__ldg(src + x) - m) * __ldg(tap + x);
}

// GCalcSpectrum::mGCalculate + GAddImages (FindCTF/GCalcSpectrum.cu:15-31,
// Util/GAddImages.cu:10-23): accumulate |F| of `ntiles` R2C outputs into a
// double buffer with the DC moved to row tile/2.
__global__ void k_amp_accumulate(const float2* __restrict__ cmp, int tile, int ntiles,
                                 double* __restrict__ acc)
{
    int cx = tile / 2 + 1;
    int n = cx * tile;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int yd = i / cx, kx = i - yd * cx;
    int ky = yd + tile / 2;
    if (ky >= tile) ky -= tile;
    const float2* p = cmp + (size_t)ky * cx + kx;
    double s = 0.0;
    // eight loads in flight (the additions keep their order)
#pragma unroll 8
    for (int b = 0; b < ntiles; ++b) {
        float2 v = p[(size_t)b * n];
        s += (double)sqrtf(v.x * v.x + v.y * v.y);
    }
    acc[i] += s;
}

__global__ void k_finalize_raw(const double* __restrict__ acc, int n, double inv, float* raw)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) raw[i] = (float)(acc[i] * inv);
}

// GFtResize2D::mGTruncate without summation (Util/GFtResize2D.cu:7-32).
// One output row per blockIdx.y (its source row computed once), columns
// over the threads of blockIdx.x.
__global__ void k_fourier_crop(const float2* __restrict__ in, int cx_in, int cy_in,
                               float2* __restrict__ out, int cx_out, int cy_out)
{
    const int y = blockIdx.y, x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= cx_out) return;
    const int ys = (y > cy_out / 2) ? y - cy_out + cy_in : y;
    out[(size_t)y * cx_out + x] = __ldg(in + (size_t)ys * cx_in + x);
}

}  // namespace

void launch_extract_tiles(const float* img, int pitch, int tile, int ntx, int offx, int offy, int stride,
                          int first_tile, int ntiles, const float* taper, double* sums, float* out,
                          cudaStream_t st)
{
    if (ntiles <= 0) return;
    k_tile_sums<<<dim3(kMeanSlices, ntiles), 256, 0, st>>>(img, pitch, tile, ntx, offx, offy, stride, first_tile,
                                                           sums);
    k_extract_tiles<<<dim3((tile + 7) / 8, ntiles), 256, 0, st>>>(img, pitch, tile, ntx, offx, offy, stride,
                                                                  first_tile, taper, sums, out);
}

void launch_amp_accumulate(const float2* cmp, int tile, int ntiles, double* acc, cudaStream_t st)
{
    int n = (tile / 2 + 1) * tile;
    k_amp_accumulate<<<(n + 255) / 256, 256, 0, st>>>(cmp, tile, ntiles, acc);
}

void launch_finalize_raw(const double* acc, int n, double inv, float* raw, cudaStream_t st)
{
    k_finalize_raw<<<(n + 255) / 256, 256, 0, st>>>(acc, n, inv, raw);
}

void launch_fourier_crop(const float2* in, int cx_in, int cy_in, float2* out, int cx_out,
                         int cy_out, cudaStream_t st)
{
    const dim3 grid((cx_out + 255) / 256, cy_out);
    k_fourier_crop<<<grid, 256, 0, st>>>(in, cx_in, cy_in, out, cx_out, cy_out);
}

}  // namespace gcf
