// gcf_post.cu -- spectrum post-processing on the averaged half spectrum:
// background removal (GRmBackground2D), moments and B-factor lowpass
// (CFindCtfBase::mRemoveBackground/mLowpass), radial average (GRadialAvg),
// gathering of the in-band pixels for the candidate kernels, the diagnostic
// full spectrum (CSpectrumImage, GCalcCTF2D::EmbedCtf) and the spectral-CC
// resolution (GSpectralCC2D).
//
// Compiled with -fmad=false: the float expressions that decide masks and
// bands are rounded operation by operation, like the oracle.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "gcf_internal.h"

namespace gcf {

namespace {

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* sh /* 32*NV */)
{
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        v[k] = warp_sum(v[k]);
        if (lane == 0) sh[k * 32 + warp] = v[k];
    }
    __syncthreads();
    int nw = (blockDim.x + 31) >> 5;
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double t = lane < nw ? sh[k * 32 + lane] : 0.0;
            t = warp_sum(t);
            if (lane == 0) sh[k * 32] = t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = sh[k * 32];
    __syncthreads();
}

// Background removal and the moments of its result (GRmBackground2D::mGRemove,
// FindCTF/GRmBackground2D.cu:18-69): the box mean of sqrt(raw) (raw if
// log_spect), squared again (log_spect: not), subtracted from raw outside the
// DC mask (fR < 0.04).  The box is separable, its sums FP64.
//
// A block makes seg rows x strip columns of one spectrum: the values of its
// rows and columns with the box's halo (rows modulo tile, columns folded at
// the Hermitian edge, GRmBackground2D.cu:42-64) go to shared memory, threads
// slide the vertical box down the columns, then the horizontal one along the
// rows (one lane per row, odd pitches: no bank conflicts), and the block
// writes its rows.  The block's shape depends on the number of spectra, its
// sums do not: float32 values (24 bits) summed over up to 137 x 137 (2^14.2) of
// them are exact in FP64 (53 bits) in any order while the largest value in reach
// is below 2^14 times the smallest but zero (2^18 for the 35 x 35 of tile 512;
// twice the exponent in the spectrum itself, whose square roots these are).  All intermediate sums stay in shared memory; the last
// block of a spectrum adds the blocks' moments in block order.
//
// Bound: latency for few spectra; for many conversions to FP64 and shared-memory
// reads (about 6 of each per output and direction) and the halo's square roots.
// Two kernels with the horizontal sums in global memory and a third, one block
// per spectrum, for the moments took 34.0 us for one spectrum of 512 x 257; this
// kernel takes 12.7 us; 256 spectra 517 us, now 458.  One spectrum of tile 1024:
// 62.6 -> 29.2 us, of tile 2048: 193 -> 166 us.
constexpr int kBgThreads = 640;   // at most, two blocks per SM; a whole number of column groups

__global__ void __maxnreg__(48)   // two blocks of 640 threads per SM
k_background(const float* __restrict__ raw, int tile, int log_spect, int box, int seg, int strip,
             float* __restrict__ ctf, double* __restrict__ part, unsigned* __restrict__ ticket,
             double* __restrict__ mom)
{
    extern __shared__ double s_bg[];
    __shared__ double s_red[64];
    const int cx = tile / 2 + 1, half_x = cx - 1, hb = box / 2, m = blockIdx.y;
    const int strips = (cx + strip - 1) / strip;
    const int x0 = (int)(blockIdx.x % strips) * strip, w = min(strip, cx - x0), e = w + 2 * hb;
    const int y0 = (int)(blockIdx.x / strips) * seg, h = min(seg, tile - y0), rows = h + 2 * hb;
    const int pe = (strip + 2 * hb) | 1, ps = strip | 1;
    double* V = s_bg;                                        // [seg][pe] vertical sums
    float* A = reinterpret_cast<float*>(s_bg + seg * pe);    // [seg + 2 hb][pe] values
    double* S = s_bg + seg * pe;                             // [seg][ps] box sums, over A
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NW = blockDim.x >> 5;
    const size_t base = (size_t)m * cx * tile;
    const float* src = raw + base;
    // a thread keeps one column: its fold is decided once
    const int ew = (strip + 2 * hb + 31) & ~31, G = blockDim.x / ew, g = tid / ew, c0 = tid - g * ew;
    if (c0 < e && g < G) {
        int u = x0 - hb + c0;
        if (u >= half_x) u -= 2 * half_x;
        const bool fold = u < 0;
        const float* col = src + (fold ? -u : u);
        float* a = A + c0;
#pragma unroll 4
        for (int r = g; r < rows; r += G) {
            int R = y0 - hb + r;
            if (R < 0) R += tile;
            else if (R >= tile) R -= tile;
            if (fold && R) R = tile - R;   // half_y - (R - half_y) modulo tile
            const float v = __ldg(col + (size_t)R * cx);
            a[r * pe] = log_spect ? v : sqrtf(v);
        }
    }
    __syncthreads();
    if (c0 < e && g < G) {   // G runs of rows per column
        const int c = c0, ya = h * g / G, yb = h * (g + 1) / G;
        double sum = 0.0;
#pragma unroll 4
        for (int k = 0; k <= 2 * hb; ++k) sum += (double)A[(ya + k) * pe + c];
        if (ya < yb) V[ya * pe + c] = sum;
#pragma unroll 4
        for (int y = ya + 1; y < yb; ++y) {
            sum += (double)A[(y + 2 * hb) * pe + c] - (double)A[(y - 1) * pe + c];
            V[y * pe + c] = sum;
        }
    }
    __syncthreads();
    {
        // a warp takes 32 rows and a run of columns
        const int RB = (seg + 31) / 32, CG = max(NW / RB, 1);
        const int xa = w * (warp / RB) / CG, xb = w * (warp / RB + 1) / CG;
        for (int y = 32 * (warp % RB) + lane; y < h && xa < xb && warp / RB < CG; y += 32 * RB) {
            const double* v = V + y * pe;
            double sum = 0.0;
#pragma unroll 4
            for (int k = 0; k <= 2 * hb; ++k) sum += v[xa + k];
            S[y * ps + xa] = sum;
#pragma unroll 4
            for (int x = xa + 1; x < xb; ++x) {
                sum += v[x + 2 * hb] - v[x - 1];
                S[y * ps + x] = sum;
            }
        }
    }
    __syncthreads();
    const double norm = (double)box * (double)box, inv = 1.0 / norm;
    double mv[2] = {0.0, 0.0};
    for (int r = warp; r < h; r += NW) {
        const int y = y0 + r, yr = y - tile / 2;
#pragma unroll 4
        for (int c = lane; c < w; c += 32) {
            const int x = x0 + c;
            const size_t i = base + (size_t)y * cx + x;
            bool masked = false;
            if (12 * x < cx) {   // beyond, x * 0.5 / (cx - 1) alone is above 0.04
                float fr = x * 0.5f / (cx - 1);
                fr = sqrtf(fr * fr + yr * yr / (float)(tile * tile));
                masked = (double)fr < 0.04;
            }
            // sum / norm: the reciprocal's product with its residual added back
            // (Markstein); a division of its own costs 90 us at 256 spectra
            const double sum = S[r * ps + c];
            double b = sum * inv;
            b = __fma_rn(__fma_rn(-b, norm, sum), inv, b);
            if (!log_spect) b *= b;
            const float v = masked ? 0.0f : (float)((double)__ldg(raw + i) - b);
            ctf[i] = v;
            mv[0] += (double)v;
            mv[1] += (double)v * (double)v;
        }
    }
    block_sum<2>(mv, s_red);
    if (warp != 0) return;
    const int nb = gridDim.x;
    double* p = part + 2 * (size_t)m * nb;
    int last = 0;
    if (lane == 0) {
        p[2 * blockIdx.x] = mv[0];
        p[2 * blockIdx.x + 1] = mv[1];
        __threadfence();
        last = atomicInc(ticket + m, nb - 1) == (unsigned)(nb - 1);   // wraps to zero for the next launch
        __threadfence();
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    mv[0] = mv[1] = 0.0;
    for (int k = lane; k < nb; k += 32) {
        mv[0] += __ldcg(p + 2 * k);
        mv[1] += __ldcg(p + 2 * k + 1);
    }
    mv[0] = warp_sum(mv[0]);
    mv[1] = warp_sum(mv[1]);
    if (lane == 0) {
        const int n = cx * tile;
        mom[2 * m] = mv[0] / n;
        mom[2 * m + 1] = mv[1] / n;
    }
}

// Mean and second moment of each half spectrum (Util/GCalcMoment2D.cu:10-58).
// One block per spectrum; each thread keeps eight loads in flight.
__global__ void __launch_bounds__(1024) k_moments(const float* __restrict__ spect, int n,
                                                  double* __restrict__ out2)
{
    __shared__ double sh[64];
    int m = blockIdx.x;
    const float* p = spect + (size_t)m * n;
    const int S = blockDim.x;
    double v[2] = {0.0, 0.0};
    int i = threadIdx.x;
    for (; i + 7 * S < n; i += 8 * S) {
        double a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = p[i + k * S];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            v[0] += a[k];
            v[1] += a[k] * a[k];
        }
    }
    for (; i < n; i += S) {
        double a = p[i];
        v[0] += a;
        v[1] += a * a;
    }
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
        out2[2 * m] = v[0] / n;
        out2[2 * m + 1] = v[1] / n;
    }
}

// Full spectrum value (DC at column tile/2) from the half spectrum
// (FindCTF/GCalcSpectrum.cu:47-69; mirror row modulo tile).
__device__ __forceinline__ float full_val(const float* half, int tile, int y, int X)
{
    int cx = tile / 2 + 1, hx = cx - 1;
    int xd = X - hx;
    if (xd >= 0) return half[(size_t)y * cx + xd];
    int ys = tile - y;
    if (ys >= tile) ys -= tile;
    return half[(size_t)ys * cx - xd];
}

// CFindCtfBase::mLowpass (FindCTF/CFindCtfBase.cpp:191-219) around a batched
// R2C / C2R pair: the full spectrum (DC at column tile/2), the B-factor
// filter exp(-B (kx^2 + ky^2) / (2 tile^2)) of GLowpass2D::DoBFactor
// (FindCTF/GLowpass2D.cu:9-23) with the 1/tile^2 of the normalised forward
// transform, and the copy of columns tile/2 .. tile back into the half
// spectrum (the last one from the periodic neighbour, column 0).
__global__ void k_lp_full(const float* __restrict__ ctf0, int tile, float* __restrict__ full)
{
    int m = blockIdx.y;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tile * tile) return;
    int y = i / tile, X = i - y * tile;
    int cx = tile / 2 + 1;
    full[(size_t)m * tile * tile + i] = full_val(ctf0 + (size_t)m * cx * tile, tile, y, X);
}

// The filter depends on the tile size and B-factor only: one table per
// context, shared by every micrograph (the same double expression per bin).
__global__ void k_lp_table(double* __restrict__ g, int tile, double bfactor)
{
    int cx = tile / 2 + 1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cx * tile) return;
    int y = i / cx, x = i - y * cx;
    int ky = (y > tile / 2) ? y - tile : y;
    double scale = -bfactor / ((double)tile * tile + (double)tile * tile);
    g[i] = exp(scale * ((double)x * x + (double)ky * ky)) / ((double)tile * tile);
}

__global__ void k_lp_filter(float2* __restrict__ cmp, int tile, const double* __restrict__ gtab)
{
    int m = blockIdx.y;
    int cx = tile / 2 + 1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cx * tile) return;
    double g = gtab[i];
    float2 v = cmp[(size_t)m * cx * tile + i];
    cmp[(size_t)m * cx * tile + i] = make_float2((float)(v.x * g), (float)(v.y * g));
}

// Variance gate of mRemoveBackground (FindCTF/CFindCtfBase.cpp:169-174):
// micrographs whose background-removed spectrum has variance < 1 keep it
// unfiltered.
__global__ void k_lp_extract(const float* __restrict__ ctf0, const float* __restrict__ full, int tile,
                             const double* __restrict__ mom, float* __restrict__ out,
                             int* __restrict__ lowpassed)
{
    int m = blockIdx.y;
    int cx = tile / 2 + 1, hx = cx - 1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double mean = mom[2 * m], var = mom[2 * m + 1] - mean * mean;
    bool run = !(var < 1.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) lowpassed[m] = run ? 1 : 0;
    if (i >= cx * tile) return;
    size_t base = (size_t)m * cx * tile;
    if (!run) {
        out[base + i] = ctf0[base + i];
        return;
    }
    int y = i / cx, x = i - y * cx;
    int X = x + hx;
    if (X >= tile) X -= tile;
    out[base + i] = full[(size_t)m * tile * tile + (size_t)y * tile + X];
}

// GRadialAvg (FindCTF/GRadialAvg.cu:11-33) with the nearest-pixel sample
// table precomputed on the host.
// One warp per radius: the lanes stride over the ring's samples.
__global__ void k_radial(const float* __restrict__ spect, int cmp_n, int cx,
                         const int* __restrict__ off, const int* __restrict__ pix,
                         float* __restrict__ radial)
{
    int m = blockIdx.y;
    int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= cx) return;
    const float* p = spect + (size_t)m * cmp_n;
    double s = 0.0;
    int a = off[r], b = off[r + 1];
    for (int k = a + lane; k < b; k += 32) s += p[pix[k]];
    s = warp_sum(s);
    if (lane == 0) radial[(size_t)m * cx + r] = (float)(s / (b - a));
}

// Spectrum of each job gathered in band order, and its sum of squares.
__global__ void k_band_gather(const float* __restrict__ ctf, int cmp_n,
                              const SearchJob* __restrict__ jobs, const BandDev* __restrict__ bands,
                              const int2* __restrict__ spec_off, float* __restrict__ band_spec,
                              double* __restrict__ sum_ss)
{
    __shared__ double sh[32];
    int j = blockIdx.x;
    const SearchJob& jb = jobs[j];
    const BandDev& b = bands[jb.band];
    const float* src = ctf + (size_t)jb.mic * cmp_n;
    float* dst = band_spec + spec_off[j].x;
    double v[1] = {0.0};
    const int S = blockDim.x;
    int k = threadIdx.x;
    for (; k + 3 * S < b.n; k += 4 * S) {   // four gathers in flight per thread
        int q[4];
        float s[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = b.idx[k + u * S];
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] = src[q[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            dst[k + u * S] = s[u];
            v[0] += (double)s[u] * (double)s[u];
        }
    }
    for (; k < b.n; k += S) {
        float s = src[b.idx[k]];
        dst[k] = s;
        v[0] += (double)s * (double)s;
    }
    block_sum<1>(v, sh);
    if (threadIdx.x == 0) sum_ss[j] = v[0];
}

// Signed CTF of GCalcCTF2D (FindCTF/GCalcCTF2D.cu:15-38), double, from a
// pixel's s^2 and polar angle.
__device__ double ctf_geo(double s2, double th, const PixOptics& o, double add, double mean, double sigma,
                          double az)
{
    double df = mean + sigma * cos(2.0 * (th - az));
    double chi = add + M_PI * (double)o.wl * s2 * (df - 0.5 * s2 * (double)o.wl * o.wl * o.cs);
    return -sin(chi);
}

// The same at one pixel (x, y) of the half spectrum.
__device__ double ctf_at(int x, int y, int cx, int cy, const PixOptics& o, double add,
                         double mean, double sigma, double az)
{
    double fx = x * 0.5 / (cx - 1);
    double fy = (double)(y - cy / 2) / cy;
    double s2 = fx * fx + fy * fy;
    double th = atan(fy / (fx + 1e-30));
    return ctf_geo(s2, th, o, add, mean, sigma, az);
}

// CSpectrumImage::mGenFullSpectrum + mEmbedCTF (FindCTF/CSpectrumImage.cpp:36-71,
// FindCTF/GCalcCTF2D.cu:49-78).
__global__ void k_full_spectrum(const float* __restrict__ ctf, int tile, const int* __restrict__ mic_of,
                                const gcf_result* __restrict__ res, const PixOptics* __restrict__ op,
                                const double* __restrict__ mom, float* __restrict__ full)
{
    int k = blockIdx.y;
    int m = mic_of[k];
    int cx = tile / 2 + 1, cy = tile, hx = cx - 1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tile * tile) return;
    int y = i / tile, X = i - y * tile;
    const float* half = ctf + (size_t)m * cx * cy;
    float v = full_val(half, tile, y, X);
    const PixOptics o = op[k];
    const gcf_result r = res[k];
    // CFindCtfBase::Setup1 resolution range (FindCTF/CFindCtfBase.cpp:64-68)
    float r0 = 25.0f * o.px, r1 = (2.0f * o.px) / 0.8f;
    if (r1 < 3.5f) r1 = 3.5f;
    float fmn = o.px / r0, fmx = o.px / r1;
    if (X < hx) {
        float fy = (y - cy * 0.5f) / cy;
        float fx = (X - (float)hx) * 0.5f / hx;
        float rr = sqrtf(fx * fx + fy * fy);
        if (!(rr < fmn || rr > fmx)) {
            double mean = mom[2 * m], var = mom[2 * m + 1] - mean * mean;
            double sd = var < 0 ? 0.0 : sqrt(var);
            // CFindCtfBase::GenFullSpectrum (FindCTF/CFindCtfBase.cpp:118-126)
            float az = r.azimuth * 0.017453f;
            float dmin = r.df_min / o.px, dmax = r.df_max / o.px;
            float ph = fmodf(r.ext_phase * 0.01745329f, 3.14159265358979f);
            float mn = 0.5f * (dmin + dmax), sg = 0.5f * (dmax - dmin);
            int ix = hx - X, iy = (cy - y) % cy;
            double c = fabs(ctf_at(ix, iy, cx, cy, o, (double)(o.amp_phase + ph), mn, sg, az));
            v = (float)((c - 0.5) * (sd * 1.5) + mean);
        }
    }
    full[(size_t)k * tile * tile + i] = v;
}

// GSpectralCC2D::mGCalc2D (FindCTF/GSpectralCC2D.cu:12-110) in two steps:
// sums over the integer-radius rings (one CTF evaluation per pixel), then
// the Pearson CC of each width-10 shell from its rings.
__global__ void k_ring_sums(const float* __restrict__ ctf, int tile, const SearchJob* __restrict__ jobs,
                            const int* __restrict__ ring_off, const int* __restrict__ ring_pix,
                            const double2* __restrict__ ring_geo, double* __restrict__ ring_sums)
{
    __shared__ double sh[5 * 32];
    int ring = blockIdx.x, j = blockIdx.y;
    const SearchJob jb = jobs[j];
    int cx = tile / 2 + 1, cy = tile;
    const PixOptics o = jb.o;
    float dmin = jb.df_mean * (1.0f - jb.ast_ratio) / o.px;
    float dmax = jb.df_mean * (1.0f + jb.ast_ratio) / o.px;
    float mn = 0.5f * (dmin + dmax), sg = 0.5f * (dmax - dmin);
    double add = (double)(o.amp_phase + jb.ext_phase * 0.01745329f);
    double az = (double)(jb.ast_angle * 0.01745329f);
    const float* sp = ctf + (size_t)jb.mic * cx * cy;
    double v[5] = {0, 0, 0, 0, 0};
    for (int k = ring_off[ring] + threadIdx.x; k < ring_off[ring + 1]; k += blockDim.x) {
        int pix = ring_pix[k];
        const double2 g = ring_geo[k];   // (s^2, polar angle) of the pixel
        double c = ctf_geo(g.x, g.y, o, add, mn, sg, az);
        double s = sp[pix];
        v[0] += c * s;
        v[1] += c;
        v[2] += s;
        v[3] += c * c;
        v[4] += s * s;
    }
    block_sum<5>(v, sh);
    if (threadIdx.x == 0) {
        double* out = ring_sums + ((size_t)j * cx + ring) * 6;
        for (int q = 0; q < 5; ++q) out[q] = v[q];
        out[5] = (double)(ring_off[ring + 1] - ring_off[ring]);
    }
}

__global__ void k_shell_cc(int tile, const double* __restrict__ ring_sums, float* __restrict__ cc_out)
{
    int j = blockIdx.x;
    int cx = tile / 2 + 1;
    const int width = 10;
    for (int b = threadIdx.x; b < cx; b += blockDim.x) {
        int lo = b - width / 2, hi = lo + width;
        if (lo < 0) {
            lo = 0;
            hi = width;
        } else if (hi > cx) {
            lo = cx - width;
            hi = cx;
        }
        double v[6] = {0, 0, 0, 0, 0, 0};
        for (int ring = lo; ring < hi; ++ring)
            for (int q = 0; q < 6; ++q) v[q] += ring_sums[((size_t)j * cx + ring) * 6 + q];
        float out = 0.0f;
        if (v[5] > 0) {
            double n = v[5];
            double cs = v[0] / n, mc = v[1] / n, ms = v[2] / n, sc = v[3] / n, ss = v[4] / n;
            sc -= mc * mc;
            ss -= ms * ms;
            if (sc > 0 && ss > 0) out = (float)((cs - mc * ms) / sqrt(sc * ss));
        }
        cc_out[(size_t)j * cx + b] = out;
    }
}

}  // namespace

namespace {

// Shared memory of a background block at two blocks, or one, per SM.
constexpr size_t kTwoPerSM = 110 * 1024, kOnePerSM = 200 * 1024;

// Rows and columns of a background block.
struct BgShape {
    int box, seg, strip;
    size_t smem;
    int blocks(int tile) const { return ((tile / 2 + strip) / strip) * ((tile + seg - 1) / seg); }
};

BgShape bg_shape(int tile, int nmic)
{
    // box of GRmBackground2D::mGRemove (FindCTF/GRmBackground2D.cu:33-36), fMinFreq = 1/15
    const float fmin = 1.0f / 15.0f;
    int box = (int)(fmin * tile);
    if (box > (0.3f * tile)) box = (int)(0.3f * tile);
    box = box / 2 * 2 + 1;
    if (box < 7) box = 7;
    BgShape b{box, 8, 0, 0};
    const int cx = tile / 2 + 1, hb = box / 2;
    // strips of at most 160 columns, narrower until a block's shared memory fits
    auto fit = [&](int seg, size_t limit) {
        b.seg = seg;
        for (int n = (cx + 159) / 160;; ++n) {
            b.strip = (cx + n - 1) / n;
            const size_t pe = (size_t)(b.strip + 2 * hb) | 1, ps = (size_t)b.strip | 1;
            b.smem = (size_t)seg * pe * 8 + std::max((size_t)(seg + 2 * hb) * pe * 4, (size_t)seg * ps * 8);
            if (b.smem <= limit || b.strip <= 8) break;
        }
    };
    // 8 rows while the chip takes all blocks at once (two per SM), then 32, then
    // 64, which load less halo per output: 512 x 257 spectra, 17.8 (8 rows) and
    // 23.8 us (32) for one, 21.1 and 24.5 for two, 32.9 and 24.7 (64 rows: 27.1)
    // for four, 43.5 and 31.8 us (32 and 64) for 12, 566 and 473 us for 256,
    // launch included.  Tiles whose box is wide leave 64 rows too narrow a strip,
    // and from 2048 on 32 rows as well unless a block has an SM to itself.
    auto one_wave = [&] { return (long long)b.blocks(tile) * nmic <= 2 * 148; };
    fit(8, kTwoPerSM);
    if (!one_wave()) fit(32, kTwoPerSM);
    if (b.strip < 48 && b.strip < cx) fit(32, kOnePerSM);
    if (!one_wave()) {
        const BgShape rows32 = b;
        fit(64, kTwoPerSM);
        if (b.strip < 64 && b.strip < cx) b = rows32;
    }
    return b;
}

}  // namespace

size_t background_blocks(int tile) { return bg_shape(tile, 1).blocks(tile); }

cudaError_t launch_background(const float* raw, int tile, int nmic, int log_spect, float* ctf, double* part,
                              unsigned* ticket, double* mom, cudaStream_t st)
{
    const BgShape b = bg_shape(tile, nmic);
    const int ew = (b.strip + 2 * (b.box / 2) + 31) & ~31;
    const int threads = ew * std::max(1, (b.smem > kTwoPerSM ? 1024 : kBgThreads) / ew);
    // the same limit on every call: the attribute is the process's, and another
    // thread's context may have a tile that needs less
    if (b.smem > kOnePerSM) return cudaErrorInvalidConfiguration;
    cudaError_t e = cudaFuncSetAttribute(k_background, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOnePerSM);
    if (e != cudaSuccess) return e;
    k_background<<<dim3(b.blocks(tile), nmic), threads, b.smem, st>>>(raw, tile, log_spect, b.box, b.seg, b.strip,
                                                                         ctf, part, ticket, mom);
    return cudaGetLastError();
}

void launch_moments(const float* spect, int n, int nmic, double* out2, cudaStream_t st)
{
    k_moments<<<nmic, 1024, 0, st>>>(spect, n, out2);
}

void launch_lp_full(const float* ctf0, int tile, int nmic, float* full, cudaStream_t st)
{
    dim3 grid((tile * tile + 255) / 256, nmic);
    k_lp_full<<<grid, 256, 0, st>>>(ctf0, tile, full);
}

void launch_lp_table(double* g, int tile, double bfactor, cudaStream_t st)
{
    int n = (tile / 2 + 1) * tile;
    k_lp_table<<<(n + 255) / 256, 256, 0, st>>>(g, tile, bfactor);
}

void launch_lp_filter(float2* cmp, int tile, int nmic, const double* g, cudaStream_t st)
{
    int n = (tile / 2 + 1) * tile;
    dim3 grid((n + 255) / 256, nmic);
    k_lp_filter<<<grid, 256, 0, st>>>(cmp, tile, g);
}

void launch_lp_extract(const float* ctf0, const float* full, int tile, int nmic, const double* moments,
                       float* out, int* lowpassed, cudaStream_t st)
{
    int n = (tile / 2 + 1) * tile;
    dim3 grid((n + 255) / 256, nmic);
    k_lp_extract<<<grid, 256, 0, st>>>(ctf0, full, tile, moments, out, lowpassed);
}

void launch_radial(const float* spect, int tile, int nmic, const int* off, const int* pix,
                   float* radial, cudaStream_t st)
{
    int cx = tile / 2 + 1;
    dim3 grid((cx + 7) / 8, nmic);
    k_radial<<<grid, 256, 0, st>>>(spect, cx * tile, cx, off, pix, radial);
}

void launch_band_gather(const float* ctf, int cmp_n, const SearchJob* jobs, const BandDev* bands,
                        const int2* spec_off, int njobs, float* band_spec, double* sum_ss,
                        cudaStream_t st)
{
    if (njobs <= 0) return;
    k_band_gather<<<njobs, 1024, 0, st>>>(ctf, cmp_n, jobs, bands, spec_off, band_spec, sum_ss);
}

void launch_full_spectrum(const float* ctf, int tile, int nmic, const int* mic_of,
                          const gcf_result* res, const PixOptics* o, const double* moments,
                          float res_lo_freq_dummy, float* full, cudaStream_t st)
{
    (void)res_lo_freq_dummy;
    if (nmic <= 0) return;
    dim3 grid((tile * tile + 255) / 256, nmic);
    k_full_spectrum<<<grid, 256, 0, st>>>(ctf, tile, mic_of, res, o, moments, full);
}

void launch_ctf_res(const float* ctf, int tile, const SearchJob* jobs, int njobs, const int* ring_off,
                    const int* ring_pix, const double2* ring_geo, double* ring_sums, float* cc,
                    cudaStream_t st)
{
    if (njobs <= 0) return;
    dim3 grid(tile / 2 + 1, njobs);
    k_ring_sums<<<grid, 128, 0, st>>>(ctf, tile, jobs, ring_off, ring_pix, ring_geo, ring_sums);
    k_shell_cc<<<njobs, 128, 0, st>>>(tile, ring_sums, cc);
}

}  // namespace gcf
