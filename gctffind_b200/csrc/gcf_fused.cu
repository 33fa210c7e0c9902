// gcf_fused.cu -- fused tile-spectrum kernel for 512 x 512 tiles
// (CGenAvgSpectrum::DoIt + GCalcMoment2D + GNormalize2D + GRoundEdge +
//  GCalcSpectrum::DoPad + GAddImages, FindCTF/CGenAvgSpectrum.cpp:77-139).
//
// A thread-block cluster of CL CTAs (16, or 8 where 16-CTA clusters do not
// fit) owns one tile at a time; the tile never leaves the chip:
//   mean    every tile mean comes from one pass of k_block_sums over the
//           images (a 512 tile is 2 x 2 blocks of 256 x 256);
//   rows    each warp reads two tile rows straight from global memory,
//           forms (x - mean) * taper as the real and imaginary parts of one
//           512-point complex FFT held in registers (16 values per lane,
//           radix-16 x radix-32 with one shared-memory transpose), splits
//           the result into the two rows' 257-bin half spectra and pushes
//           each bin into the shared memory of the CTA that owns its
//           frequency column (16-byte DSMEM stores, [column][row]);
//   columns each warp transforms one frequency column (512 rows) read from
//           its own CTA's shared memory; the real kx = 0 and kx = 256
//           columns share one complex FFT;
//   |F|     amplitudes (DC moved to row 256) accumulate in registers across
//           all tiles of a work item and are written once.
// That is the one-line kernel, k_fused_spectrum, whose shapes the autotuner
// times and a caller can ask for; the default is k_fused_spectrum_pair, the
// same work on 8-CTA clusters with two lines per warp, the taper and the sums
// in tensor memory and the rows' bins exchanged by bulk copies.
// With CL = 16 the column buffer is double-buffered, so one cluster barrier
// per tile separates writers from readers.  Beside the cluster launch,
// k_fused_spectrum_solo runs one CTA on each SM that the clusters leave free
// (8-CTA clusters fit twice per GPC) and takes items from the back of the
// same queue.  Work items are (image, tile
// range) pairs, handed out in order through a counter; their partial
// spectra are summed in item order by k_item_reduce, so the result does not
// depend on which cluster took which item.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "gcf_internal.h"

namespace cg = cooperative_groups;

namespace gcf {

namespace {

constexpr int FT = 512;          // tile edge

// exp(-2 pi i k / 32), k < 16, rounded to float from double like the host
// twiddle tables; written once per device before the first launch.
__constant__ float2 c_tw32[16];
constexpr int FCX = FT / 2 + 1;  // 257 half-spectrum columns
constexpr int FSCR = 16 * 34;    // per-warp scratch, float2 units
constexpr int FROW = 34;         // transpose row stride: 64-bit accesses of either side hit distinct banks

// Complex product, scalar.  The per-lane twiddles (read from shared
// memory) use it: a packed form with the twiddle stored pre-arranged
// (wx, wx, -wy, wy) measured slower, with twice the shared-memory reads.
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// Complex product by a compile-time or constant-bank twiddle w as two packed
// operations: a * w = (a.x, a.y) (wx, wx) + (a.y, a.x) (-wy, wy).  (The form
// with a's halves broadcast, (a.x, a.x) w + (a.y, a.y) (-wy, wx), measured
// slower.)
__device__ __forceinline__ float2 cmul_k(float2 a, float2 w)
{
    return __ffma2_rn(make_float2(a.y, a.x), make_float2(-w.y, w.y), __fmul2_rn(a, make_float2(w.x, w.x)));
}
// Complex additions as packed two-float operations (one f32x2 instruction
// each; exact IEEE round-to-nearest like the scalar pair): halves the issue
// slots of the butterflies.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

// Forward 4-point DFT in place (W4 = -i).
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3)
{
    float2 s02 = cadd(a0, a2), d02 = csub(a0, a2);
    float2 s13 = cadd(a1, a3), d13 = csub(a1, a3);
    a0 = cadd(s02, s13);
    a2 = csub(s02, s13);
    const float2 sw = make_float2(d13.y, d13.x);
    a1 = __ffma2_rn(sw, make_float2(1.0f, -1.0f), d02);   // d02 - i d13
    a3 = __ffma2_rn(sw, make_float2(-1.0f, 1.0f), d02);   // d02 + i d13
}

// exp(-2 pi i m / 16) for the compile-time products m = n2 * k1 <= 9
__device__ __forceinline__ float2 w16(int m)
{
    constexpr float C1 = 0.92387953251128674f, C2 = 0.70710678118654752f, C3 = 0.38268343236508977f;
    switch (m) {
    case 0: return make_float2(1.0f, 0.0f);
    case 1: return make_float2(C1, -C3);
    case 2: return make_float2(C2, -C2);
    case 3: return make_float2(C3, -C1);
    case 4: return make_float2(0.0f, -1.0f);
    case 6: return make_float2(-C2, -C2);
    default: return make_float2(-C1, C3);   // m = 9
    }
}

// Slot of spectrum bin K (0..511) in the warp scratch when a whole FFT
// output is staged: bins 256..511 are shifted by 8 slots, so the 16-lane
// halves of the (m + 16 k + 256 p) stores hit distinct banks.
__device__ __forceinline__ int sslot(int K) { return K + ((K >> 8) << 3); }

// |z| with the fast square root (relative error within 2^-22): the
// amplitudes only enter averages compared at 1e-4.
__device__ __forceinline__ float amp(float x, float y)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x * x + y * y));
    return r;
}

// Position of output k of dft16 in its register array.
__host__ __device__ constexpr int P16(int k) { return (k & 3) * 4 + (k >> 2); }

// Forward 16-point DFT in registers, natural-order input, output k in
// v[P16(k)] (radix-4 x radix-4: n = 4 n1 + n2, k = k1 + 4 k2).
__device__ __forceinline__ void dft16(float2 (&v)[16])
{
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
#pragma unroll
    for (int k1 = 1; k1 < 4; ++k1)
#pragma unroll
        for (int n2 = 1; n2 < 4; ++n2) {
            if (n2 * k1 == 4) v[4 * k1 + n2] = make_float2(v[4 * k1 + n2].y, -v[4 * k1 + n2].x);   // * (-i)
            else v[4 * k1 + n2] = cmul_k(v[4 * k1 + n2], w16(n2 * k1));
        }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4(v[4 * k1 + 0], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
}

// 512-point forward FFT held by one warp.  In: lane l holds x[32 j + l] in
// v[j].  Out: lane 2m+p holds X[m + 16 k + 256 p] in v[P16(k)].
// scr: FSCR float2 of warp-private shared memory; twl[k1 * 32 + l] =
// exp(-2 pi i l k1 / 512); the 32-point twiddles are c_tw32.
__device__ __forceinline__ void fft512_warp(float2 (&v)[16], float2* scr, const float2* twl, int lane)
{
    dft16(v);
#pragma unroll
    for (int k1 = 1; k1 < 16; ++k1) v[P16(k1)] = cmul(v[P16(k1)], twl[k1 * 32 + lane]);
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) scr[k1 * FROW + lane] = v[P16(k1)];
    __syncwarp();
    const int m = lane >> 1, p = lane & 1;
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = scr[m * FROW + 2 * q + p];
    dft16(v);
    // radix-2 across the lane pair: lane p = 1 multiplies its odd half by
    // the twiddle before the exchange, then lane 0 forms E0 + W E1 and
    // lane 1 forms E0 - W E1
    const float sg = p ? -1.0f : 1.0f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        float2 u = cmul_k(v[P16(k)], c_tw32[k]);
        if (!p) u = v[P16(k)];
        float2 o;
        o.x = __shfl_xor_sync(0xffffffffu, u.x, 1);
        o.y = __shfl_xor_sync(0xffffffffu, u.y, 1);
        v[P16(k)] = __ffma2_rn(make_float2(sg, sg), u, o);
    }
    __syncwarp();
}

// cmul and amp as the one-line kernels compile them (where the compiler
// contracts a product into the sum is its choice, so it is pinned here):
// the two kernels' spectra are the same bits.
__device__ __forceinline__ float2 cmul_pinned(float2 a, float2 b)
{
    return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}
__device__ __forceinline__ float amp_xy(float x, float y)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(__fmaf_rn(x, x, __fmul_rn(y, y))));
    return r;
}

// Two 512-point forward FFTs held by one warp, line h on the lanes of parity
// h: lane 2a + h holds x[32 j + 2a] of its line in e[j] and x[32 j + 2a + 1]
// in o[j] on entry, X[a + 16 k] in e[P16(k)] and X[a + 16 k + 256] in
// o[P16(k)] on return.  Every operation on a line is fft512_warp's (radix 16,
// twiddles, radix 16 over the even and odd l, radix 2), so the values are the
// same bits; what changes is where they live.  A lane holds whole 32-point
// second stages, so the radix 2 needs no lane exchange (32 shuffles and 32
// selects per line less), pairs of neighbours move as 16-byte accesses (half
// the shared-memory instructions), and two lines per warp give the scheduler
// twice the independent work.  scr: line h's 256 float4; row k1 keeps its
// 16-byte chunk c at c ^ k1 ^ 4 h, so that neither side of the transpose has
// bank conflicts without padding.  tw4[k1 * 16 + a] = (exp(-2 pi i 2a k1 / 512),
// exp(-2 pi i (2a + 1) k1 / 512)).  between(0..3) runs at four points of the
// transform: the caller spreads its global loads over them (32 loads of 256
// bytes in a row stall a warp for 1000 cycles in the load queue).
template <class F>
__device__ __forceinline__ void fft512_pair(float2 (&e)[16], float2 (&o)[16], float4* scr, const float4* tw4,
                                            int lane, F between)
{
    const int a = lane >> 1, ax = a ^ ((lane & 1) << 2);
    between(0);
    dft16(e);
    between(1);
    dft16(o);
    between(2);
#pragma unroll
    for (int k1 = 1; k1 < 16; ++k1) {
        const float4 t = tw4[k1 * 16 + a];
        e[P16(k1)] = cmul_pinned(e[P16(k1)], make_float2(t.x, t.y));
        o[P16(k1)] = cmul_pinned(o[P16(k1)], make_float2(t.z, t.w));
    }
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1)
        scr[k1 * 16 + (ax ^ k1)] = make_float4(e[P16(k1)].x, e[P16(k1)].y, o[P16(k1)].x, o[P16(k1)].y);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const float4 z = scr[a * 16 + (q ^ ax)];
        e[q] = make_float2(z.x, z.y);
        o[q] = make_float2(z.z, z.w);
    }
    between(3);
    dft16(e);
    dft16(o);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 u = cmul_k(o[P16(k)], c_tw32[k]), E = e[P16(k)];
        e[P16(k)] = cadd(E, u);
        o[P16(k)] = csub(E, u);
    }
}

// Two adjacent samples of a row; v2: the row is 8-byte aligned at even x.
__device__ __forceinline__ float2 row2(const float* p, bool v2)
{
    float2 r;
    if (v2)
        asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "l"(p));
    else
        r = make_float2(__ldg(p), __ldg(p + 1));
    return r;
}

// The split of one FFT of two real rows (fft512_pair's output z, rows A + i B)
// into twice the rows' bins K = a + 16 kk, kk < 16: f(kk, (2 A, 2 B)), with the
// real DC and Nyquist bins of both rows packed at K = 0.  The partner Z[512 - K]
// of lane a is lane 16 - a's; for a = 0 its own, one index on.
template <class F>
__device__ __forceinline__ void split_rows(const float2 (&e)[16], const float2 (&o)[16], int lane, F f)
{
    const int a = lane >> 1, from = (lane & 1) | ((16 - a) & 15) << 1;
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
        const float2 zk = e[P16(kk)];
        float2 s = o[P16(15 - kk)];
        if (a == 0) s = kk ? o[P16((16 - kk) & 15)] : zk;
        float2 zn;
        zn.x = __shfl_sync(0xffffffffu, s.x, from);
        zn.y = __shfl_sync(0xffffffffu, s.y, from);
        // twice the two rows' bins (the 1/2 of the split is applied once,
        // exactly, to the averaged spectrum in k_item_reduce)
        float4 AB = make_float4(zk.x + zn.x, zk.y - zn.y, zk.y + zn.y, zn.x - zk.x);
        if (kk == 0 && a == 0) {
            const float2 zh = o[P16(0)];
            AB = make_float4(2.0f * zk.x, 2.0f * zh.x, 2.0f * zk.y, 2.0f * zh.y);
        }
        f(kk, AB);
    }
}

// |F| of the packed column (0, 256) of a tile, on the even lanes: kx = 0 is
// added to acc, kx = 256 to accN; the odd lanes' column is an ordinary one.
// Both columns are real lines' transforms, so |F[512 - ky]| = |F[ky]| bit for
// bit: per tile only ky = a + 16 kk <= 256 are added, and mirror_column fills
// in the others when the item ends.
__device__ __forceinline__ void packed_column(const float2 (&e)[16], const float2 (&o)[16], int lane, float* accN,
                                              float (&acc)[32])
{
    const int a = lane >> 1, from = (lane & 1) | ((16 - a) & 15) << 1;
    const bool odd = lane & 1;
#pragma unroll
    for (int kk = 0; kk < 17; ++kk) {
        const float2 zk = kk < 16 ? e[P16(kk & 15)] : o[P16(0)];
        float2 s = kk < 16 ? o[P16((15 - kk) & 15)] : e[P16(15)];
        if (a == 0) s = kk == 0 ? e[P16(0)] : o[P16((16 - kk) & 15)];
        float2 zn;
        zn.x = __shfl_sync(0xffffffffu, s.x, from);
        zn.y = __shfl_sync(0xffffffffu, s.y, from);
        if (odd) {
            acc[kk] += amp_xy(zk.x, zk.y);
        } else if (kk < 16 || a == 0) {
            float ax = 0.5f * (zk.x + zn.x), ay = 0.5f * (zk.y - zn.y);
            float bx = 0.5f * (zk.y + zn.y), by = -0.5f * (zk.x - zn.x);
            acc[kk] += amp_xy(ax, ay);
            accN[a + 16 * kk] += amp_xy(by, bx);
        }
    }
#pragma unroll
    for (int kk = 17; kk < 32; ++kk) {
        const float2 zk = o[P16(kk & 15)];
        if (odd) acc[kk] += amp_xy(zk.x, zk.y);
    }
}

// The bins ky > 256 of kx = 0 from their mirrors 512 - ky (lane 16 - a's, or
// its own for a = 0).
__device__ __forceinline__ void mirror_column(int lane, float (&acc)[32])
{
    const int a = lane >> 1, from = (lane & 1) | ((16 - a) & 15) << 1;
#pragma unroll
    for (int kk = 16; kk < 32; ++kk) {
        const float s = __shfl_sync(0xffffffffu, a == 0 ? acc[32 - kk] : acc[31 - kk], from);
        if ((lane & 1) == 0 && (kk > 16 || a > 0)) acc[kk] = s;
    }
}

struct FusedTab {
    const float* img;
    const double* bsum;   // sums of the stride x stride blocks, [nty + 1][ntx + 1]
    int pitch;
    int ntx, nty;
    int offx, offy, stride;
    int vec;              // 2: 8-byte aligned tile rows, 1: 4-byte
    int nbx;              // ntx + 1
};

// Sums of the stride x stride blocks that tile every image (tile = 2 stride,
// so a tile is 2 x 2 blocks): one pass over the images gives every tile mean
// of GCalcMoment2D (Util/GCalcMoment2D.cu:10-58) without a second read.
// Each warp sums whole block rows with 16-byte loads when the rows are
// 16-byte aligned (4 independent FP64 partial sums per lane keep several
// loads in flight); otherwise it falls back to 4-byte loads.  The rows of a
// block are summed in kSumRows interleaved groups whatever the number of
// warps, so that a sum does not depend on the launch's other images.
constexpr int kSumRows = 32;
template <int NW>
__global__ void __launch_bounds__(32 * NW) k_block_sums(const FusedTab* __restrict__ imgs,
                                                        double* const* __restrict__ out)
{
    constexpr int GW = kSumRows / NW;   // row groups per warp: warp, warp + NW, ...
    constexpr int S = FT / 2;           // block rows and columns: the tiles' stride
    static_assert((GW == 1 || GW == 4) && S % kSumRows == 0, "whole groups, and the reduction below");
    __shared__ double sh[kSumRows];
    const FusedTab im = imgs[blockIdx.y];
    const int nby = im.nty + 1;
    const int b = blockIdx.x;
    if (b >= im.nbx * nby) return;
    const int bx = b % im.nbx, by = b / im.nbx;
    const float* src = im.img + (size_t)(im.offy + by * S) * im.pitch + im.offx + bx * S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool v4 = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) && (im.pitch % 4 == 0);
    double s[GW][4];
#pragma unroll
    for (int g = 0; g < GW; ++g) s[g][0] = s[g][1] = s[g][2] = s[g][3] = 0.0;
    // all groups of the warp at once, so that several loads per thread are in
    // flight: 41 micrographs of 4096 x 4096 (2.75 GB, bound by HBM) in 0.38 ms,
    // 0.56 ms with one group after the other
    if (v4) {
        const size_t step = (size_t)NW * im.pitch / 4;
        for (int y = warp; y < S; y += kSumRows) {
            const float4* row = reinterpret_cast<const float4*>(src + (size_t)y * im.pitch) + lane;
#pragma unroll
            for (int x = 0; x < S / 4; x += 32) {
#pragma unroll
                for (int g = 0; g < GW; ++g) {
                    const float4 v = __ldg(row + g * step + x);
                    s[g][0] += (double)v.x;
                    s[g][1] += (double)v.y;
                    s[g][2] += (double)v.z;
                    s[g][3] += (double)v.w;
                }
            }
        }
    } else {
        const size_t step = (size_t)NW * im.pitch;
        for (int y = warp; y < S; y += kSumRows) {
            const float* row = src + (size_t)y * im.pitch + lane;
#pragma unroll 4
            for (int x = 0; x < S; x += 128) {
#pragma unroll
                for (int g = 0; g < GW; ++g)
#pragma unroll
                    for (int k = 0; k < 4; ++k) s[g][k] += (double)__ldg(row + g * step + x + 32 * k);
            }
        }
    }
    double t[GW];
#pragma unroll
    for (int g = 0; g < GW; ++g) t[g] = (s[g][0] + s[g][1]) + (s[g][2] + s[g][3]);
    // each group's sum over the lanes, by halves: of four groups a lane keeps
    // two, then one (6 exchanges, not 20)
    const bool up = GW > 1 && (lane & 16), vp = GW > 1 && (lane & 8);
    double r = t[0];
    if constexpr (GW == 4) {
        const double a0 = (up ? t[2] : t[0]) + __shfl_xor_sync(0xffffffffu, up ? t[0] : t[2], 16);
        const double a1 = (up ? t[3] : t[1]) + __shfl_xor_sync(0xffffffffu, up ? t[1] : t[3], 16);
        r = (vp ? a1 : a0) + __shfl_xor_sync(0xffffffffu, vp ? a0 : a1, 8);
    } else {
        r += __shfl_xor_sync(0xffffffffu, r, 16);
        r += __shfl_xor_sync(0xffffffffu, r, 8);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if ((lane & 7) == 0) sh[warp + NW * (2 * up + vp)] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int g = 0; g < kSumRows; ++g) v += sh[g];
        out[blockIdx.y][b] = v;
    }
}

// The work-item queue of one launch: a 64-bit counter whose low half counts
// items taken from the front (by clusters) and whose high half counts items
// taken from the back (by the cluster-less CTAs).  An index >= nitems means
// the queue is empty.
__device__ __forceinline__ int take_front(unsigned long long* q, int nitems)
{
    const unsigned long long old = atomicAdd(q, 1ull);
    const unsigned front = (unsigned)old, back = (unsigned)(old >> 32);
    return front + back < (unsigned)nitems ? (int)front : nitems;
}
// From the back, while more than `reserve` items remain: a cluster-less CTA
// takes about eight times as long per item as a cluster, so it must not
// take one of the last items, or it would end the launch late.
__device__ __forceinline__ int take_back(unsigned long long* q, int nitems, int reserve)
{
    const unsigned long long cur = atomicAdd(q, 0ull);
    if ((long long)nitems - (long long)((unsigned)cur + (unsigned)(cur >> 32)) <= (long long)reserve) return nitems;
    const unsigned long long old = atomicAdd(q, 1ull << 32);
    const unsigned front = (unsigned)old, back = (unsigned)(old >> 32);
    return front + back < (unsigned)nitems ? nitems - 1 - (int)back : nitems;
}

// Compile-time shape of one cluster configuration.
template <int CL_, int NW_, bool DB_, bool PF_ = true, int MINB_ = 1>
struct FusedShape {
    static constexpr int CL = CL_;                   // CTAs per cluster
    static constexpr int NW = NW_;                   // warps per CTA
    static constexpr bool DB = DB_;                  // double-buffered column buffer
    static constexpr bool PF = PF_;                  // register prefetch of the next row pair
    static constexpr int MINB = MINB_;               // CTAs per SM the registers are sized for
    static constexpr int THR = NW * 32;
    static constexpr int R = FT / CL;                // tile rows per CTA
    static constexpr int C = FT / 2 / CL;            // frequency columns per CTA
    static constexpr int PW = R / 2 / NW;            // row pairs per warp
    static constexpr int NR = C / NW;                // column rounds per warp
    static constexpr int YS = FT + 2;                // column stride of the buffer (16-byte rows, pad)
    static constexpr size_t BUF = (size_t)C * YS * sizeof(float2);   // this CTA's C columns x 512 rows
    static constexpr size_t SCR = (size_t)NW * FSCR * sizeof(float2);
    static constexpr size_t TWL = 16 * 32 * sizeof(float2);
    static constexpr size_t ACCN = FT * sizeof(float);
    static constexpr size_t SMEM = (DB ? 2 : 1) * BUF + SCR + TWL + ACCN;
    static_assert(R % 32 == 0 && PW >= 1 && NR >= 1 && R / 2 == PW * NW && C == NR * NW && C <= 32, "shape");
};
using Shape16 = FusedShape<16, 16, true>;         // 16-CTA clusters, 512 threads
using Shape8W16 = FusedShape<8, 16, false, false>;  // 8-CTA clusters, 512 threads, 128 registers
// 16-CTA clusters of 256 threads at <= 128 registers and 107 KB of shared
// memory: two CTAs (of different clusters, or of one) per SM, so one CTA's
// cluster barrier or DSMEM exchange overlaps the other's FFTs
using Shape16x2 = FusedShape<16, 8, false, false, 2>;
// 16-CTA clusters of 8 warps with the column buffer double-buffered (one
// cluster barrier per tile) and half the per-warp accumulators of an 8 x 8 shape
using Shape16W8 = FusedShape<16, 8, true>;

template <class S>
__global__ void __launch_bounds__(S::THR, S::MINB)
k_fused_spectrum(const FusedTab* __restrict__ imgs, const int4* __restrict__ items, int nitems,
                 const float* __restrict__ taper, const float2* __restrict__ twg,
                 float* __restrict__ partial, unsigned long long* __restrict__ next_item)
{
    constexpr int CL = S::CL, NW = S::NW, R = S::R, C = S::C, PW = S::PW, NR = S::NR, YS = S::YS;
    extern __shared__ __align__(16) unsigned char smem[];
    float2* colbuf0 = reinterpret_cast<float2*>(smem);
    float2* scr_all = reinterpret_cast<float2*>(smem + (S::DB ? 2 : 1) * S::BUF);
    float2* twl = reinterpret_cast<float2*>(smem + (S::DB ? 2 : 1) * S::BUF + S::SCR);
    float* accN = reinterpret_cast<float*>(twl + 16 * 32);

    __shared__ int s_item[2];   // the item rank 0 fetched, by item parity
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = lane >> 1, p = lane & 1;
    float2* scr = scr_all + warp * FSCR;

    // per-lane twiddles exp(-2 pi i l k1 / 512)
    for (int i = tid; i < 16 * 32; i += S::THR) twl[i] = twg[((i & 31) * (i >> 5)) & (FT - 1)];
    __syncthreads();

    int par = 0;    // column-buffer parity (double buffering)
    int ipar = 0;   // s_item parity
    for (;;) {
        // Items are taken in order from one counter, so clusters that become
        // resident late (SMs held by concurrent kernels) simply take fewer.
        // Each s_item slot is rewritten two items later, after a cluster
        // barrier that every peer reaches only once it has read the slot.
        if (r == 0 && tid == 0) s_item[ipar] = take_front(next_item, nitems);
        cluster.sync();
        const int it = *cluster.map_shared_rank(&s_item[ipar], 0);
        ipar ^= 1;
        if (it >= nitems) break;
        const int4 item = items[it];   // (image, first tile, end tile, item index)
        const FusedTab im = imgs[item.x];
        float acc[NR][16];
#pragma unroll
        for (int a = 0; a < NR; ++a)
#pragma unroll
            for (int k = 0; k < 16; ++k) acc[a][k] = 0.0f;
        for (int i = tid; i < FT; i += S::THR) accN[i] = 0.0f;

        for (int t = item.y; t < item.z; ++t) {
            const int tx = t % im.ntx, ty = t / im.ntx;
            const float* src = im.img + (size_t)(im.offy + ty * im.stride + r * R) * im.pitch +
                               im.offx + tx * im.stride;
            // tile mean = four block sums / tile area
            const double* bs = im.bsum + (size_t)ty * im.nbx + tx;
            const float mean = (float)((bs[0] + bs[1] + bs[im.nbx] + bs[im.nbx + 1]) / ((double)FT * FT));
            float2* colbuf = colbuf0 + (S::DB ? (size_t)par * (S::BUF / sizeof(float2)) : 0);
            // peers are done reading this CTA's column buffer: an execution
            // barrier only (the values those reads returned were consumed by
            // the column transforms before the arrive), so the arrive is
            // relaxed and carries no memory fence
            if (!S::DB) {
                asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
                asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
            }

            // ---- row transforms: two rows per FFT, rows read straight from global ----
            // S::PF: the next row pair is loaded into registers while this one
            // is transformed (for 8-warp CTAs, whose 255 registers allow it)
            float na[S::PF ? 16 : 1], nb[S::PF ? 16 : 1];
            if constexpr (S::PF) {
                const float* ga = src + (size_t)(2 * warp) * im.pitch;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    na[j] = __ldg(ga + 32 * j + lane);
                    nb[j] = __ldg(ga + im.pitch + 32 * j + lane);
                }
            }
#pragma unroll
            for (int q4 = 0; q4 < PW; ++q4) {
                const int pp = warp + q4 * NW;
                const int y0 = 2 * pp, Y0 = r * R + y0;
                float ca[16], cb[16];
                if constexpr (S::PF) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        ca[j] = na[j];
                        cb[j] = nb[j];
                    }
                    if (q4 + 1 < PW) {   // prefetch the next row pair
                        const float* ga = src + (size_t)(2 * (pp + NW)) * im.pitch;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            na[j] = __ldg(ga + 32 * j + lane);
                            nb[j] = __ldg(ga + im.pitch + 32 * j + lane);
                        }
                    }
                } else {
                    const float* ga = src + (size_t)y0 * im.pitch;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        ca[j] = __ldg(ga + 32 * j + lane);
                        cb[j] = __ldg(ga + im.pitch + 32 * j + lane);
                    }
                }
                float2 v[16];
                const float* ta = taper + (size_t)Y0 * FT;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    int X = 32 * j + lane;
                    v[j] = make_float2((ca[j] - mean) * __ldg(ta + X), (cb[j] - mean) * __ldg(ta + FT + X));
                }
                fft512_warp(v, scr, twl, lane);
#pragma unroll
                for (int k = 0; k < 16; ++k) scr[sslot(m + 16 * k + 256 * p)] = v[P16(k)];
                __syncwarp();
                // split into the two rows' half spectra and push bin K of both rows
                // into the shared memory of CTA K / C (column K % C, rows Y0, Y0 + 1)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int K = lane + 32 * i;
                    float2 zk = scr[sslot(K)], zn = scr[sslot((FT - K) & (FT - 1))];
                    // twice the two rows' bins (the 1/2 of the split is applied
                    // once, exactly, to the averaged spectrum in k_item_reduce)
                    float4 AB = make_float4(zk.x + zn.x, zk.y - zn.y, zk.y + zn.y, zn.x - zk.x);
                    if (K == 0) {   // pack the real DC and Nyquist bins of both rows
                        float2 zh = scr[sslot(FT / 2)];
                        AB = make_float4(2.0f * zk.x, 2.0f * zh.x, 2.0f * zk.y, 2.0f * zh.y);
                    }
                    float2* dst = cluster.map_shared_rank(colbuf, K / C) + (size_t)(K % C) * YS + Y0;
                    *reinterpret_cast<float4*>(dst) = AB;
                }
                __syncwarp();
            }
            // every column buffer of the cluster is complete (with double
            // buffering this also tells writers of the other buffer that its
            // previous readers are done)
            cluster.sync();

            // ---- column transforms from local shared memory ---------------------
            if (t + 1 < item.z) {   // next tile's rows into L2 while the columns run
                const int t1 = t + 1, tx1 = t1 % im.ntx, ty1 = t1 / im.ntx;
                const float* src1 = im.img + (size_t)(im.offy + ty1 * im.stride + r * R) * im.pitch +
                                    im.offx + tx1 * im.stride;
                for (int q = tid; q < R * 16; q += S::THR) {   // 128-byte lines
                    const float* g = src1 + (size_t)(q >> 4) * im.pitch + (q & 15) * 32;
                    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(g));
                }
            }
#pragma unroll
            for (int rho = 0; rho < NR; ++rho) {
                const int cl = NW * rho + warp;   // local column
                const int K = C * r + cl;         // frequency bin; 0 = packed (0, 256)
                float2 v[16];
                const float2* col = colbuf + (size_t)cl * YS;
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = col[32 * j + lane];
                fft512_warp(v, scr, twl, lane);
                if (K != 0) {
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        float2 z = v[P16(k)];
                        acc[rho][k] += amp(z.x, z.y);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 16; ++k) scr[sslot(m + 16 * k + 256 * p)] = v[P16(k)];
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        int Kk = m + 16 * k + 256 * p;
                        float2 zk = v[P16(k)], zn = scr[sslot((FT - Kk) & (FT - 1))];
                        float ax = 0.5f * (zk.x + zn.x), ay = 0.5f * (zk.y - zn.y);
                        float bx = 0.5f * (zk.y + zn.y), by = -0.5f * (zk.x - zn.x);
                        acc[rho][k] += amp(ax, ay);
                        accN[Kk] += amp(bx, by);
                    }
                    __syncwarp();
                }
            }
            par ^= 1;
        }
        // ---- write this item's partial spectrum (DC moved to row 256) -----------
        float* out = partial + (size_t)item.w * FCX * FT;
#pragma unroll
        for (int rho = 0; rho < NR; ++rho) {
            const int kx = C * r + NW * rho + warp;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                int ky = m + 16 * k + 256 * p;
                int yd = (ky + FT / 2) & (FT - 1);
                out[(size_t)yd * FCX + kx] = acc[rho][k];
            }
        }
        __syncthreads();
        if (r == 0 && warp == 0) {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                int Kk = m + 16 * k + 256 * p;
                int yd = (Kk + FT / 2) & (FT - 1);
                out[(size_t)yd * FCX + FT / 2] = accN[Kk];
            }
        }
        __syncthreads();
    }
    cluster.sync();   // keep shared memory alive until every peer is done
}

// ---- the same with two lines per warp ----------------------------------------
// k_fused_spectrum's work on 8-CTA clusters of 8 warps, with every FFT from
// fft512_pair: a warp transforms four rows (two row pairs), then two columns,
// at a time.  Values, splits and the order of every addition are the same, so
// the spectra are the same bits.
//
// Bound: instruction issue and latency at 8 warps per SM, and the 64 bytes per
// clock of the exchange between SMs.  The one-line kernel issued on 35 % of
// the cycles, mostly waiting for shared memory, shuffles and their queue.  Per
// 512 x 512 tile and cluster: 16.3 us one line per warp (its 8 x 8 shape), 17.8
// two lines, 16.0 with the taper and the sums in tensor memory, 13.3 with the
// bulk copies and the split barrier, 11.8 with the rows half a tile ahead; a
// launch over 41 micrographs of 4096 x 4096 7.99 -> 6.18 ms.
//
// Tensor memory (256 KB per SM, no matrix product here needs it) holds what
// would not fit in registers or shared memory:
//  * the taper of the CTA's 64 rows (128 KB; a CTA keeps its rank, so it is
//    loaded once per launch), which otherwise doubles the tile's L2 reads and
//    stalls each round for their latency;
//  * the item's |F| sums (64 KB), whose 64 registers per thread hold rows in
//    flight instead;
//  * the first 32 of the next tile's 64 rows, parked while the other 32 come
//    in (64 KB): all of a tile's rows are read half a tile ahead.
// Every warp only touches its own lanes and columns, so no barrier is needed.
//
// Exchange: a warp stages its four rows' bins in its transpose scratch as one
// 1 KB block per destination CTA ([column][4 rows]) and eight lanes issue one
// bulk copy each to their CTA's column buffer; the copies signal an mbarrier
// there, which the column transforms wait for (bounded).  16-byte stores into
// the peers' memory, in the same order from every warp, kept the store queue
// full and needed a releasing cluster barrier per tile (a quarter of the
// warps' time in both).  The barrier that says "the column buffers have been
// read" is arrived at after a tile's last column loads and waited for after
// the next tile's first row transforms.
//
// A wait that gives up sets *err (the spectra of the launch are void) and tells
// every CTA of its cluster (s_dead).  A thread that gave up, or whose next wait is
// not over at once and finds that another did, sends, announces and waits for no
// bytes any more; rank 0 takes no further item, and only the cluster barriers that
// keep the CTAs together still run.  Every CTA's copies are complete before the
// last of these, so none lands in shared memory that has been given back.  (With
// s_dead read before every send and wait, and the cold path inline, the kernel took
// 1102 us for 11520 x 8184, against 1070 us and 1067 us without any of this.)
template <int CL_, int NW_>
struct PairShape {
    static constexpr int CL = CL_;                  // CTAs per cluster
    static constexpr int NW = NW_;                  // warps per CTA
    static constexpr int THR = 32 * NW;
    static constexpr int MINB = 8 / NW;             // CTAs per SM
    static constexpr int R = FT / CL;               // tile rows per CTA
    static constexpr int C = FT / 2 / CL;           // frequency columns per CTA
    static constexpr int BLOCK = C * 4;             // float2 of a block: 4 rows of every column of a CTA
    static constexpr int ROUNDS = C / (2 * NW);     // dual FFTs per warp, phase and tile
    static constexpr size_t BUF = (size_t)C * FT * sizeof(float2);
    static constexpr size_t SCR = (size_t)NW * 2 * FT * sizeof(float2);
    static constexpr size_t SMEM = BUF + SCR + 16 * 32 * sizeof(float2) + FT * sizeof(float);
    // tensor-memory columns: per group of four warps (one per lane quarter)
    // the taper of each round (two rows of 32 values per lane), the sums, the
    // parked rows
    static constexpr int TM_TAPER = 64 * ROUNDS, TM_ACC = 32 * ROUNDS, TM_PARK = 64;
    static constexpr int TM_ACC0 = NW / 4 * TM_TAPER, TM_PARK0 = TM_ACC0 + NW / 4 * TM_ACC;
    static constexpr int TM_COLS = 512 / MINB;
    static_assert(ROUNDS == 2 && R == 4 * NW * ROUNDS && NW % 4 == 0 && CL <= 16, "shape");
    static_assert(TM_PARK0 + NW / 4 * TM_PARK <= TM_COLS, "tensor memory");
    static_assert(C == 32 && BUF >= (size_t)FT * 33 * sizeof(float), "write-out stage");
};
using Pair8 = PairShape<8, 8>;

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Waits for the mbarrier phase of the given parity, about a second at most and
// no longer than until *gave_up is set.
__device__ bool wait_phase(uint32_t bar, uint32_t parity, const volatile int* gave_up)
{
    unsigned long long t0 = 0;
    for (uint32_t it = 0;; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((it & 63) == 63) {
            if (*gave_up) return false;
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            if (now - t0 > 1000000000ull) return false;
        }
    }
}

// A wait gave up: for the host, and for every CTA of this thread's cluster.  Not
// inline: the hot loop keeps its registers.
__device__ __noinline__ void tell_gave_up(int* err, uint32_t flag, int ctas)
{
    atomicExch(err, 8);
    for (int k = 0; k < ctas; ++k)
        asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(cluster_addr(flag, k)) : "memory");
}

// 32 values per lane between registers and tensor memory (the warp's lane
// quarter, 32 columns from addr); a get waits for the warp's earlier puts.
__device__ __forceinline__ void tmem_get32(uint32_t addr, float (&v)[32])
{
    asm volatile(
        "tcgen05.wait::st.sync.aligned;\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]),
          "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]),
          "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_put32(uint32_t addr, const float (&v)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
        "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]),
        "f"(v[19]), "f"(v[20]), "f"(v[21]), "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]),
        "f"(v[28]), "f"(v[29]), "f"(v[30]), "f"(v[31]));
}

template <class S>
__global__ void __launch_bounds__(S::THR, S::MINB)
k_fused_spectrum_pair(const FusedTab* __restrict__ imgs, const int4* __restrict__ items, int nitems,
                      const float* __restrict__ taper, const float2* __restrict__ twg,
                      float* __restrict__ partial, unsigned long long* __restrict__ next_item, int* __restrict__ err,
                      uint32_t tile_bytes)   // bytes a tile brings to a CTA's column buffer: S::BUF
{
    extern __shared__ __align__(16) unsigned char smem[];
    float2* colbuf = reinterpret_cast<float2*>(smem);
    float4* scr_all = reinterpret_cast<float4*>(smem + S::BUF);
    float2* twl = reinterpret_cast<float2*>(smem + S::BUF + S::SCR);
    float* accN = reinterpret_cast<float*>(twl + 16 * 32);
    const float4* tw4 = reinterpret_cast<const float4*>(twl);

    __shared__ int s_item[2];   // the item rank 0 fetched, by item parity
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead;      // a wait of this cluster gave up
    __shared__ __align__(8) unsigned long long s_bar;   // the column buffer's bytes of one tile
    const volatile int* const gave_up = &s_dead;
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int a = lane >> 1, h = lane & 1;
    float4* stage = scr_all + (size_t)warp * FT;   // the warp's scratch: two lines, or the blocks it sends
    float4* scr = stage + h * (FT / 2);
    const uint32_t bar = smem_addr(&s_bar);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&s_tmem)),
                     "r"(S::TM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        s_dead = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < 16 * 32; i += S::THR) twl[i] = twg[((i & 31) * (i >> 5)) & (FT - 1)];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const uint32_t tm_taper = tmem + (uint32_t)((warp >> 2) * S::TM_TAPER);
    const uint32_t tm_park = tmem + (uint32_t)(S::TM_PARK0 + (warp >> 2) * S::TM_PARK);
    const uint32_t tm_acc = tmem + (uint32_t)(S::TM_ACC0 + (warp >> 2) * S::TM_ACC);
#pragma unroll 1
    for (int q = 0; q < 2 * S::ROUNDS; ++q) {   // round q / 2, row q % 2 of this half's pair
        const float* ta =
            taper + (size_t)(r * S::R + 4 * (warp + q / 2 * S::NW) + 2 * h + (q & 1)) * FT + 2 * a;
        float v[32];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float2 w = __ldg(reinterpret_cast<const float2*>(ta + 32 * j));
            v[2 * j] = w.x;
            v[2 * j + 1] = w.y;
        }
        tmem_put32(tm_taper + 32 * q, v);
    }

    int ipar = 0;       // s_item parity
    uint32_t phase = 0; // of s_bar: one per tile
    bool dead = false;  // a wait of this thread gave up
    for (;;) {
        // as in k_fused_spectrum: items in order from one counter, each slot
        // rewritten two items later
        if (r == 0 && tid == 0) s_item[ipar] = *gave_up ? nitems : take_front(next_item, nitems);
        cluster.sync();
        const int it = *cluster.map_shared_rank(&s_item[ipar], 0);
        ipar ^= 1;
        if (it >= nitems) break;
        const int4 item = items[it];   // (image, first tile, end tile, item index)
        const FusedTab im = imgs[item.x];
        const bool v2 = im.vec == 2;
        // this lane's first two samples of its half's first row pair in tile t
        auto rows_of = [&](int t) {
            return im.img +
                   (size_t)(im.offy + t / im.ntx * im.stride + r * S::R + 4 * warp + 2 * h) * im.pitch + im.offx +
                   t % im.ntx * im.stride + 2 * a;
        };
        // tile mean = four block sums / tile area
        auto mean_of = [&](int t) {
            const double* bs = im.bsum + (size_t)(t / im.ntx) * im.nbx + t % im.ntx;
            return (float)((bs[0] + bs[1] + bs[im.nbx] + bs[im.nbx + 1]) / ((double)FT * FT));
        };
        for (int i = tid; i < FT; i += S::THR) accN[i] = 0.0f;
        // rows in flight: na, nb hold a row pair of this half, quarter by quarter
        float2 na[16], nb[16];
        auto load_part = [&](const float* p, int part) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                na[4 * part + j] = row2(p + 32 * (4 * part + j), v2);
                nb[4 * part + j] = row2(p + im.pitch + 32 * (4 * part + j), v2);
            }
        };
        auto load_rows = [&](const float* p) {
#pragma unroll
            for (int part = 0; part < 4; ++part) load_part(p, part);
        };
        auto park_rows = [&] {
            float w[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                w[2 * j] = na[j].x;
                w[2 * j + 1] = na[j].y;
            }
            tmem_put32(tm_park, w);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                w[2 * j] = nb[j].x;
                w[2 * j + 1] = nb[j].y;
            }
            tmem_put32(tm_park + 32, w);
        };
        const size_t half_rows = (size_t)(4 * S::NW) * im.pitch;
        // the copies out of this warp's staging have been read
        auto sent = [&] {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
        };
        const float* src = rows_of(item.y);
        float mean = mean_of(item.y);
        load_rows(src);
        park_rows();
        load_rows(src + half_rows);

        for (int t = item.y; t < item.z; ++t) {
            if (tid == 0 && !dead)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(tile_bytes)
                             : "memory");
            const int t1 = t + 1 < item.z ? t + 1 : t;
            const float* src1 = rows_of(t1);
            const float mean1 = mean_of(t1);

            // ---- row transforms: four rows per warp and round ------------------
#pragma unroll
            for (int q = 0; q < S::ROUNDS; ++q) {
                float2 e[16], o[16];
                float w[32];
                if (q == 0) {
                    float x[32];
                    tmem_get32(tm_park, x);
                    tmem_get32(tm_taper, w);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        e[j].x = (x[2 * j] - mean) * w[2 * j];
                        o[j].x = (x[2 * j + 1] - mean) * w[2 * j + 1];
                    }
                    tmem_get32(tm_park + 32, x);
                    tmem_get32(tm_taper + 32, w);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        e[j].y = (x[2 * j] - mean) * w[2 * j];
                        o[j].y = (x[2 * j + 1] - mean) * w[2 * j + 1];
                    }
                    fft512_pair(e, o, scr, tw4, lane, [](int) {});
                } else {
                    tmem_get32(tm_taper + 64, w);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        e[j].x = (na[j].x - mean) * w[2 * j];
                        o[j].x = (na[j].y - mean) * w[2 * j + 1];
                    }
                    tmem_get32(tm_taper + 96, w);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        e[j].y = (nb[j].x - mean) * w[2 * j];
                        o[j].y = (nb[j].y - mean) * w[2 * j + 1];
                    }
                    sent();
                    fft512_pair(e, o, scr, tw4, lane, [&](int part) { load_part(src1, part); });
                }
                __syncwarp();
                // Z[K] and Z[512 - K], K < 256, to CTA K / C: the block's halves
                // hold [column][h] of each, column K % C at K ^ 2 (row block & 3):
                // neither these stores nor the column loads have bank conflicts.
                // (Z[0] and Z[256] meet in column 0.)
                float2* zk = reinterpret_cast<float2*>(stage) + ((a ^ (2 * (warp & 3))) * 2 + h);
                float2* zn = reinterpret_cast<float2*>(stage) + S::BLOCK / 2 + ((((16 - a) & 15) ^ (2 * (warp & 3))) * 2 + h);
                const int up = a == 0 ? 1 : 0;   // bin 256 + 16 k is column 256 - 16 k: one group of 16 up
#pragma unroll
                for (int kk = 0; kk < 16; ++kk) {
                    zk[(kk >> 1) * S::BLOCK + (kk & 1) * 32] = e[P16(kk)];
                    const int g = (15 - kk + up) & 15;   // column group of bin a + 16 kk + 256
                    zn[(g >> 1) * S::BLOCK + (g & 1) * 32] = o[P16(kk)];
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (q == 0 && t > item.y) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
                if (lane < S::CL && !dead) {
                    const uint32_t block = smem_addr(colbuf + (size_t)(S::R / 4 * r + warp + q * S::NW) * S::BLOCK);
                    asm volatile(
                        "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                        ::"r"(cluster_addr(block, lane)),
                        "r"(smem_addr(stage + lane * (S::BLOCK / 2))), "r"((uint32_t)(S::BLOCK * sizeof(float2))),
                        "r"(cluster_addr(bar, lane))
                        : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            sent();
            // every block of this tile has landed in the column buffer
            if (!dead && !wait_phase(bar, phase, gave_up)) [[unlikely]] {
                dead = true;
                tell_gave_up(err, smem_addr(&s_dead), S::CL);
            }
            phase ^= 1;

            // ---- column transforms: two columns per warp and round --------------
#pragma unroll
            for (int q = 0; q < S::ROUNDS; ++q) {
                const int cl = 2 * (warp + q * S::NW) + h;   // local column
                float2 e[16], o[16];
                // rows 32 j + 2a, + 1 (block 8 j + a / 2): the two real rows' bins
                // from one FFT's, twice their value (the 1/2 of the split is applied
                // once, exactly, to the averaged spectrum in k_item_reduce)
                const float2* col = colbuf + (a >> 1) * S::BLOCK + (cl ^ (a & 6)) * 2 + (a & 1);
                const bool packed = q == 0 && r == 0 && warp == 0;   // column 0 on the even lanes: (0, 256)
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float2 zk = col[8 * j * S::BLOCK], zn = col[8 * j * S::BLOCK + S::BLOCK / 2];
                    e[j] = make_float2(zk.x + zn.x, zk.y - zn.y);
                    o[j] = make_float2(zk.y + zn.y, zn.x - zk.x);
                    if (packed && h == 0) {
                        e[j] = make_float2(2.0f * zk.x, 2.0f * zn.x);
                        o[j] = make_float2(2.0f * zk.y, 2.0f * zn.y);
                    }
                }
                if (q == 0) {
                    park_rows();
                    fft512_pair(e, o, scr, tw4, lane, [&](int part) { load_part(src1 + half_rows, part); });
                } else {
                    fft512_pair(e, o, scr, tw4, lane, [](int) {});
                }
                // this warp's column loads of the tile are done
                if (q == S::ROUNDS - 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
                float acc[32];
                if (t > item.y) {
                    tmem_get32(tm_acc + 32 * q, acc);
                } else {
#pragma unroll
                    for (int k = 0; k < 32; ++k) acc[k] = 0.0f;
                }
                if (packed) {
                    packed_column(e, o, lane, accN, acc);
                } else {
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        acc[k] += amp_xy(e[P16(k)].x, e[P16(k)].y);
                        acc[k + 16] += amp_xy(o[P16(k)].x, o[P16(k)].y);
                    }
                }
                tmem_put32(tm_acc + 32 * q, acc);
            }
            src = src1;
            mean = mean1;
        }
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // of the last tile's arrive
        // ---- write this item's partial spectrum (DC moved to row 256) -----------
        // through the column buffer ([row][33], free until the next item's
        // cluster barrier), so that a warp writes 32 adjacent columns of a row
        float* stage_out = reinterpret_cast<float*>(smem);
        __syncthreads();   // every warp is done with the column buffer
#pragma unroll
        for (int q = 0; q < S::ROUNDS; ++q) {
            float acc[32];
            tmem_get32(tm_acc + 32 * q, acc);
            if (q == 0 && r == 0 && warp == 0) mirror_column(lane, acc);
#pragma unroll
            for (int k = 0; k < 32; ++k)
                stage_out[((a + 16 * k + FT / 2) & (FT - 1)) * 33 + 2 * (warp + q * S::NW) + h] = acc[k];
        }
        __syncthreads();
        float* out = partial + (size_t)item.w * FCX * FT + S::C * r + lane;
#pragma unroll 8
        for (int y = warp; y < FT; y += S::NW) out[(size_t)y * FCX] = stage_out[y * 33 + lane];
        if (r == 0)
            for (int ky = tid; ky < FT; ky += S::THR)
                partial[(size_t)item.w * FCX * FT + (size_t)((ky + FT / 2) & (FT - 1)) * FCX + FT / 2] =
                    accN[ky <= FT / 2 ? ky : FT - ky];
        // this thread's plain accesses to the column buffer come before the
        // peers' bulk copies into it, which the next item's cluster barrier
        // admits (another proxy: the barrier alone does not order them)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // this thread's copies have arrived
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster.sync();   // keep shared memory alive until every peer is done
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(S::TM_COLS)
                     : "memory");
}

// ---- tiles on the SMs that the clusters leave free --------------------------
// 8-CTA clusters fit twice per GPC, so some SMs stay idle beside the cluster
// kernel.  One CTA of this kernel runs on each of them, takes work items
// from the same counter and transforms whole tiles alone: the row spectra go
// to the CTA's column buffer in global memory (L2-resident scratch), the
// column transforms read them back, and the item's |F| sums live in a second
// global buffer until the item ends, when they are written to the item's
// partial spectrum in the cluster kernel's layout.  The transforms, the split
// and the order of every addition are those of the cluster kernels, so an
// item's partial spectrum does not depend on which kernel took it.  Two lines
// per warp (fft512_pair), the next round's rows and taper, or columns, in
// flight during each transform.
constexpr int kSoloThreads = 256;
constexpr int kSoloWarps = kSoloThreads / 32;
constexpr int kSoloYS = FT + 2;                                      // column stride, float2
constexpr size_t kSoloColFloat2 = (size_t)(FT / 2) * kSoloYS;        // columns 0..255 of one tile
constexpr size_t kSoloAccFloats = (size_t)(FT / 2) * FT;             // |F| sums, [column pair][8][lane][4]
constexpr size_t kSoloSmem = (size_t)kSoloWarps * 2 * FT * sizeof(float2) + 16 * 32 * sizeof(float2) +
                             FT * sizeof(float);
constexpr int kSoloRounds = FT / 4 / kSoloWarps;                     // rounds of two row pairs, or two columns, per warp

__global__ void __launch_bounds__(kSoloThreads, 1)
k_fused_spectrum_solo(const FusedTab* __restrict__ imgs, const int4* __restrict__ items, int nitems,
                      const float* __restrict__ taper, const float2* __restrict__ twg,
                      float* __restrict__ partial, unsigned long long* __restrict__ next_item, int reserve,
                      float2* __restrict__ colg_all, float* __restrict__ accg_all)
{
    extern __shared__ __align__(16) unsigned char smem[];
    float4* scr_all = reinterpret_cast<float4*>(smem);
    float2* twl = reinterpret_cast<float2*>(scr_all + kSoloWarps * FT);
    const float4* tw4 = reinterpret_cast<const float4*>(twl);
    float* accN = reinterpret_cast<float*>(twl + 16 * 32);
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int a = lane >> 1, h = lane & 1;
    float4* scr = scr_all + (size_t)warp * FT + h * (FT / 2);
    float2* colg = colg_all + (size_t)blockIdx.x * kSoloColFloat2;
    float4* accg = reinterpret_cast<float4*>(accg_all + (size_t)blockIdx.x * kSoloAccFloats) + lane;
    for (int i = tid; i < 16 * 32; i += kSoloThreads) twl[i] = twg[((i & 31) * (i >> 5)) & (FT - 1)];
    for (;;) {
        __syncthreads();   // the previous item is written; every thread has read s_item
        if (tid == 0) s_item = take_back(next_item, nitems, reserve);
        __syncthreads();
        const int it = s_item;
        if (it >= nitems) break;
        const int4 item = items[it];   // (image, first tile, end tile, item index)
        const FusedTab im = imgs[item.x];
        const bool v2 = im.vec == 2;
        for (int i = tid; i < FT; i += kSoloThreads) accN[i] = 0.0f;   // read after the row phase's barrier
        for (int t = item.y; t < item.z; ++t) {
            const bool first = t == item.y;
            const int tx = t % im.ntx, ty = t / im.ntx;
            const double* bs = im.bsum + (size_t)ty * im.nbx + tx;
            const float mean = (float)((bs[0] + bs[1] + bs[im.nbx] + bs[im.nbx + 1]) / ((double)FT * FT));
            // this half's row pair of round q: rows 4 (warp + 8 q) + 2h, + 1
            const int Y = 4 * warp + 2 * h;
            const float* src =
                im.img + (size_t)(im.offy + ty * im.stride + Y) * im.pitch + im.offx + tx * im.stride + 2 * a;
            const float* tap = taper + (size_t)Y * FT + 2 * a;

            // ---- row transforms: the next round's rows and taper in flight ------
            {
                float2 na[16], nb[16], wa[16], wb[16];
                auto load_part = [&](int q, int part) {
                    const float* p = src + (size_t)(4 * kSoloWarps * q) * im.pitch;
                    const float* w = tap + (size_t)(4 * kSoloWarps * q) * FT;
#pragma unroll
                    for (int j = 4 * part; j < 4 * part + 4; ++j) {
                        na[j] = row2(p + 32 * j, v2);
                        nb[j] = row2(p + im.pitch + 32 * j, v2);
                        wa[j] = __ldg(reinterpret_cast<const float2*>(w + 32 * j));
                        wb[j] = __ldg(reinterpret_cast<const float2*>(w + FT + 32 * j));
                    }
                };
#pragma unroll
                for (int part = 0; part < 4; ++part) load_part(0, part);
#pragma unroll 1
                for (int q = 0; q < kSoloRounds; ++q) {
                    float2 e[16], o[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        e[j] = make_float2((na[j].x - mean) * wa[j].x, (nb[j].x - mean) * wb[j].x);
                        o[j] = make_float2((na[j].y - mean) * wa[j].y, (nb[j].y - mean) * wb[j].y);
                    }
                    const int qn = min(q + 1, kSoloRounds - 1);
                    fft512_pair(e, o, scr, tw4, lane, [&](int part) { load_part(qn, part); });
                    float2* dst = colg + (size_t)a * kSoloYS + Y + 4 * kSoloWarps * q;
                    split_rows(e, o, lane, [&](int kk, float4 AB) {
                        *reinterpret_cast<float4*>(dst + (size_t)(16 * kk) * kSoloYS) = AB;
                    });
                }
            }
            __syncthreads();   // the tile's column buffer is complete

            // ---- column transforms from the global column buffer ----------------
            {
                const float2* col = colg + (size_t)(2 * warp + h) * kSoloYS + 2 * a;   // column 2 (warp + 8 q) + h
                float4 nx[16];
                auto load_part = [&](int q, int part) {
                    const float2* p = col + (size_t)(2 * kSoloWarps * q) * kSoloYS;
#pragma unroll
                    for (int j = 4 * part; j < 4 * part + 4; ++j) nx[j] = *reinterpret_cast<const float4*>(p + 32 * j);
                };
#pragma unroll
                for (int part = 0; part < 4; ++part) load_part(0, part);
#pragma unroll 1
                for (int q = 0; q < kSoloRounds; ++q) {
                    float2 e[16], o[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        e[j] = make_float2(nx[j].x, nx[j].y);
                        o[j] = make_float2(nx[j].z, nx[j].w);
                    }
                    float4* ap = accg + (size_t)(warp + kSoloWarps * q) * 8 * 32;
                    float acc[32];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : ap[32 * i];
                        acc[4 * i] = v.x;
                        acc[4 * i + 1] = v.y;
                        acc[4 * i + 2] = v.z;
                        acc[4 * i + 3] = v.w;
                    }
                    const int qn = min(q + 1, kSoloRounds - 1);
                    fft512_pair(e, o, scr, tw4, lane, [&](int part) { load_part(qn, part); });
                    if (q == 0 && warp == 0) {   // column 0 is the packed (0, 256)
                        packed_column(e, o, lane, accN, acc);
                    } else {
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            acc[k] += amp_xy(e[P16(k)].x, e[P16(k)].y);
                            acc[k + 16] += amp_xy(o[P16(k)].x, o[P16(k)].y);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        ap[32 * i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
                }
            }
            __syncthreads();   // the column buffer is free again; accN is complete
        }
        // ---- the item's partial spectrum (DC moved to row 256) ------------------
        float* out = partial + (size_t)item.w * FCX * FT;
#pragma unroll 1
        for (int q = 0; q < kSoloRounds; ++q) {
            const float4* ap = accg + (size_t)(warp + kSoloWarps * q) * 8 * 32;
            float acc[32];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 v = ap[32 * i];
                acc[4 * i] = v.x;
                acc[4 * i + 1] = v.y;
                acc[4 * i + 2] = v.z;
                acc[4 * i + 3] = v.w;
            }
            if (q == 0 && warp == 0) mirror_column(lane, acc);
            const int kx = 2 * (warp + kSoloWarps * q) + h;
#pragma unroll
            for (int k = 0; k < 32; ++k) out[(size_t)((a + 16 * k + FT / 2) & (FT - 1)) * FCX + kx] = acc[k];
        }
        for (int ky = tid; ky < FT; ky += kSoloThreads)
            out[(size_t)((ky + FT / 2) & (FT - 1)) * FCX + FT / 2] = accN[ky <= FT / 2 ? ky : FT - ky];
    }
}

// raw[img] = sum of the img's item partials (in item order) / ntiles / 2.
// group[img] > 1: each partial is one tile, and that many consecutive ones make
// an item; their FP32 sum, in tile order, is what a cluster that takes the
// whole item accumulates, bit for bit.  Where a bounded wait gave up (*err), the
// partials are void and so is the spectrum: NaN throughout, for callers that
// have no other sign of it (gcf_avg_spectrum_noalloc).
__global__ void k_item_reduce(const float* __restrict__ partial, const int* __restrict__ first,
                              const int* __restrict__ group, const float* __restrict__ inv,
                              const int* __restrict__ err, float* __restrict__ raw)
{
    const int n = FCX * FT;
    int img = blockIdx.y;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    const int end = first[img + 1], g = group ? group[img] : 1;
    const float* p = partial + i;
    if (g == 1) {
        for (int k = first[img]; k < end; ++k) s += p[(size_t)k * n];
    } else {
        for (int k = first[img]; k < end; k += g) {
            float f = 0.0f;
            const int m = min(g, end - k);
#pragma unroll 8
            for (int u = 0; u < m; ++u) f += p[(size_t)(k + u) * n];
            s += f;
        }
    }
    if (*err) s = __longlong_as_double(0x7ff8000000000000ll);
    raw[(size_t)img * n + i] = (float)(s * (double)inv[img] * 0.5);   // rows were split without the 1/2
}

template <class S>
cudaLaunchConfig_t fused_cfg(int nclusters, cudaStream_t st, cudaLaunchAttribute* attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nclusters * S::CL, 1, 1);
    cfg.blockDim = dim3(S::THR, 1, 1);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S::CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// c_tw32 of the current device, once.
cudaError_t init_constants()
{
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return cudaSuccess;
    float2 w[16];
    for (int k = 0; k < 16; ++k) {
        double a = -2.0 * M_PI * (double)(16 * k) / FT;
        w[k] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    e = cudaMemcpyToSymbol(c_tw32, w, sizeof(w));
    if (e == cudaSuccess) done[dev] = true;
    return e;
}

template <class S>
cudaError_t prepare_kernel()
{
    cudaError_t ec = init_constants();
    if (ec != cudaSuccess) return ec;
    cudaError_t e = cudaFuncSetAttribute(k_fused_spectrum<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)S::SMEM);
    if (e != cudaSuccess) return e;
    if (S::CL > 8) e = cudaFuncSetAttribute(k_fused_spectrum<S>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

template <class S>
cudaLaunchConfig_t pair_cfg(int nclusters, cudaStream_t st, cudaLaunchAttribute* attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nclusters * S::CL, 1, 1);
    cfg.blockDim = dim3(S::THR, 1, 1);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S::CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <class S>
cudaError_t prepare_pair()
{
    cudaError_t e = init_constants();
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_fused_spectrum_pair<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (e == cudaSuccess && S::CL > 8)
        e = cudaFuncSetAttribute(k_fused_spectrum_pair<S>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

template <class S>
cudaError_t max_pair_clusters(int* n)
{
    *n = 0;
    cudaError_t e = prepare_pair<S>();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = pair_cfg<S>(64, nullptr, attr);
    return cudaOccupancyMaxActiveClusters(n, (void*)k_fused_spectrum_pair<S>, &cfg);
}

template <class S>
cudaError_t launch_pair(int nclusters, cudaStream_t st, const void* descs, const int4* items, int nitems,
                        const float* taper, const float2* tw, float* partial, unsigned long long* next_item, int* err,
                        uint32_t extra_bytes)
{
    if (!err) return cudaErrorInvalidValue;
    cudaError_t e = prepare_pair<S>();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = pair_cfg<S>(nclusters, st, attr);
    return cudaLaunchKernelEx(&cfg, k_fused_spectrum_pair<S>, reinterpret_cast<const FusedTab*>(descs), items, nitems,
                              taper, tw, partial, next_item, err, (uint32_t)S::BUF + extra_bytes);
}

template <class S>
cudaError_t max_clusters(int* n)
{
    *n = 0;
    cudaError_t e = prepare_kernel<S>();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = fused_cfg<S>(64, nullptr, attr);
    return cudaOccupancyMaxActiveClusters(n, (void*)k_fused_spectrum<S>, &cfg);
}

// ---- B-factor lowpass of 512 x 512 spectra with the warp FFT ----------------
// CFindCtfBase::mLowpass (FindCTF/CFindCtfBase.cpp:191-219) filters the full
// spectrum F (512 x 512 real, DC at column 256) by a forward R2C, the
// factor exp(-B (kx^2 + ky^2) / (2 N^2)) / N^2 (GLowpass2D::DoBFactor,
// FindCTF/GLowpass2D.cu:9-23) and a C2R.  The factor is a product of one
// real, even function per axis, so the filter is separable: rows first,
// then columns, each  r' = IDFT(g DFT(r)) / N  with g(k) = exp(-B k^2 / (2 N^2))
// (k wrapped to -N/2 .. N/2).  Because g is real and even it keeps real
// signals real, so two rows (columns) a, b go through one complex FFT as
// a + i b and come back as a' + i b' with no split; the inverse is the
// forward FFT of the conjugate.
constexpr int kLpWarps = 8;

// Filter values g(K) / N for the output layout of fft512_warp: lane 2m+p
// holds bin K = m + 16k + 256p in v[P16(k)].
__device__ __forceinline__ void lp_filter_pass(float2 (&v)[16], float2* scr, const float2* twl, const float* gk,
                                               int lane)
{
    const int m = lane >> 1, p = lane & 1;
    fft512_warp(v, scr, twl, lane);
    // multiply, conjugate and put the spectrum back into natural order
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int K = m + 16 * k + 256 * p;
        const float g = gk[K];
        scr[sslot(K)] = make_float2(v[P16(k)].x * g, -v[P16(k)].y * g);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = scr[sslot(32 * j + lane)];
    __syncwarp();
    fft512_warp(v, scr, twl, lane);   // conj(result) = the filtered pair, bin order
}

// The filter's values g(k) / N, once per context.
__global__ void k_lp_axis(float* __restrict__ g, double bfactor)
{
    const double scale = -bfactor / (2.0 * (double)FT * FT);
    const int k = threadIdx.x, kw = k <= FT / 2 ? k : k - FT;
    g[k] = (float)(exp(scale * (double)kw * kw) / (double)FT);
}

__device__ __forceinline__ void lp_setup(float2* twl, float* gk, const float2* twg, const float* axis)
{
    for (int i = threadIdx.x; i < 16 * 32; i += blockDim.x) twl[i] = twg[((i & 31) * (i >> 5)) & (FT - 1)];
    for (int k = threadIdx.x; k < FT; k += blockDim.x) gk[k] = axis[k];
    __syncthreads();
}

// Rows: one warp per row pair of the full spectrum built from the half
// spectrum (GCalcSpectrum::GenFullSpect's mirror, DC at column 256);
// filtered rows to rowf [m][512][512], only the columns that the column pass
// reads (0, 1 and 256 on).
__global__ void __launch_bounds__(kLpWarps * 32)
k_lowpass_rows(const float* __restrict__ ctf0, const float2* __restrict__ twg, const float* __restrict__ axis,
               float* __restrict__ rowf)
{
    __shared__ float2 s_twl[16 * 32];
    __shared__ float s_g[FT];
    __shared__ float2 s_scr[kLpWarps][FSCR];
    lp_setup(s_twl, s_g, twg, axis);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = blockIdx.y, y0 = 2 * (blockIdx.x * kLpWarps + warp);
    const float* half = ctf0 + (size_t)m * FCX * FT;
    float2 v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int X = 32 * j + lane, xd = X - (FCX - 1);
        float a, b;
        if (xd >= 0) {
            a = half[(size_t)y0 * FCX + xd];
            b = half[(size_t)(y0 + 1) * FCX + xd];
        } else {
            const int ya = (FT - y0) & (FT - 1), yb = (FT - y0 - 1) & (FT - 1);
            a = half[(size_t)ya * FCX - xd];
            b = half[(size_t)yb * FCX - xd];
        }
        v[j] = make_float2(a, b);
    }
    float2* scr = s_scr[warp];
    lp_filter_pass(v, scr, s_twl, s_g, lane);
    // the pair leaves through the scratch in bin order: coalesced rows
    const int mm = lane >> 1, p = lane & 1;
#pragma unroll
    for (int k = 0; k < 16; ++k) scr[sslot(mm + 16 * k + 256 * p)] = v[P16(k)];
    __syncwarp();
    float* ra = rowf + ((size_t)m * FT + y0) * FT;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        if (j > 0 && j < 8) continue;
        if (j == 0 && lane > 1) continue;
        const float2 z = scr[sslot(32 * j + lane)];
        ra[32 * j + lane] = z.x;          // conjugate: a' = Re, b' = -Im
        ra[FT + 32 * j + lane] = -z.y;
    }
}

// Columns: a CTA takes 16 adjacent columns of the row-filtered spectrum (a
// 512 x 16 block through shared memory, 64-byte rows), one column pair per
// warp, and writes them back through the same block; only the columns of the
// half spectrum are kept: out[y][x] = filtered[y][x + 256] (x < 256) and
// out[y][256] = filtered[y][0] (CFindCtfBase.cpp:212-218).  Spectra whose
// background-removed variance is below 1 keep ctf0 (the variance gate of
// mRemoveBackground, FindCTF/CFindCtfBase.cpp:169-174).
//
// Bound: latency (one pair's two FFTs per warp) for few spectra, traffic for
// many.  32 columns per CTA with the results written straight from the lanes
// (one 4-byte piece of 32 rows per store), the filter's exponentials taken by
// every block and all 512 columns handed over by the row pass took, both
// passes together, 25.2 us for one spectrum and 331 us for 256; now
// 13.1 and 232 us.
constexpr int kLpCols = 2 * kLpWarps, kLpPitch = kLpCols + 1;

__global__ void __launch_bounds__(kLpWarps * 32)
k_lowpass_cols(const float* __restrict__ rowf, const float* __restrict__ ctf0, const float2* __restrict__ twg,
               const float* __restrict__ axis, const double* __restrict__ mom, float* __restrict__ out,
               int* __restrict__ lowpassed)
{
    extern __shared__ float s_blk[];   // [512][kLpPitch]
    __shared__ float2 s_twl[16 * 32];
    __shared__ float s_g[FT];
    __shared__ float2 s_scr[kLpWarps][FSCR];
    const int m = blockIdx.y;
    // all but the last block: columns 256 + 16 b ..; the last: columns 0 and 1 (column 0 kept)
    const bool tail = blockIdx.x == FT / 2 / kLpCols;
    const int c0 = tail ? 0 : FT / 2 + kLpCols * blockIdx.x;
    const int ncol = tail ? 2 : kLpCols, nkeep = tail ? 1 : kLpCols, xo = tail ? FT / 2 : c0 - FT / 2;
    const double mean = mom[2 * m], var = mom[2 * m + 1] - mean * mean;
    const bool run = !(var < 1.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) lowpassed[m] = run ? 1 : 0;
    float* o = out + (size_t)m * FCX * FT + xo;
    const int c = threadIdx.x & (kLpCols - 1), r = threadIdx.x / kLpCols;
    constexpr int RS = kLpWarps * 32 / kLpCols;   // rows per pass of the block
    if (!run) {
        const float* h0 = ctf0 + (size_t)m * FCX * FT + xo;
        for (int y = r; y < FT && c < nkeep; y += RS) o[(size_t)y * FCX + c] = h0[(size_t)y * FCX + c];
        return;
    }
    const float* src = rowf + (size_t)m * FT * FT + c0;
    if (c < ncol) {
#pragma unroll 8
        for (int y = r; y < FT; y += RS) s_blk[y * kLpPitch + c] = src[(size_t)y * FT + c];
    }
    lp_setup(s_twl, s_g, twg, axis);
    const int lane = threadIdx.x & 31, cl = 2 * (threadIdx.x >> 5);   // local column of a; b = cl + 1
    if (cl < ncol) {
        float2 v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int y = 32 * j + lane;
            v[j] = make_float2(s_blk[y * kLpPitch + cl], s_blk[y * kLpPitch + cl + 1]);
        }
        lp_filter_pass(v, s_scr[threadIdx.x >> 5], s_twl, s_g, lane);
        const int mm = lane >> 1, p = lane & 1;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int y = mm + 16 * k + 256 * p;
            s_blk[y * kLpPitch + cl] = v[P16(k)].x;          // conjugate: a' = Re, b' = -Im
            s_blk[y * kLpPitch + cl + 1] = -v[P16(k)].y;
        }
    }
    __syncthreads();
    if (c < nkeep) {
#pragma unroll 8
        for (int y = r; y < FT; y += RS) o[(size_t)y * FCX + c] = s_blk[y * kLpPitch + c];
    }
}

}  // namespace

int fused_tile_supported(int tile) { return tile == FT ? 1 : 0; }

cudaError_t launch_lp_axis(float* axis, double bfactor, cudaStream_t st)
{
    k_lp_axis<<<1, FT, 0, st>>>(axis, bfactor);
    return cudaGetLastError();
}

cudaError_t launch_lowpass512(const float* ctf0, const float2* tw, const float* axis, int nmic, const double* moments,
                              float* rowf, float* out, int* lowpassed, cudaStream_t st)
{
    if (nmic <= 0) return cudaSuccess;
    cudaError_t e = init_constants();
    if (e != cudaSuccess) return e;
    k_lowpass_rows<<<dim3(FT / 2 / kLpWarps, nmic), kLpWarps * 32, 0, st>>>(ctf0, tw, axis, rowf);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const size_t sm = (size_t)FT * kLpPitch * sizeof(float);
    if ((e = cudaFuncSetAttribute(k_lowpass_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) !=
        cudaSuccess)
        return e;
    k_lowpass_cols<<<dim3(FT / 2 / kLpCols + 1, nmic), kLpWarps * 32, sm, st>>>(rowf, ctf0, tw, axis, moments, out,
                                                                                lowpassed);
    return cudaGetLastError();
}

// Picks the cluster shape: 8-CTA clusters with two lines per warp wherever they
// can be resident (16 micrographs of 4096 x 4096: 2.30 ms; the one-line shapes
// 816, 168, 162 and 16 take 3.53, 3.51, 3.84 and 4.81 ms), else 16-CTA ones.
cudaError_t fused_max_clusters(int* n, int* shape)
{
    cudaError_t e = max_pair_clusters<Pair8>(n);
    *shape = 8;
    if (e == cudaSuccess && *n > 0) return e;
    cudaGetLastError();
    *shape = 16;
    return max_clusters<Shape16>(n);
}

// Co-resident clusters of one shape: 8 (8 CTAs x 8 warps, two lines per warp), 816 (8 CTAs x 16
// warps, 128 registers), 16 (16 CTAs x 16 warps, double buffered), 162 (16
// CTAs x 8 warps, two CTAs per SM), 168 (16 CTAs x 8 warps, double buffered).
cudaError_t fused_clusters_of(int shape, int* n)
{
    *n = 0;
    switch (shape) {
    case 8: return max_pair_clusters<Pair8>(n);
    case 816: return max_clusters<Shape8W16>(n);
    case 16: return max_clusters<Shape16>(n);
    case 162: return max_clusters<Shape16x2>(n);
    case 168: return max_clusters<Shape16W8>(n);
    default: return cudaErrorInvalidValue;
    }
}

// Host launcher.  descs/items/first/inv are device arrays prepared by the caller.
size_t solo_scratch_float2(int nsolo) { return (size_t)nsolo * kSoloColFloat2; }
size_t solo_scratch_floats(int nsolo) { return (size_t)nsolo * kSoloAccFloats; }

cudaError_t launch_fused(const void* descs, double* const* bsum_out, int max_blocks, const int4* items,
                         int nitems, const int* first, const int* group, const float* inv, int img0, int nimg,
                         const float* taper, const float2* tw, float* partial, float* raw,
                         unsigned long long* next_item, int* err, int nclusters, int shape, cudaStream_t st,
                         cudaEvent_t ev0, cudaEvent_t ev1, const SoloLaunch* solo, unsigned extra_bytes)
{
    if (nclusters < 1) nclusters = 1;
    // few blocks: one per SM, bound by how many loads it has in flight, so 1024
    // threads (1024 x 1024 frame, 16 blocks: 14.1 us with 256 threads, 5.6 with
    // 1024; 2048 x 2048, 64: 20.8 and 6.8 us); many: 256, four blocks per SM
    const auto* tabs = reinterpret_cast<const FusedTab*>(descs) + img0;
    if ((long long)max_blocks * nimg <= 148)
        k_block_sums<32><<<dim3(max_blocks, nimg), 1024, 0, st>>>(tabs, bsum_out + img0);
    else
        k_block_sums<8><<<dim3(max_blocks, nimg), 256, 0, st>>>(tabs, bsum_out + img0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(next_item, 0, sizeof(unsigned long long), st)) != cudaSuccess) return e;
    if (ev0 && (e = record_timing(ev0, st)) != cudaSuccess) return e;
    const bool use_solo = solo && solo->n > 0 && nitems > nclusters;
    if (use_solo) {
        if ((e = cudaEventRecord(solo->fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(solo->st, solo->fork, 0)) != cudaSuccess) return e;
    }
    cudaLaunchAttribute attr[1];
    if (shape == 16) {
        if ((e = prepare_kernel<Shape16>()) != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = fused_cfg<Shape16>(nclusters, st, attr);
        e = cudaLaunchKernelEx(&cfg, k_fused_spectrum<Shape16>, reinterpret_cast<const FusedTab*>(descs), items,
                               nitems, taper, tw, partial, next_item);
    } else if (shape == 168) {
        if ((e = prepare_kernel<Shape16W8>()) != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = fused_cfg<Shape16W8>(nclusters, st, attr);
        e = cudaLaunchKernelEx(&cfg, k_fused_spectrum<Shape16W8>, reinterpret_cast<const FusedTab*>(descs),
                               items, nitems, taper, tw, partial, next_item);
    } else if (shape == 162) {
        if ((e = prepare_kernel<Shape16x2>()) != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = fused_cfg<Shape16x2>(nclusters, st, attr);
        e = cudaLaunchKernelEx(&cfg, k_fused_spectrum<Shape16x2>, reinterpret_cast<const FusedTab*>(descs),
                               items, nitems, taper, tw, partial, next_item);
    } else if (shape == 816) {
        if ((e = prepare_kernel<Shape8W16>()) != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = fused_cfg<Shape8W16>(nclusters, st, attr);
        e = cudaLaunchKernelEx(&cfg, k_fused_spectrum<Shape8W16>, reinterpret_cast<const FusedTab*>(descs),
                               items, nitems, taper, tw, partial, next_item);
    } else {
        e = launch_pair<Pair8>(nclusters, st, descs, items, nitems, taper, tw, partial, next_item, err, extra_bytes);
    }
    if (e != cudaSuccess) return e;
    if (use_solo) {
        // after the cluster launch, so that its clusters are placed first and
        // these CTAs land on the SMs they leave free
        if ((e = cudaFuncSetAttribute(k_fused_spectrum_solo, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSoloSmem)) != cudaSuccess)
            return e;
        k_fused_spectrum_solo<<<solo->n, kSoloThreads, kSoloSmem, solo->st>>>(
            reinterpret_cast<const FusedTab*>(descs), items, nitems, taper, tw, partial, next_item,
            solo->reserve_per_cluster * nclusters, solo->col, solo->acc);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = cudaEventRecord(solo->join, solo->st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(st, solo->join, 0)) != cudaSuccess) return e;
    }
    if (ev1 && (e = record_timing(ev1, st)) != cudaSuccess) return e;
    dim3 g((FCX * FT + 255) / 256, nimg);
    k_item_reduce<<<g, 256, 0, st>>>(partial, first + img0, group ? group + img0 : nullptr, inv + img0, err, raw);
    return cudaGetLastError();
}

}  // namespace gcf

// ===========================================================================
// Allocation-free spectrum entry point.
//
// Some callers cannot call cudaMalloc: a host application whose framework
// owns every device allocation (a fixed arena or a pool with a hard budget),
// or an acquisition loop that must not allocate because cudaMalloc can
// synchronise the device.  gcf_avg_spectrum_noalloc computes the same
// averaged amplitude spectrum as the fused path above with the same kernel,
// but every byte of device storage it needs beyond the caller's input and
// output lives in the file-scope array below.
// ===========================================================================
namespace gcf {
namespace {

constexpr int kNaMaxItems = 16;                 // partial spectra in the scratch
constexpr int kNaMaxTilesPerItem = 256;         // => at most 4096 tiles per image
constexpr size_t kNaPartialBytes = (size_t)kNaMaxItems * FCX * FT * sizeof(float);   // 8.4 MB
constexpr size_t kNaTaperOff = kNaPartialBytes;                                        // 1 MB taper
constexpr size_t kNaTwOff = kNaTaperOff + (size_t)FT * FT * sizeof(float);            // 4 KB twiddles
constexpr size_t kNaBsumOff = kNaTwOff + (size_t)FT * sizeof(float2);                 // block sums
constexpr int kNaMaxBlocks = 2 * kNaMaxItems * kNaMaxTilesPerItem + 2;                 // (ntx+1)(nty+1)
constexpr size_t kNaMetaOff = kNaBsumOff + (size_t)kNaMaxBlocks * sizeof(double);      // descriptors
struct NaMeta {
    FusedTab desc;
    double* bsum_ptr[1];
    int4 items[kNaMaxItems];
    int first[2];
    float inv[1];
    unsigned long long next_item;
    int err;   // a bounded wait of the tile kernel gave up
};
constexpr size_t kNaBytes = kNaMetaOff + ((sizeof(NaMeta) + 255) / 256) * 256;

// The scratch.  In host code this name is only a stand-in; its device
// address comes from cudaGetSymbolAddress at set-up (na_setup).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
unsigned char* g_na_base[kNaMaxDevices] = {};
int g_na_clusters[kNaMaxDevices] = {};
int g_na_shape[kNaMaxDevices] = {};

// Writes one call's descriptors into the scratch.  They travel as a kernel
// parameter (by value), so no host buffer has to outlive the call.
__global__ void k_na_meta(NaMeta m, NaMeta* dst)
{
    const int n = (int)(sizeof(NaMeta) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(&m);
    int* d = reinterpret_cast<int*>(dst);
    for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = src[i];
}

// Once per device, with that device current: find the scratch address and
// fill the constant taper / twiddle tables inside it.  The address is looked
// up on every call (cheap) and compared with the cached one, so a context
// that was torn down and re-created (cudaDeviceReset) is set up again.
gcf_status na_setup(int dev, unsigned char** base, int* clusters)
{
    std::lock_guard<std::mutex> lk(g_na_mutex);
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return GCF_ERR_CUDA;
    if (g_na_base[dev] == static_cast<unsigned char*>(p)) {
        *base = g_na_base[dev];
        *clusters = g_na_clusters[dev];
        return GCF_OK;
    }
    g_na_base[dev] = nullptr;
    std::vector<float> taper((size_t)FT * FT);
    const double c = FT * 0.5, s = FT;
    for (int y = 0; y < FT; ++y)
        for (int x = 0; x < FT; ++x) {   // GRoundEdge (FindCTF/GRoundEdge.cu:7-25)
            double fx = 2.0 * std::fabs(x - c) / s, fy = 2.0 * std::fabs(y - c) / s;
            double r = std::sqrt(fx * fx + fy * fy), v = 0.0;
            if (r < 1.0) {
                double q = 0.5 * (1.0 - std::cos(M_PI * r));
                v = 1.0 - q * q * q;
            }
            taper[(size_t)y * FT + x] = (float)v;
        }
    std::vector<float2> tw(FT);
    for (int t = 0; t < FT; ++t) {
        double a = -2.0 * M_PI * (double)t / FT;
        tw[t] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    unsigned char* b = static_cast<unsigned char*>(p);
    if (cudaMemcpy(b + kNaTaperOff, taper.data(), taper.size() * sizeof(float), cudaMemcpyHostToDevice) !=
            cudaSuccess ||
        cudaMemcpy(b + kNaTwOff, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice) != cudaSuccess)
        return GCF_ERR_CUDA;
    // the copies come from pageable memory and may return before their DMA
    // lands; the caller's stream may be non-blocking: wait for them here
    if (cudaDeviceSynchronize() != cudaSuccess) return GCF_ERR_CUDA;
    int n = 0, shape = 0;
    if (fused_max_clusters(&n, &shape) != cudaSuccess || n <= 0) return GCF_ERR_CUDA;
    g_na_base[dev] = b;
    g_na_clusters[dev] = n;
    g_na_shape[dev] = shape;
    *base = b;
    *clusters = n;
    return GCF_OK;
}

}  // namespace
}  // namespace gcf

namespace gcf {
namespace {

// extra_bytes: see launch_fused
gcf_status na_spectrum(const float* dev_img, int width, int height, int pitch, float* dev_raw_out, cudaStream_t st,
                       unsigned extra_bytes)
{
    if (!dev_img || !dev_raw_out || width < FT || height < FT || pitch < width)
        return GCF_ERR_INVALID_ARG;
    // tile layout of CGenAvgSpectrum::SetSizes (FindCTF/CGenAvgSpectrum.cpp:40-75)
    int ov = (int)(FT * 0.50f) / 2 * 2, stride = FT - ov;
    int ntx = (width - ov) / stride, nty = (height - ov) / stride;
    int nt = ntx * nty;
    if (ntx <= 0 || nty <= 0) return GCF_ERR_IMAGE_TOO_SMALL;
    if (nt > kNaMaxItems * kNaMaxTilesPerItem) return GCF_ERR_INVALID_ARG;   // > 4096 tiles
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDevices) return GCF_ERR_CUDA;
    unsigned char* base = nullptr;
    int clusters = 0;
    gcf_status s = na_setup(dev, &base, &clusters);
    if (s != GCF_OK) return s;
    NaMeta meta;
    std::memset(&meta, 0, sizeof(meta));
    double* bsum = reinterpret_cast<double*>(base + kNaBsumOff);
    meta.desc.img = dev_img;
    meta.desc.bsum = bsum;
    meta.desc.pitch = pitch;
    meta.desc.ntx = ntx;
    meta.desc.nty = nty;
    meta.desc.offx = (width - ntx * FT + (ntx - 1) * ov) / 2;
    meta.desc.offy = (height - nty * FT + (nty - 1) * ov) / 2;
    meta.desc.stride = stride;
    meta.desc.vec = ((meta.desc.offx % 2) == 0 && (stride % 2) == 0 && (pitch % 2) == 0 &&
                     ((uintptr_t)dev_img % 8) == 0) ? 2 : 1;
    meta.desc.nbx = ntx + 1;
    meta.bsum_ptr[0] = bsum;
    // no more items than clusters where that many fit: 294 tiles (5760 x 4092)
    // as 16 items on 15 clusters took two rounds, 355 us against 237 us
    int nitems = std::min(nt, std::min(kNaMaxItems, std::max(clusters, 1)));
    int chunk = (nt + nitems - 1) / nitems;
    nitems = 0;
    for (int t0 = 0; t0 < nt; t0 += chunk, ++nitems)
        meta.items[nitems] = make_int4(0, t0, t0 + chunk < nt ? t0 + chunk : nt, nitems);
    meta.first[0] = 0;
    meta.first[1] = nitems;
    meta.inv[0] = 1.0f / nt;
    // Every partial element is written by the kernel before it is read, so
    // nothing in the scratch has to start at zero; the descriptors below are
    // rewritten on every call.
    NaMeta* dmeta = reinterpret_cast<NaMeta*>(base + kNaMetaOff);
    k_na_meta<<<1, 128, 0, st>>>(meta, dmeta);
    if (cudaGetLastError() != cudaSuccess) return GCF_ERR_CUDA;
    int ncl = clusters < nitems ? clusters : nitems;
    cudaError_t e = launch_fused(&dmeta->desc, dmeta->bsum_ptr, (ntx + 1) * (nty + 1), dmeta->items,
                                 nitems, dmeta->first, nullptr, dmeta->inv, 0, 1,
                                 reinterpret_cast<const float*>(base + kNaTaperOff),
                                 reinterpret_cast<const float2*>(base + kNaTwOff),
                                 reinterpret_cast<float*>(base), dev_raw_out, &dmeta->next_item, &dmeta->err, ncl,
                                 g_na_shape[dev], st, nullptr, nullptr, nullptr, extra_bytes);
    if (e != cudaSuccess) return GCF_ERR_CUDA;
    return GCF_OK;
}

}  // namespace
}  // namespace gcf

extern "C" gcf_status gcf_avg_spectrum_noalloc(const float* dev_img, int width, int height, int pitch,
                                               float* dev_raw_out, void* cuda_stream)
{
    return gcf::na_spectrum(dev_img, width, height, pitch, dev_raw_out, static_cast<cudaStream_t>(cuda_stream), 0);
}

extern "C" gcf_status gcf_avg_spectrum_gave_up(const float* dev_img, int width, int height, int pitch,
                                               float* dev_raw_out, void* cuda_stream)
{
    return gcf::na_spectrum(dev_img, width, height, pitch, dev_raw_out, static_cast<cudaStream_t>(cuda_stream), 16);
}
