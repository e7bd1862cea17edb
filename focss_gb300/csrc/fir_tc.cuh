// fir_tc.cuh -- complex FIR filters on the tensor cores: a filter with fixed
// taps is the product of the Hankel matrix of its input with the Toeplitz
// matrix of its taps, in split FP16 (see triplet_tc_kernel in triplet.cu for
// the operand layout, which is the same here).
//
// Precision.  The tensor core's FP32 accumulator truncates, which shrinks a
// plain split product by ~2e-7 -- a bias that 80 filters in a row add up to
// 1.8e-5.  Here the leading words lie on fixed grids: x scaled to at most 1,
// x_hi a multiple of 2^-11, h scaled to at most 1, h_hi a multiple of 2^-a with
// 11 + a + log2(sum |h_hi|) <= 22, so that every partial sum of x_hi h_hi is
// exact in FP32.  The rest, x_lo = x - x_hi (11 bits) and h - h_hi in two words
// h_mid, h_lo (all 24 bits of h), accumulates apart at the scale 2^-11, where
// the truncation does not matter:
//   y = E0 + 2^-11 (E1 + E2),  E0 = x_hi h_hi,  E1 = x_hi h_mid + x_lo h_hi,
//   E2 = x_hi h_lo + x_lo h_mid   (words other than x_hi, h_hi stored times 2^11).
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace fg {
namespace firtc {

constexpr int ROW = 16;                    // outputs per matrix row
constexpr int M = 128;                     // rows
constexpr int TILE = M * ROW;              // outputs of one product
constexpr int THREADS = 256;               // 8 warps: 4 lane quarters x 2 halves of a row
constexpr int OUT = 8;                     // consecutive outputs per thread
constexpr uint32_t D_COLS = 256;           // FP32 columns: (Re x: E0 E2 E1 | Im x: E0 E2 E1) x h re/im x 16, of 192
constexpr uint32_t STEP_BYTES = 4096;      // Toeplitz bytes per 16 taps: 2 x 128 rows x 16 bytes
__host__ __device__ constexpr int ksteps(int taps) { return (taps + ROW - 1 + 15) / 16; }
// FP16 elements of one array of the split input: the taps' reach behind the
// last row, rounded up to the swizzle's period
__host__ __device__ constexpr int qcap(int ks) { return (16 * ks + TILE - ROW + 127) / 128 * 128; }
constexpr int CAP_MAX = qcap(ksteps(255));  // for the longest filter
// kind::f16, FP32 accumulator, FP16 operands, both K-major
__host__ __device__ constexpr uint32_t idesc(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ uint32_t swz32(uint32_t o) { return o ^ ((o >> 3) & 0x10u); }
// staging index: 8 consecutive float2 per lane, lanes 16 apart, conflict-free
__host__ __device__ constexpr int pad(int o) { return o + (o >> 4); }

// Toeplitz matrices of n filters of T taps and (block n) one of T2 taps, B[x][r] = h[x - r]: per
// 8 taps 128 rows of 16 bytes, 32 rows (r / 16 + r = real / imaginary part of
// output r) each of h_mid, h_hi, h_lo 2^11, h_mid 2^11.  h is scaled to at most
// 1 by a power of two, whose inverse goes to unscale.  conj_rev: the adjoint
// filter conj(h[T-1-t]).
__global__ void toeplitz_kernel(const float2* __restrict__ h, int T, int n, const float2* __restrict__ h2, int T2,
                                int conj_rev, __half* __restrict__ bmat, float* __restrict__ unscale) {
    __shared__ unsigned s_max;
    __shared__ float s_sum;
    if (threadIdx.x == 0) {
        s_max = 0u;
        s_sum = 0.f;
    }
    __syncthreads();
    bmat += (size_t)blockIdx.x * ksteps(T) * (STEP_BYTES / 2);
    h += (size_t)blockIdx.x * T;
    if ((int)blockIdx.x == n) {
        h = h2;
        T = T2;
    }
    float mx = 0.f, re = 0.f, im = 0.f;
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        mx = fmaxf(mx, fmaxf(fabsf(h[t].x), fabsf(h[t].y)));
        re += fabsf(h[t].x);
        im += fabsf(h[t].y);
    }
    mx = warp_max(mx);
    re = warp_sum(re) + warp_sum(im);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&s_max, __float_as_uint(mx));
        atomicAdd(&s_sum, re);
    }
    __syncthreads();
    // 2^ex > max; clamped so that both scale and inverse are normal
    int ex = (int)((s_max >> 23) & 255u) - 126;
    ex = ex < -120 ? -120 : ex > 120 ? 120 : ex;
    const float scale = __uint_as_float((unsigned)(127 - ex) << 23);
    if (threadIdx.x == 0) unscale[blockIdx.x] = __uint_as_float((unsigned)(127 + ex) << 23);
    // grid 2^-a of h_hi: sum |h_hi| <= sum (1 + grid) < 2^bits
    const int bits = (int)((__float_as_uint(s_sum * scale + 1.0f) >> 23) & 255u) - 126;
    const int a = 11 - (bits < 1 ? 1 : bits > 10 ? 10 : bits);
    const float grid = __uint_as_float((unsigned)(127 + a) << 23), inv_grid = __uint_as_float((unsigned)(127 - a) << 23);
    const int ks = ksteps(T);
    for (int i = threadIdx.x; i < ks * (int)(STEP_BYTES / 2); i += blockDim.x) {
        const int x = (i >> 10) * 8 + (i & 7), row = (i >> 3) & 127, word = row >> 5;
        const int d = x - (row & 15);
        float v = 0.f;
        if (d >= 0 && d < T) {
            const float2 c = conj_rev ? make_float2(h[T - 1 - d].x, -h[T - 1 - d].y) : h[d];
            v = ((row >> 4) & 1 ? c.y : c.x) * scale;
        }
        const float hi = rintf(v * grid) * inv_grid, rest = v - hi;   // exact
        const __half mid = __float2half_rn(rest * 2048.f);
        const float low = rest - __half2float(mid) * 0x1p-11f;        // exact
        bmat[i] = word == 0 ? __float2half_rn(rest) : word == 1 ? __float2half_rn(hi) : word == 2 ? __float2half_rn(low * 2048.f) : mid;
    }
}

// The power-of-two scale 2^-e of an input whose largest |x|^2 is pmax: |x| < 2^e.
__device__ __forceinline__ int split_exponent(unsigned pmax_bits) {
    const int E = (int)((pmax_bits >> 23) & 255u) - 126;  // pmax < 2^E
    return pmax_bits ? (E + 1) >> 1 : 0;
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((unsigned)(127 + e) << 23); }

// Splits 8 consecutive scaled samples into the arrays {re hi, im hi, re lo,
// im lo} (pitch bytes apart) at element o, a multiple of 8: one 16-byte store
// each.
__device__ __forceinline__ void split_store8(unsigned char* xs, uint32_t pitch, int o, const float2 (&v)[8], float scale) {
    __half2 a[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const float2 re = make_float2(v[2 * u].x * scale, v[2 * u + 1].x * scale);
        const float2 im = make_float2(v[2 * u].y * scale, v[2 * u + 1].y * scale);
        // multiples of 2^-11: adding 1.5 2^12 leaves the sum an ulp of 2^-11
        const float2 rf = make_float2((re.x + 6144.f) - 6144.f, (re.y + 6144.f) - 6144.f);
        const float2 jf = make_float2((im.x + 6144.f) - 6144.f, (im.y + 6144.f) - 6144.f);
        a[0][u] = __floats2half2_rn(rf.x, rf.y);
        a[1][u] = __floats2half2_rn(jf.x, jf.y);
        a[2][u] = __floats2half2_rn((re.x - rf.x) * 2048.f, (re.y - rf.y) * 2048.f);
        a[3][u] = __floats2half2_rn((im.x - jf.x) * 2048.f, (im.y - jf.y) * 2048.f);
    }
    unsigned char* w = xs + swz32(2u * (unsigned)o);
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(w + q * pitch) = *reinterpret_cast<const uint4*>(a[q]);
}

// The product of the split input at xs with the Toeplitz matrix at bs into
// tensor memory at d, issued by one converged warp and committed to `done`.
__device__ __forceinline__ void issue(uint32_t d, uint32_t xs, uint32_t pitch, uint32_t bs, int ks, unsigned long long* done) {
    uint64_t arh = tcg::smem_desc_sw32(xs), aih = tcg::smem_desc_sw32(xs + pitch);
    uint64_t arl = tcg::smem_desc_sw32(xs + 2 * pitch), ail = tcg::smem_desc_sw32(xs + 3 * pitch);
    // rows from 32 on: h_hi, h_lo, h_mid (96 columns E0 E2 E1); from 0: h_mid,
    // h_hi (64 columns E2 E1)
    uint64_t bl = tcg::smem_desc(bs, 2048, 128), bh = tcg::smem_desc(bs + 512, 2048, 128);
    for (int k = 0; k < ks; ++k) {
        tcg::mma_f16_warp(d, arh, bh, idesc(96), k != 0);
        tcg::mma_f16_warp(d + 96, aih, bh, idesc(96), k != 0);
        tcg::mma_f16_warp(d + 32, arl, bl, idesc(64), true);
        tcg::mma_f16_warp(d + 128, ail, bl, idesc(64), true);
        arh += 2;  // 16 taps: 32 bytes along the input, 4096 along the matrix
        aih += 2;
        arl += 2;
        ail += 2;
        bl += 256;
        bh += 256;
    }
    tcg::mma_commit_warp(done);
}

// Reads back the thread's 8 outputs (row 32 (warp & 3) + lane, half warp >> 2),
// times `f`.
__device__ __forceinline__ void read_outputs(uint32_t tmem, int warp, float f, float2 (&y)[OUT]) {
    const uint32_t t = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(OUT * (warp >> 2));
    // Re y = Re x Re h - Im x Im h, Im y = Re x Im h + Im x Re h; the columns of
    // Im x are 96 further, those of Im h 16
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const uint32_t tr = t + 16 * q, ti = t + 96 + 16 * (1 - q);
        const float sg = q ? 1.0f : -1.0f;
        uint32_t a0[8], b0[8], a1[8], b1[8];
        tcg::ld_x8_async(tr + 32, a0);
        tcg::ld_x8_async(tr + 64, a1);
        tcg::ld_x8_async(ti + 32, b0);
        tcg::ld_x8_async(ti + 64, b1);
        tcg::wait_ld8(a0, a1, b0, b1);
        float low[OUT];
#pragma unroll
        for (int r = 0; r < OUT; ++r)
            low[r] = fmaf(sg, __uint_as_float(b0[r]) + __uint_as_float(b1[r]), __uint_as_float(a0[r]) + __uint_as_float(a1[r]));
        tcg::ld_x8_async(tr, a0);
        tcg::ld_x8_async(ti, b0);
        tcg::wait_ld8(a0, b0, a1, b1);
#pragma unroll
        for (int r = 0; r < OUT; ++r) {
            const float v = fmaf(low[r], 0x1p-11f, fmaf(sg, __uint_as_float(b0[r]), __uint_as_float(a0[r]))) * f;
            if (q)
                y[r].y = v;
            else
                y[r].x = v;
        }
    }
}

}  // namespace firtc
}  // namespace fg
