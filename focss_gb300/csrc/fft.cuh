// fft.cuh -- FFT building blocks for the SSFM kernels.
//
// A length-L sub-FFT (L = P*Q) is computed by a group of P threads of Q
// elements each, with one exchange through shared memory per transform:
//   1. Q-point DFT in registers over j          (radix-2 DIF, constant twiddles)
//   2. twiddle W_L^{t' u'}                      (table in shared memory)
//   3. write (u, t), read row u of P elements   (caller-chosen conflict-free layout)
//   4. P-point DFT in registers.
// Sign convention: forward = exp(-2 pi i nk/L), unnormalized (FFTW_FORWARD).
//
// Centred indices.  Thread t stands for t' = t or, from P/2 on, t - P, and row
// u of the exchange for u' = u or, from Q/2 on, u - Q: the twiddle angle
// 2 pi t' u' / L is then at most pi/2, one lifting rotation (three FMAs, an
// 8-byte table entry) without a quarter-turn placement.  The relabelling only
// moves indices: thread t holds x[(t' + P j) mod L], j = 0..Q-1,
// and the rows u' hold X[u' + Q s], which fft_pq puts back in order:
//   Q = P:  register j holds X[(t' + P j) mod L] (the layout of the input),
//   Q = 2P: register j holds X[t + P j].
// The double-float twiddle product (16-byte entry, 8 FP32 instructions) that
// this replaced cost ~10 of the row pass's 143 instructions per sample.
//
// Precision.  The split-step loop applies the same transforms thousands of
// times, so a rounding error that depends only on a constant (a twiddle
// factor) repeats identically every step and grows linearly with the step
// count, while roundings that depend on the data decorrelate and grow like
// sqrt(steps).  Every twiddle is therefore a lifting rotation that the inverse
// transform undoes operation by operation (see lift_rot).
#pragma once

#include "common.cuh"

namespace fg {

// a * (w_hi + w_lo) with w = {re_hi, im_hi, re_lo, im_lo}: compensated complex
// product; the representation error of w drops out, data roundings remain.
__device__ __forceinline__ float2 cmul_df(float2 a, float4 w) {
    const float re = fmaf(a.x, w.x, fmaf(-a.y, w.y, fmaf(a.x, w.z, -a.y * w.w)));
    const float im = fmaf(a.x, w.y, fmaf(a.y, w.x, fmaf(a.x, w.w, a.y * w.z)));
    return make_float2(re, im);
}
__host__ __device__ __forceinline__ constexpr int bitrev(int i, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((i >> b) & 1) << (bits - 1 - b);
    return r;
}

__host__ __device__ __forceinline__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n >> 1); }

// Thread-group shape for a sub-FFT of length L.
template <int L>
struct PQ;
template <> struct PQ<16> { static constexpr int P = 4, Q = 4; };
template <> struct PQ<32> { static constexpr int P = 4, Q = 8; };
template <> struct PQ<64> { static constexpr int P = 8, Q = 8; };
template <> struct PQ<128> { static constexpr int P = 8, Q = 16; };
template <> struct PQ<256> { static constexpr int P = 16, Q = 16; };
template <> struct PQ<512> { static constexpr int P = 16, Q = 32; };
template <> struct PQ<1024> { static constexpr int P = 32, Q = 32; };

// Shared-memory layouts for the exchange (element (u, s), u < Q, s < P).
// Row kernels: one group per row, padded rows of P+1 (conflict-free reads).
template <int P>
struct RowLayout {
    int base;
    __device__ __forceinline__ int operator()(int u, int s) const { return base + u * (P + 1) + s; }
};
// Column kernels: C columns interleaved, column index fastest.
template <int P, int C>
struct ColLayout {
    int c;
    __device__ __forceinline__ int operator()(int u, int s) const { return (u * P + s) * C + c; }
};

// Centred index of thread t of P.
template <int P>
__host__ __device__ __forceinline__ int centred(int t) { return t < P / 2 ? t : t - P; }

// ---------------------------------------------------------------------------
// Rotations by lifting (three shears, A. W. Paeth, "A fast algorithm for
// general raster rotation", Graphics Interface 1986): with ts = {tan(theta/2),
// sin(theta)} in FP32,
//     x -= t y;  y += s x;  x -= t y
// rotates (x, y) by theta in three FMAs, and the same shears undone in reverse
// order invert it exactly up to the data's own roundings, whatever the
// rounding of t and s.  A forward transform whose inverse is its exact mirror
// therefore adds no error that repeats identically from step to step (the
// rounding of a plain FP32 twiddle does), which is what the column pass needs:
// it applies the inverse transform, a Kerr phase close to identity and the
// forward transform.  |theta| <= pi/2 keeps |t| <= 1.
__device__ __forceinline__ float2 lift_rot(float2 v, float2 ts) {
    float x = fmaf(-ts.x, v.y, v.x);
    const float y = fmaf(ts.y, x, v.y);
    x = fmaf(-ts.x, y, x);
    return make_float2(x, y);
}
__device__ __forceinline__ float2 lift_rot_inv(float2 v, float2 ts) {
    float x = fmaf(ts.x, v.y, v.x);
    const float y = fmaf(-ts.y, x, v.y);
    x = fmaf(ts.x, y, x);
    return make_float2(x, y);
}
// W_N^e = exp(-2 pi i e/N) as a lifting pair {tan(theta/2), sin(theta)} for
// |e| <= ~N/4 (theta = -2 pi e/N, |theta| <= ~pi/2), N = 2^log2N.  e/N is exact,
// so the pair is a deterministic function of (e, N): a rotation applied in one
// launch is undone exactly in another.
__device__ __forceinline__ float2 sixstep_factor(int e, int log2N) {
    const float r = (float)e * __int_as_float((127 - log2N) << 23);
    float sp, cp;
    sincospif(r, &sp, &cp);  // sin, cos of pi*r;  theta = -2 pi r
    return make_float2(-sp / cp, -2.0f * sp * cp);
}

// v * (-i)^q (exact).
__device__ __forceinline__ float2 quarter_turns(float2 v, int q) {
    const float2 r = (q & 1) ? make_float2(v.y, -v.x) : v;
    return (q & 2) ? make_float2(-r.x, -r.y) : r;
}

// ---------------------------------------------------------------------------
// Mirrored sub-FFTs: twiddles as lifting rotations, and an inverse that undoes
// the forward operation by operation in reverse order (see lift_rot).

// {tan(theta/2), sin(theta)} for theta = -pi*r/32, r = 0..8 (forward sign).
__host__ __device__ __forceinline__ constexpr float2 lift_pi32(int r) {
    constexpr float2 t[9] = {{0.0f, 0.0f},
                             {-0.049126848578453064f, -0.0980171412229538f},
                             {-0.09849140048027039f, -0.19509032368659973f},
                             {-0.1483359932899475f, -0.290284663438797f},
                             {-0.1989123672246933f, -0.3826834261417389f},
                             {-0.25048696994781494f, -0.4713967442512512f},
                             {-0.3033466935157776f, -0.5555702447891235f},
                             {-0.3578057289123535f, -0.6343932747840881f},
                             {-0.4142135679721832f, -0.7071067690849304f}};
    return r >= 0 ? t[r] : float2{-t[-r].x, -t[-r].y};
}

// a * exp(-i pi idx/32) = (-i)^q * rot(-pi r/32), idx = 16 q + r, |r| <= 8.
__device__ __forceinline__ float2 twlift(float2 a, int idx) {
    idx &= 63;
    const int q = (idx + 8) >> 4, r = idx - 16 * q;
    if (r != 0) a = lift_rot(a, lift_pi32(r));
    return quarter_turns(a, q & 3);
}
// Exact inverse of twlift.
__device__ __forceinline__ float2 twlift_inv(float2 a, int idx) {
    idx &= 63;
    const int q = (idx + 8) >> 4, r = idx - 16 * q;
    a = quarter_turns(a, -q & 3);
    return r != 0 ? lift_rot_inv(a, lift_pi32(r)) : a;
}

template <int R>
__device__ __forceinline__ void bitrev_swap(float2 (&v)[R]) {
    constexpr int bits = ilog2c(R);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = bitrev(i, bits);
        if (i < r) {
            const float2 tmp = v[i];
            v[i] = v[r];
            v[r] = tmp;
        }
    }
}

// Forward in-register DFT (radix-2 DIF, natural order in and out).
template <int R>
__device__ __forceinline__ void dft_lift(float2 (&v)[R]) {
#pragma unroll
    for (int half = R / 2; half >= 1; half >>= 1) {
#pragma unroll
        for (int base = 0; base < R; base += 2 * half) {
#pragma unroll
            for (int j = 0; j < half; ++j) {
                const float2 a = v[base + j], b = v[base + j + half];
                v[base + j] = cadd(a, b);
                v[base + j + half] = twlift(csub(a, b), j * (32 / half));
            }
        }
    }
    bitrev_swap<R>(v);
}
// Its mirror: R times the inverse DFT.
template <int R>
__device__ __forceinline__ void dft_lift_inv(float2 (&v)[R]) {
    bitrev_swap<R>(v);
#pragma unroll
    for (int half = 1; half < R; half <<= 1) {
#pragma unroll
        for (int base = 0; base < R; base += 2 * half) {
#pragma unroll
            for (int j = 0; j < half; ++j) {
                const float2 s = v[base + j], d = twlift_inv(v[base + j + half], j * (32 / half));
                v[base + j] = cadd(s, d);
                v[base + j + half] = csub(s, d);
            }
        }
    }
}

// Forward sub-FFT on P threads (layouts in the file comment), and L times its
// inverse.  twPQ[u*P + t] = lifting pair of W_L^{t' u'}: the P threads of a
// group read P consecutive entries (conflict-free).
// BLOCK_SYNC selects __syncthreads (group spans warps) or __syncwarp.
template <int P, int Q, bool BLOCK_SYNC, class Lay>
__device__ __forceinline__ void fft_pq_lift(float2 (&v)[Q], float2* __restrict__ sm, const Lay lay, int t,
                                            const float2* __restrict__ twPQ) {
    static_assert(Q == P || Q == 2 * P, "one or two rows per thread");
    constexpr int M = Q / P;
    dft_lift<Q>(v);
#pragma unroll
    for (int u = 1; u < Q; ++u) v[u] = lift_rot(v[u], twPQ[u * P + t]);
#pragma unroll
    for (int u = 0; u < Q; ++u) sm[lay(u, t)] = v[u];
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
#pragma unroll
    for (int i = 0; i < M; ++i) {
        float2 w[P];
        const int u = t + P * i;
#pragma unroll
        for (int s = 0; s < P; ++s) w[s] = sm[lay(u, s)];
        dft_lift<P>(w);
        // w[s] = X[u' + Q s]; rows from Q/2 on (i = 1 when Q = 2P) have u' = u - Q
#pragma unroll
        for (int s = 0; s < P; ++s) v[i + M * ((s - i) & (P - 1))] = w[s];
    }
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
}
template <int P, int Q, bool BLOCK_SYNC, class Lay>
__device__ __forceinline__ void fft_pq_lift_inv(float2 (&v)[Q], float2* __restrict__ sm, const Lay lay, int t,
                                                const float2* __restrict__ twPQ) {
    static_assert(Q == P || Q == 2 * P, "one or two rows per thread");
    constexpr int M = Q / P;
#pragma unroll
    for (int i = 0; i < M; ++i) {
        float2 w[P];
#pragma unroll
        for (int s = 0; s < P; ++s) w[s] = v[i + M * ((s - i) & (P - 1))];
        dft_lift_inv<P>(w);
        const int u = t + P * i;
#pragma unroll
        for (int s = 0; s < P; ++s) sm[lay(u, s)] = w[s];
    }
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
#pragma unroll
    for (int u = 0; u < Q; ++u) v[u] = sm[lay(u, t)];
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
#pragma unroll
    for (int u = 1; u < Q; ++u) v[u] = lift_rot_inv(v[u], twPQ[u * P + t]);
    dft_lift_inv<Q>(v);
}

// ---------------------------------------------------------------------------
// Column sub-FFT with half the registers: L = 2 Q^2 on P = 2Q threads of Q
// elements (L = 32, 128, 512).  Thread t holds x[(t' + P j) mod L]; after an
// in-register Q-point DFT over j, the twiddle W_L^{t' u'} and one exchange,
// lane pair (u = t >> 1, h = t & 1) holds the even (h = 0) or odd (h = 1) half
// of the P-point DFT over t for row u, transforms it in registers and finishes
// with one radix-2 butterfly across the pair (__shfl_xor, the partner lane
// differs by `pair_xor`).  Output: thread t holds X[(u' + Q k + Q^2 h) mod L],
// k = 0..Q-1.  The inverse mirrors the forward operation by operation.
template <int Q, bool BLOCK_SYNC, class Lay>
__device__ __forceinline__ void fft_p2q_lift(float2 (&v)[Q], float2* __restrict__ sm, const Lay lay, int t,
                                             const float2* __restrict__ twPQ, int pair_xor) {
    constexpr int P = 2 * Q;
    dft_lift<Q>(v);
#pragma unroll
    for (int u = 1; u < Q; ++u) v[u] = lift_rot(v[u], twPQ[u * P + t]);
#pragma unroll
    for (int u = 0; u < Q; ++u) sm[lay(u, t)] = v[u];
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
    const int u = t >> 1, h = t & 1;
#pragma unroll
    for (int s = 0; s < Q; ++s) v[s] = sm[lay(u, h + 2 * s)];
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
    dft_lift<Q>(v);
    const float sg = h ? -1.0f : 1.0f;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        // h = 0: Z = Y0 + W Y1;  h = 1: Z = Y0 - W Y1, W = W_P^k
        const float2 tw = twlift(v[k], k * (32 / Q));
        const float2 mine = h ? tw : v[k];
        const float ox = __shfl_xor_sync(0xffffffffu, mine.x, pair_xor);
        const float oy = __shfl_xor_sync(0xffffffffu, mine.y, pair_xor);
        v[k] = make_float2(fmaf(sg, mine.x, ox), fmaf(sg, mine.y, oy));
    }
}
template <int Q, bool BLOCK_SYNC, class Lay>
__device__ __forceinline__ void fft_p2q_lift_inv(float2 (&v)[Q], float2* __restrict__ sm, const Lay lay, int t,
                                                 const float2* __restrict__ twPQ, int pair_xor) {
    constexpr int P = 2 * Q;
    const int u = t >> 1, h = t & 1;
    const float sg = h ? -1.0f : 1.0f;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        // h = 0: 2 Y0 = Z0 + Z1;  h = 1: 2 Y1 = W^-1 (Z0 - Z1)
        const float ox = __shfl_xor_sync(0xffffffffu, v[k].x, pair_xor);
        const float oy = __shfl_xor_sync(0xffffffffu, v[k].y, pair_xor);
        const float2 sd = make_float2(fmaf(sg, v[k].x, ox), fmaf(sg, v[k].y, oy));
        const float2 tw = twlift_inv(sd, k * (32 / Q));
        v[k] = h ? tw : sd;
    }
    dft_lift_inv<Q>(v);
#pragma unroll
    for (int s = 0; s < Q; ++s) sm[lay(u, h + 2 * s)] = v[s];
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
#pragma unroll
    for (int w = 0; w < Q; ++w) v[w] = sm[lay(w, t)];
    if (BLOCK_SYNC) __syncthreads(); else __syncwarp();
#pragma unroll
    for (int w = 1; w < Q; ++w) v[w] = lift_rot_inv(v[w], twPQ[w * P + t]);
    dft_lift_inv<Q>(v);
}

// Column-pass sub-FFT shape: lane-pair form (P = 2Q) where L = 2 Q^2, else PQ.
template <int L>
struct ColFFT {
    static constexpr bool PAIR = (L == 32 || L == 128 || L == 512);
    static constexpr int Q = PAIR ? (L == 32 ? 4 : L == 128 ? 8 : 16) : PQ<L>::Q;
    static constexpr int P = L / Q;
    // Spectral rows k1 >= KC of the two-pass layout stand for the negative
    // index k1 - L (see col_work); L/2 less the overhang of a thread's first
    // element.
    static constexpr int KC = L / 2 - (PAIR ? Q / 2 : P / 2);
    static_assert(PAIR || P == Q, "column lengths 16, 64, 256, 1024 have P = Q");
};
// Threads per group of the column pass for length L, and KC (host side of ColFFT).
__host__ __device__ __forceinline__ int col_group_p(int L) {
    return L == 32 ? 8 : L == 128 ? 16 : L == 512 ? 32 : (L <= 32 ? 4 : L <= 128 ? 8 : L <= 512 ? 16 : 32);
}
__host__ __device__ __forceinline__ int col_kc(int L) {
    const int P = col_group_p(L), Q = L / P;
    return L / 2 - (P == Q ? P / 2 : Q / 2);
}

// ---------------------------------------------------------------------------
// v * exp(2 pi i x) for a 64-bit fixed-point turn fraction, given as
// Y = 2^64 x + 2^54 (the 2^54 rounds the table index to nearest).  T[j] =
// exp(2 pi i j/512) (times the linear step's gain) is a double-float table
// {re_hi, im_hi, re_lo, im_lo}; the residual rotation theta = 2 pi r, |theta| <=
// pi/512, goes into the low words, T (cos theta - 1 + i sin theta) + T_lo, which
// are at most 6e-3 and so carry it to ~2e-10 in FP32; one compensated product
// then rotates the data.
__device__ __forceinline__ float2 turns_rotate(float2 v, unsigned long long Y, const float4* __restrict__ T512) {
    const unsigned yh = (unsigned)(Y >> 32);
    const float4 t = T512[yh >> 23];
    // 32 bits of the residual below the table index, in units of 2^-41 turn
    const int r = (int)((unsigned)(Y >> 23) ^ 0x80000000u);
    const float th = (float)r * 2.857261873568671e-12f;  // 2 pi / 2^41
    const float th2 = th * th;
    const float s = fmaf(th * th2, -1.0f / 6.0f, th);
    const float cm1 = th2 * fmaf(th2, 1.0f / 24.0f, -0.5f);
    const float lr = fmaf(t.x, cm1, fmaf(-t.y, s, t.z));
    const float li = fmaf(t.y, cm1, fmaf(t.x, s, t.w));
    return cmul_df(v, make_float4(t.x, t.y, lr, li));
}

// A double-float table entry times an FP32 gain, renormalized.
__device__ __forceinline__ float4 scale_df(float4 w, float g) {
    const float re = g * w.x, im = g * w.y;
    return make_float4(re, im, fmaf(g, w.z, fmaf(g, w.x, -re)), fmaf(g, w.w, fmaf(g, w.y, -im)));
}

}  // namespace fg
