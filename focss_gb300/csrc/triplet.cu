// triplet.cu -- first-order perturbation (triplet) sum and equalizer.
//
//   y_mode[k] = sum_{(m,n)} C_mn A_mode[k+m] sum_p A_p[k+n] conj(A_p[k+m+n])
//
// for k in [R, N-R), zero elsewhere (SINO::term / SINO::cubic,
// src/focss/equalizer/sino.cpp:161-171, 203-220), and the equalizer
// (rx - y) / linear_weight (:193-196).  Samples outside [0, N) count as zero,
// so box-shaped term sets (|m|, |n| <= R) are accepted as well as the
// reference's diamond |m| + |n| <= R.
//
// Terms are grouped by m on the host into dense n-runs, and outputs into tiles
// of TK = 1024.  Per m a tile forms Q_m[j] = sum_p A_p[j] conj(A_p[j+m]) once;
// S_m[k] = sum_n C_mn Q_m[k+n] is then a correlation with a fixed tap vector,
// i.e. a product of the Hankel matrix Q_m[8 i + x] (k = 8 i + r) with a
// Toeplitz matrix T_m[x][r] = C_m,nlo+x-r, and y += A[k+m] S_m[k].
//
// triplet_tc_kernel runs that product on the tensor cores in split FP16;
// triplet_tile_fp32 is the same sum in FP32 on the CUDA cores, for tiles and
// term lists outside the split's range (see use_tensor and the tile check).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <list>
#include <string>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "tcgen05.cuh"

namespace fg {
namespace {

constexpr int TT = 8;     // outputs per thread
constexpr int NT = 128;   // threads of the FP32 sum
constexpr int TK = TT * NT;

__device__ __forceinline__ int padi(int j) { return j + (j >> 3); }

struct TripletArgs {
    const float2* in;       // batch realizations, `in_bstride` apart, modes x N each
    size_t in_bstride;
    const float2* rx;       // equalizer: batch x modes x N, or null
    float2* out;
    float2 inv_lw;          // 1 / linear_weight (equalizer)
    int modes, samples, radius;
    int groups;
    const int* g_m;         // m of each group
    const int* g_nlo;       // first n of each group's dense run
    const int* g_off;       // groups+1 offsets into coef (each run a multiple of TT long)
    const float2* coef;     // dense C_mn runs
    int halo_q;             // max |n| + TT over groups (Q range beyond the tile)
    int halo_a;             // halo_q + max |m| (A range beyond the tile)
    // tensor cores
    const int4* grp;        // {m, nlo, K steps of 16, byte offset into bmat} of each group
    const unsigned char* bmat;  // Toeplitz matrices (toeplitz_kernel)
    int a_lo, alen;         // the tile reads samples k0 + a_lo + [0, alen)
    int qcap;               // elements of a Q array, a multiple of 8
    int bslot;              // bytes of a Toeplitz buffer
    int coef_exp;           // the matrices hold the coefficients times 2^-coef_exp
    float2* part;           // splits > 1: partial sums, splits x batch x modes x N
    int splits;
    int fp32_units, fp32_pitch;  // teams that sum a tile in FP32 in the tensor-core kernel, and their buffers' pitch
};

// Output o = sample k of a row: zero outside [radius, N - radius), and the equalizer.
__device__ __forceinline__ void finish_output(const TripletArgs& a, size_t o, int k, float2 acc) {
    float2 y = (k >= a.radius && k < a.samples - a.radius) ? acc : make_float2(0.f, 0.f);
    if (a.rx) y = cmul(csub(a.rx[o], y), a.inv_lw);
    a.out[o] = y;
}
__device__ __forceinline__ void write_output(const TripletArgs& a, int b, int modes, int p, int k, float2 acc) {
    if (k >= a.samples) return;
    const size_t o = ((size_t)b * modes + p) * a.samples + k;
    if (a.splits > 1)
        a.part[(size_t)blockIdx.z * gridDim.y * modes * a.samples + o] = acc;
    else
        finish_output(a, o, k, acc);
}
// Joins the partial sums of the splits in order.
__global__ void triplet_join_kernel(const TripletArgs a, size_t n) {
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < n; o += (size_t)gridDim.x * blockDim.x) {
        float2 y = a.part[o];
        for (int z = 1; z < a.splits; ++z) y = cadd(y, a.part[z * n + o]);
        finish_output(a, o, (int)(o % a.samples), y);
    }
}

// One tile in FP32, by NT threads: each owns TT consecutive outputs and slides
// a register window over Q_m along n, so one shared-memory load feeds TT
// complex multiply-adds.  Shared arrays use a padded index j + j/8 so the
// per-thread stride is odd and reads are conflict-free.  Sums groups
// [g0, g1).  Out of line: the tensor-core kernel calls it for single tiles, where
// `unit` numbers the teams of NT threads at work on it, each with buffers of its own.
// `other`: null, or the buffers of the team two further (two back), which sums the
// rest of the groups; it leaves its sums there for this one to add.
__device__ __forceinline__ void team_sync(int id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }
template <int MODES>
__device__ __noinline__ void triplet_tile_fp32(const TripletArgs& a, float2* sh, int k0, int g0, int g1, int unit, float2* other) {
    const int N = a.samples;
    const int b = blockIdx.y, tid = threadIdx.x % NT;
    const auto tile_sync = [&] { team_sync(1 + unit, NT); };
    tile_sync();  // the buffers are free (second tile of a team)
    const int alen = TK + 2 * a.halo_a;
    const int qlen = TK + 2 * a.halo_q;
    float2* As = sh;                           // MODES x padi(alen)
    const int astride = padi(alen) + 1;
    float2* Qs = As + MODES * astride;         // padi(qlen)
    const float2* in = a.in + (size_t)b * a.in_bstride;

    // A tile: index i <-> sample k0 - halo_a + i (zero outside [0, N))
    for (int p = 0; p < MODES; ++p)
        for (int i = tid; i < alen; i += NT) {
            const int s = k0 - a.halo_a + i;
            As[p * astride + padi(i)] = (s >= 0 && s < N) ? in[(size_t)p * N + s] : make_float2(0.f, 0.f);
        }

    float2 acc[MODES][TT];
#pragma unroll
    for (int p = 0; p < MODES; ++p)
#pragma unroll
        for (int r = 0; r < TT; ++r) acc[p][r] = make_float2(0.f, 0.f);

    const int kl = tid * TT;  // first local output of this thread
    for (int g = g0; g < g1; ++g) {
        const int m = a.g_m[g];
        const int nlo = a.g_nlo[g];
        const int off = a.g_off[g], len = a.g_off[g + 1] - off;
        tile_sync();  // previous Q consumed (and A tile ready on the first)
        // Q tile: index i <-> j = k0 - halo_q + i
        for (int i = tid; i < qlen; i += NT) {
            const int ia = i + (a.halo_a - a.halo_q);  // A index of j
            float2 q = make_float2(0.f, 0.f);
#pragma unroll
            for (int p = 0; p < MODES; ++p)
                q = cadd(q, cmulc(As[p * astride + padi(ia)], As[p * astride + padi(ia + m)]));
            Qs[padi(i)] = q;
        }
        tile_sync();
        float2 s[TT];
#pragma unroll
        for (int r = 0; r < TT; ++r) s[r] = make_float2(0.f, 0.f);
        // window w[x] = Q at local output index kl + n + x
        const int qbase = kl + a.halo_q;  // Q index of local output kl at n = 0
        float2 w[2 * TT];
#pragma unroll
        for (int x = 0; x < TT; ++x) w[x] = Qs[padi(qbase + nlo + x)];
        for (int d0 = 0; d0 < len; d0 += TT) {
#pragma unroll
            for (int x = 0; x < TT; ++x) w[TT + x] = Qs[padi(qbase + nlo + d0 + TT + x)];
#pragma unroll
            for (int d = 0; d < TT; ++d) {
                const float2 c = __ldg(a.coef + off + d0 + d);
#pragma unroll
                for (int r = 0; r < TT; ++r) {
                    const float2 q = w[r + d];
                    s[r].x = fmaf(c.x, q.x, fmaf(-c.y, q.y, s[r].x));
                    s[r].y = fmaf(c.x, q.y, fmaf(c.y, q.x, s[r].y));
                }
            }
#pragma unroll
            for (int x = 0; x < TT; ++x) w[x] = w[TT + x];
        }
        // acc_p[k] += A_p[k + m] * s[k]
#pragma unroll
        for (int p = 0; p < MODES; ++p)
#pragma unroll
            for (int r = 0; r < TT; ++r)
                acc[p][r] = cadd(acc[p][r], cmul(As[p * astride + padi(kl + r + m + a.halo_a)], s[r]));
    }

    if (unit >= 2) {
        tile_sync();  // nobody reads the A tile any more
#pragma unroll
        for (int p = 0; p < MODES; ++p)
#pragma unroll
            for (int r = 0; r < TT; ++r) sh[(p * TT + r) * NT + tid] = acc[p][r];
    }
    if (other) team_sync(5 + (unit & 1), 2 * NT);
    if (unit >= 2) return;
#pragma unroll
    for (int p = 0; p < MODES; ++p)
#pragma unroll
        for (int r = 0; r < TT; ++r) {
            if (other) acc[p][r] = cadd(acc[p][r], other[(p * TT + r) * NT + tid]);
            write_output(a, b, MODES, p, k0 + kl + r, acc[p][r]);
        }
}

template <int MODES>
__global__ void __launch_bounds__(NT) triplet_kernel(const TripletArgs a) {
    extern __shared__ float2 sh[];
    triplet_tile_fp32<MODES>(a, sh, blockIdx.x * TK, 0, a.groups, 0, nullptr);
}

// ---------------------------------------------------------------- tensor cores
// S_m on tcgen05: for k = 16 i + r, A[i][x] = Q[16 i + x] (M = 128 rows, one of
// Re Q / Im Q) and B the Toeplitz matrix B[x][r] = C_m,nlo+x-r (re and im
// columns); Re Q B and Im Q B accumulate apart and join as a complex product
// in the epilogue, so one B serves both.  Rows of the 32-byte-swizzled K-major
// layout are 32 bytes = 16 FP16 values apart, exactly the Hankel row pitch, so
// the (swizzled) array Q itself is the operand and a step of 16 taps is an
// address offset.
//
// Precision.  Q and C are scaled by powers of two to just below 2^15 and split
// into FP16 pairs hi + lo 2^-11 (22 bits down to 2^-28 of the largest, below
// that an absolute error of 2^-51 of it), and the
// products hi hi, hi lo, lo hi accumulate in FP32, the last two in columns of
// their own that join with the factor 2^-11 at the end; lo lo (2^-22 of a
// product at most) is left out.  The sum over m is compensated (Kahan).  The
// scale of Q is the tile's largest power; tiles whose power spans more than
// 2^12 between its largest sample and the mean of its weakest 32-sample run,
// or with non-finite values, take the FP32 sum, and so do lists whose
// coefficients span more than 2^28 (plan_tensor).  Relative error against 64
// bits at R = 75 on 2^20 symbols: 1.9e-7 .. 2.3e-7 (the FP32 sum 2.7e-7 ..
// 4.2e-7 on the same inputs).
//
// One CTA per 2048 outputs and SM: warps 8-13 form and split Q_m (a thread of
// them starts the bulk copy of the group's B matrix), warps 14 and 15 issue 4
// MMAs per 16 taps, warps 0-7 read the accumulators back and add A[k+m] S_m.
// What bounds it: shared-memory bandwidth.  An MMA reads 4 KB of A and 1 or 2
// KB of B, ~44 cycles whatever its N, hence 16 outputs per row of A; forming
// Q costs another ~660 cycles of it per group and the epilogue ~130, together
// ~1900 of the ~2300 cycles a group of R = 75 takes.
// R = 75 (11 389 terms) on 2^20 symbols: 0.636 ms = 150 TFLOP/s of the sum's 8
// flops per term (0.69 ms without splitting the tiles of the last wave), where the FP32 kernel took 2.30 ms (42 TFLOP/s, 53 % of the
// FP32 FMA peak); on the way 0.86 ms with 8 outputs per row of A, 0.82 ms
// with one thread issuing from divergent code, 0.75 ms with one issuing warp.
constexpr int TC_ROW = 16;                // outputs per row of A
constexpr int TC_K = NT * TC_ROW;         // outputs per CTA
constexpr int TC_THREADS = 512;
constexpr int kSt = 4;                    // groups in flight: Q buffers and accumulators
constexpr int kEpiWarps = 8, kProdWarps = 6;
constexpr int kPairs = 2 * 32 * kProdWarps, kBatch = 3;
constexpr int kMaxKSteps = 14;            // taps per group: 16 * kMaxKSteps - 15
constexpr int kMaxTcGroups = 512;
constexpr int kHeadroom = 15;             // both factors' FP16 words reach up to 2^15
constexpr uint32_t kDCols = 128;          // FP32 columns: (Re Q | Im Q) x (hi hi | mixed) x C re/im x 16 r
constexpr uint32_t kStepBytes = 2048;     // B bytes per 16 taps: 2 x 64 rows x 16 bytes
// kind::f16, FP32 accumulator (bits 4-5 = 1), FP16 operands, both K-major
__host__ __device__ constexpr uint32_t tri_idesc(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(NT >> 4) << 24);
}
__device__ __forceinline__ int padt(int j) { return j + (j >> 4); }
// Byte offset `o` in the 32-byte-swizzled layout: 16-byte chunks swapped in
// every other 128 bytes (address bit 4 ^= bit 7).
__device__ __forceinline__ uint32_t swz32(uint32_t o) { return o ^ ((o >> 3) & 0x10u); }

template <int MODES>
__global__ void __launch_bounds__(TC_THREADS, 1) triplet_tc_kernel(const TripletArgs a) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) unsigned long long full[kSt], done[kSt], bfull[kSt], drain[2];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ unsigned s_max, s_min;
    __shared__ int s_bad;
    // kSt buffers of {re hi, im hi, re lo, im lo}, each 2 qcap bytes, on a
    // 1024-byte boundary (the swizzle follows absolute address bits)
    unsigned char* Qs = sm + ((1024u - (tcg::smem_addr(sm) & 1023u)) & 1023u);
    unsigned char* Bs = Qs + (size_t)kSt * 8 * a.qcap;                     // kSt buffers of B
    int4* s_grp = reinterpret_cast<int4*>(Bs + (size_t)kSt * a.bslot);
    float2* As = reinterpret_cast<float2*>(s_grp + a.groups);              // MODES x padt(alen)
    const int astride = padt(a.alen) + 1;
    const int N = a.samples, b = blockIdx.y, k0 = blockIdx.x * TC_K;
    const int g0 = (int)((long long)a.groups * blockIdx.z / a.splits);
    const int g1 = (int)((long long)a.groups * (blockIdx.z + 1) / a.splits), ng = g1 - g0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        s_max = 0u;
        s_min = 0x7F7FFFFFu;
        s_bad = 0;
        for (int i = 0; i < kSt; ++i) {
            tcg::mbar_init(&full[i], kProdWarps + kEpiWarps);
            tcg::mbar_init(&done[i], 1);
            tcg::mbar_init(&bfull[i], 1);
        }
        tcg::mbar_init(&drain[0], 1);
        tcg::mbar_init(&drain[1], 1);
        tcg::fence_mbar_init();
    }
    __syncthreads();
    // A tile (zero outside [0, N)), its largest sample power and the smallest
    // non-zero power of a run of 32
    {
        const float2* in = a.in + (size_t)b * a.in_bstride;
        float mx = 0.f, mn = 3.4e38f;
        bool bad = false;
        for (int i0 = warp * 32; i0 < a.alen; i0 += TC_THREADS) {
            const int i = i0 + lane, s = k0 + a.a_lo + i;
            float pw = 0.f;
#pragma unroll
            for (int p = 0; p < MODES; ++p) {
                const float2 v = (i < a.alen && s >= 0 && s < N) ? in[(size_t)p * N + s] : make_float2(0.f, 0.f);
                if (i < a.alen) As[p * astride + padt(i)] = v;
                pw += cnorm(v);
            }
            const float sum = warp_sum(pw);
            bad = bad || !(sum <= 1e30f);
            if (sum > 0.f) mn = fminf(mn, sum);
            mx = fmaxf(mx, pw);
        }
        mx = warp_max(mx);
        if (lane == 0) {
            atomicMax(&s_max, __float_as_uint(mx));
            atomicMin(&s_min, __float_as_uint(mn));
            if (bad) s_bad = 1;
        }
        for (int g = threadIdx.x; g < a.groups; g += TC_THREADS) s_grp[g] = a.grp[g];
    }
    __syncthreads();
    const float pmax = __uint_as_float(s_max), pmin = __uint_as_float(s_min);
    if (s_bad || (pmax > 0.f && (!(pmax > 1e-30f) || pmax > 128.f * pmin))) {  // 2^12 over the run's mean
        // teams of NT threads: one for each TK outputs, or two with half of the groups each
        // (R = 75 on 2^20 symbols, every tile out of range: 2.6 ms; 4.2 with one team, which
        // takes both TK in turn, 2.9 in launches of the FP32 kernel alone)
        const int unit = threadIdx.x / NT, units = a.fp32_units, gm = units == 4 ? (g0 + g1) / 2 : g1;
        float2* sh = reinterpret_cast<float2*>(sm) + (size_t)unit * a.fp32_pitch;
        if (unit < units)
            for (int k = k0 + (units == 1 ? 0 : unit & 1) * TK; k < k0 + TC_K && k < N; k += TK * min(units, 2))
                triplet_tile_fp32<MODES>(a, sh, k, unit >= 2 ? gm : g0, unit >= 2 ? g1 : gm, unit,
                                         units < 4 ? nullptr : unit >= 2 ? sh : sh + 2 * (size_t)a.fp32_pitch);
        return;
    }
    // |Q| <= pmax < 2^e: scale to below 2^kHeadroom
    const int e = (pmax > 0.f ? (int)((__float_as_uint(pmax) >> 23) & 255u) - 126 : 0) - kHeadroom;
    const float qscale = __uint_as_float((unsigned)(127 - e) << 23);
    if (warp == 14) tcg::tmem_alloc(&tmem_base, kSt * kDCols);
    tcg::fence_before_sync();
    __syncthreads();
    tcg::fence_after_sync();
    const uint32_t tmem = tmem_base;

    // epilogue threads: row 32 (warp & 3) + lane, outputs 8 (warp >> 2) .. + 7 of it
    const int kl = (32 * (warp & 3) + lane) * TC_ROW + TT * (warp >> 2);
    float2 acc[MODES][TT], low[MODES][TT];  // sum and its compensation
#pragma unroll
    for (int p = 0; p < MODES; ++p)
#pragma unroll
        for (int r = 0; r < TT; ++r) acc[p][r] = low[p][r] = make_float2(0.f, 0.f);
    int loads = 0;                          // loader: groups whose copy was queued
    if (warp < 8) {
        const uint32_t t0 = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(TT * (warp >> 2));
        if (lane == 0)
            for (int i = 0; i < kSt; ++i) tcg::mbar_arrive(&full[i]);  // every accumulator is free
        for (int i = 0; i < ng; ++i) {
            const int st = i % kSt, m = s_grp[g0 + i].x;
            if (!tcg::mbar_wait(&done[st], (i / kSt) & 1, &abort_flag)) break;
            tcg::fence_after_sync();
            const uint32_t t = t0 + (uint32_t)st * kDCols;
            float2 sv[TT];  // S_m of the thread's outputs
            {
                // Re S = Re Q Re C - Im Q Im C
                uint32_t h0[8], l0[8], h1[8], l1[8];
                tcg::ld_x8_async(t, h0);
                tcg::ld_x8_async(t + 32, l0);
                tcg::ld_x8_async(t + 80, h1);
                tcg::ld_x8_async(t + 112, l1);
                tcg::wait_ld8(h0, l0, h1, l1);
#pragma unroll
                for (int r = 0; r < TT; ++r)
                    sv[r].x = fmaf(__uint_as_float(l0[r]) - __uint_as_float(l1[r]), 0x1p-11f,
                                   __uint_as_float(h0[r]) - __uint_as_float(h1[r]));
            }
            {
                // Im S = Re Q Im C + Im Q Re C
                uint32_t h0[8], l0[8], h1[8], l1[8];
                tcg::ld_x8_async(t + 16, h0);
                tcg::ld_x8_async(t + 48, l0);
                tcg::ld_x8_async(t + 64, h1);
                tcg::ld_x8_async(t + 96, l1);
                tcg::wait_ld8(h0, l0, h1, l1);
#pragma unroll
                for (int r = 0; r < TT; ++r)
                    sv[r].y = fmaf(__uint_as_float(l0[r]) + __uint_as_float(l1[r]), 0x1p-11f,
                                   __uint_as_float(h0[r]) + __uint_as_float(h1[r]));
            }
            tcg::fence_before_sync();
            __syncwarp();
            if (lane == 0) tcg::mbar_arrive(&full[st]);
            const int ia = kl + m - a.a_lo;
#pragma unroll
            for (int r = 0; r < TT; ++r) {
#pragma unroll
                for (int p = 0; p < MODES; ++p) {
                    const float2 x = cmul(As[p * astride + padt(ia + r)], sv[r]);
                    const float2 sum = cadd(acc[p][r], x);
                    low[p][r] = cadd(low[p][r], csub(x, csub(sum, acc[p][r])));
                    acc[p][r] = sum;
                }
            }
        }
    } else if (warp < 14) {
        const int pt = threadIdx.x - 256;
        for (int i = 0; i < ng; ++i) {
            const int st = i % kSt;
            const int4 G = s_grp[g0 + i];
            if (i >= kSt && !tcg::mbar_wait(&done[st], (i / kSt - 1) & 1, &abort_flag)) break;
            if (threadIdx.x == 256) {
                const uint32_t bytes = kStepBytes * G.z;
                tcg::mbar_expect_tx(&bfull[st], bytes);
                tcg::bulk_load(tcg::smem_addr(Bs) + (uint32_t)st * a.bslot, a.bmat + G.w, bytes, &bfull[st]);
                loads = i + 1;
            }
            unsigned char* q = Qs + (size_t)st * 8 * a.qcap;
            const int len = 16 * G.z + TC_K - 16, m = G.x;
            // pairs el, el + 1; kBatch pairs of a thread in flight at a time
            // (a pair alone waits out the latency of its loads and conversions)
            for (int e0 = 2 * pt; e0 < len; e0 += kBatch * kPairs) {
                float2 q0[kBatch], q1[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) q0[u] = q1[u] = make_float2(0.f, 0.f);
#pragma unroll
                for (int p = 0; p < MODES; ++p) {
                    const float2* A = As + p * astride;
                    float2 x0[kBatch], x1[kBatch], y0[kBatch], y1[kBatch];
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        const int ia = G.y - a.a_lo + min(e0 + u * kPairs, len - 2);
                        x0[u] = A[padt(ia)];
                        x1[u] = A[padt(ia + 1)];
                        y0[u] = A[padt(ia + m)];
                        y1[u] = A[padt(ia + 1 + m)];
                    }
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        q0[u].x = fmaf(x0[u].x, y0[u].x, fmaf(x0[u].y, y0[u].y, q0[u].x));
                        q0[u].y = fmaf(x0[u].y, y0[u].x, fmaf(-x0[u].x, y0[u].y, q0[u].y));
                        q1[u].x = fmaf(x1[u].x, y1[u].x, fmaf(x1[u].y, y1[u].y, q1[u].x));
                        q1[u].y = fmaf(x1[u].y, y1[u].x, fmaf(-x1[u].x, y1[u].y, q1[u].y));
                    }
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int el = e0 + u * kPairs;
                    const float2 re = make_float2(q0[u].x * qscale, q1[u].x * qscale);
                    const float2 im = make_float2(q0[u].y * qscale, q1[u].y * qscale);
                    const __half2 rh = __floats2half2_rn(re.x, re.y), ih = __floats2half2_rn(im.x, im.y);
                    const float2 rf = __half22float2(rh), jf = __half22float2(ih);
                    const __half2 rl = __floats2half2_rn((re.x - rf.x) * 2048.f, (re.y - rf.y) * 2048.f);
                    const __half2 il = __floats2half2_rn((im.x - jf.x) * 2048.f, (im.y - jf.y) * 2048.f);
                    if (el < len) {
                        unsigned char* w = q + swz32(2u * el);
                        *reinterpret_cast<__half2*>(w) = rh;
                        *reinterpret_cast<__half2*>(w + 2 * a.qcap) = ih;
                        *reinterpret_cast<__half2*>(w + 4 * a.qcap) = rl;
                        *reinterpret_cast<__half2*>(w + 6 * a.qcap) = il;
                    }
                }
            }
            // warp 8 also vouches for the group's B copy, so that the issuing
            // warp has one barrier per group to look at
            if (warp == 8 && !tcg::mbar_wait(&bfull[st], (i / kSt) & 1, &abort_flag)) break;
            tcg::fence_async_smem();
            __syncwarp();
            if (lane == 0) tcg::mbar_arrive(&full[st]);
        }
    } else {
        // Two issuing warps take turns: a single one gets an MMA out every ~70
        // cycles, where its operands need 48 of shared-memory bandwidth.  A
        // look at a barrier takes ~250 cycles even when its phase is over, so
        // the warp's next barrier is looked at between this group's MMAs.
        int i = warp - 14;
        bool ready = i < ng && tcg::mbar_wait_warp(&full[i], 0, &abort_flag);
        for (; i < ng && ready; i += 2) {
            const int st = i % kSt;
            const int ks = __shfl_sync(0xffffffffu, s_grp[g0 + i].z, 0);
            tcg::fence_after_sync();
            const uint32_t d = tmem + (uint32_t)st * kDCols;
            // A: the four Q arrays; B: 1024 bytes (64 rows) per 8 taps,
            // rows 0-31 the hi words, 32-63 the lo words
            const uint32_t qa = tcg::smem_addr(Qs) + (uint32_t)st * 8u * a.qcap, qn = 2u * a.qcap;
            uint64_t arh = tcg::smem_desc_sw32(qa), aih = tcg::smem_desc_sw32(qa + qn);
            uint64_t arl = tcg::smem_desc_sw32(qa + 2 * qn), ail = tcg::smem_desc_sw32(qa + 3 * qn);
            uint64_t bd = tcg::smem_desc(tcg::smem_addr(Bs) + (uint32_t)st * a.bslot, 1024, 128);
            for (int k = 0; k < ks; ++k) {
                tcg::mma_f16_warp(d, arh, bd, tri_idesc(64), k != 0);
                tcg::mma_f16_warp(d + 64, aih, bd, tri_idesc(64), k != 0);
                tcg::mma_f16_warp(d + 32, arl, bd, tri_idesc(32), true);
                tcg::mma_f16_warp(d + 96, ail, bd, tri_idesc(32), true);
                arh += 2;  // 16 taps: 32 bytes along Q, 2048 along B
                aih += 2;
                arl += 2;
                ail += 2;
                bd += 128;
                if (k == (ks - 1) / 2 && i + 2 < ng)
                    ready = tcg::mbar_wait_warp(&full[(i + 2) % kSt], ((i + 2) / kSt) & 1, &abort_flag);
            }
            tcg::mma_commit_warp(&done[st]);
        }
    }
    __syncthreads();
    const bool ok = !abort_flag;
    if (!ok) {
        // a wait ran out: the queued copies and MMAs land before the CTA
        // leaves (bounded again), and the tile is marked invalid
        if (threadIdx.x == 256)
            for (int i = loads > kSt ? loads - kSt : 0; i < loads; ++i)
                tcg::mbar_wait(&bfull[i % kSt], (i / kSt) & 1, nullptr);
        if (warp >= 14) {
            tcg::mma_commit_warp(&drain[warp - 14]);
            tcg::mbar_wait_warp(&drain[warp - 14], 0, nullptr);
        }
        __syncthreads();
    }
    if (warp < 8) {
        // both scales back, in two halves: no product leaves the range unless the
        // sums or the outputs do
        const int back = e + a.coef_exp, half = back / 2;
        const float f0 = __uint_as_float((unsigned)(127 + half) << 23);
        const float f1 = ok ? __uint_as_float((unsigned)(127 + back - half) << 23) : __int_as_float(0x7fc00000);
#pragma unroll
        for (int p = 0; p < MODES; ++p)
#pragma unroll
            for (int r = 0; r < TT; ++r) write_output(a, b, MODES, p, k0 + kl + r, cscale(cscale(cadd(acc[p][r], low[p][r]), f0), f1));
    }
    tcg::fence_before_sync();
    __syncthreads();
    tcg::fence_after_sync();
    if (warp == 14) tcg::tmem_free(tmem, kSt * kDCols);
}

struct Terms {
    std::vector<int> gm, gnlo, goff, len;  // len: taps of a run before its padding
    std::vector<float2> coef;
    int halo_q = 0, halo_a = 0;
    // tensor cores (empty grp: outside its range)
    std::vector<int4> grp;
    size_t bmat_bytes = 0;
    int a_lo = 0, a_hi = 0, ksteps = 0;
    int exp = 0;
};

// Toeplitz matrices of the groups in B's shared-memory layout, FP16: each
// 8-tap chunk holds 64 rows of 16 bytes, rows r / 16 + r = the real /
// imaginary output r, rows 32.. the same in the lo words.  One CTA per group.
__global__ void toeplitz_kernel(const float2* __restrict__ coef, const int* __restrict__ off, const int4* __restrict__ grp,
                                const int* __restrict__ len, float scale, __half* __restrict__ bmat) {
    const int g = blockIdx.x, ks = grp[g].z, taps = len[g];
    const float2* c = coef + off[g];
    __half* b = bmat + grp[g].w / 2;
    for (int i = threadIdx.x; i < ks * 1024; i += blockDim.x) {
        const int x = (i >> 9) * 8 + (i & 7), row = (i >> 3) & 63, r = row & 15;
        const int d = x - r;
        float v = 0.f;
        if (d >= 0 && d < taps) v = ((row >> 4) & 1 ? c[d].y : c[d].x) * scale;
        const __half hi = __float2half_rn(v);
        b[i] = row < 32 ? hi : __float2half_rn((v - __half2float(hi)) * 2048.f);
    }
}

// Groups of the tensor-core sum.  Left empty when a run has
// more than 16 kMaxKSteps - 15 taps, there are more than kMaxTcGroups groups,
// the coefficients' magnitude leaves [2^-100, 2^100] or they span more than
// 2^28 (zeros aside): the smallest would keep fewer than 22 bits, and where the
// large ones have no part in a symbol they alone make it up.
void plan_tensor(Terms& t) {
    // magnitudes as bits, which order like non-negative floats (this loop is vectorized)
    uint32_t top = 0u, low = 0xFFFFFFFFu;  // low: of the smallest non-zero one, less 1
    const uint32_t* w = reinterpret_cast<const uint32_t*>(t.coef.data());
    for (size_t i = 0; i < 2 * t.coef.size(); i += 2) {
        const uint32_t mag = std::max(w[i] & 0x7FFFFFFFu, w[i + 1] & 0x7FFFFFFFu);
        top = std::max(top, mag);
        low = std::min(low, mag - 1u);
    }
    if (top >= 0x7F800000u || top == 0u || (int)t.gm.size() > kMaxTcGroups) return;  // not finite, or all zero
    low += 1u;
    float cmax, cmin;
    std::memcpy(&cmax, &top, sizeof cmax);
    std::memcpy(&cmin, &low, sizeof cmin);
    if (!(cmax > 0x1p-100f && cmax < 0x1p100f) || cmin < 0x1p-28f * cmax) return;
    for (int l : t.len)
        if (l + 15 > 16 * kMaxKSteps) return;
    std::frexp(cmax, &t.exp);
    t.exp -= kHeadroom;
    t.a_lo = 0;
    t.a_hi = TC_K;
    for (size_t g = 0; g < t.gm.size(); ++g) {
        const int ks = (t.len[g] + 15 + 15) / 16, m = t.gm[g], nlo = t.gnlo[g];
        t.grp.push_back(make_int4(m, nlo, ks, (int)t.bmat_bytes));
        t.bmat_bytes += kStepBytes * (size_t)ks;
        t.ksteps = std::max(t.ksteps, ks);
        t.a_lo = std::min({t.a_lo, m, nlo, nlo + m});
        t.a_hi = std::max({t.a_hi, TC_K + m, nlo + 16 * ks + TC_K - 16, nlo + m + 16 * ks + TC_K - 16});
    }
}

// Terms sorted by (m, n) through an index array (duplicates add in list order).
void build_terms(int n_terms, const int32_t* m, const int32_t* n, const double* c, Terms& t) {
    std::vector<int> at(n_terms);
    for (int i = 0; i < n_terms; ++i) at[i] = i;
    auto before = [&](int i, int j) { return m[i] != m[j] ? m[i] < m[j] : n[i] < n[j]; };
    if (!std::is_sorted(at.begin(), at.end(), before)) std::stable_sort(at.begin(), at.end(), before);
    int max_n = 0, max_m = 0;
    t.goff.push_back(0);
    for (int i = 0; i < n_terms;) {
        int e = i;
        const int mm = m[at[i]], nlo = n[at[i]];
        while (e < n_terms && m[at[e]] == mm) ++e;
        const int run = n[at[e - 1]] - nlo + 1, len = (run + TT - 1) / TT * TT;
        t.gm.push_back(mm);
        t.gnlo.push_back(nlo);
        t.len.push_back(run);
        const size_t base = t.coef.size();
        t.coef.resize(base + len, make_float2(0.f, 0.f));
        while (i < e) {
            const int nn = n[at[i]];
            double re = 0, im = 0;
            for (; i < e && n[at[i]] == nn; ++i) {
                re += c[2 * at[i]];
                im += c[2 * at[i] + 1];
            }
            t.coef[base + (nn - nlo)] = make_float2((float)re, (float)im);
        }
        t.goff.push_back((int)t.coef.size());
        max_m = std::max(max_m, std::abs(mm));
        max_n = std::max({max_n, std::abs(nlo), std::abs(nlo + len - 1)});
    }
    t.halo_q = max_n + TT;
    t.halo_a = t.halo_q + max_m;
    plan_tensor(t);
}
}  // namespace

// Device term tables of recent term lists, per context, most recent first: an
// equalizer applied again with the same coefficients skips the host grouping
// and the upload.  A list is recognised by its contents (compared with a host
// copy: ~20 us for the 11 361 terms of R = 75, where hashing them took 0.6 ms
// of every call).
struct TermEntry {
    std::vector<int32_t> m, n;
    std::vector<double> coef;
    void* dev = nullptr;
    int ng = 0, halo_q = 0, halo_a = 0, a_lo = 0, alen = 0, ksteps = 0, exp = 0;
    size_t coef_offset = 0, grp_offset = 0, len_offset = 0, bmat_offset = 0;
};
struct TermCache {
    std::list<TermEntry> entries;
};
void free_term_cache(TermCache* t) {
    if (!t) return;
    for (TermEntry& e : t->entries) cudaFree(e.dev);
    delete t;
}

namespace {
constexpr size_t kMaxTermPlans = 16;

bool same_terms(const TermEntry& e, int n_terms, const int32_t* m, const int32_t* n, const double* c) {
    const size_t k = (size_t)n_terms;
    return e.m.size() == k && !std::memcmp(e.m.data(), m, sizeof(int32_t) * k) &&
           !std::memcmp(e.n.data(), n, sizeof(int32_t) * k) && !std::memcmp(e.coef.data(), c, sizeof(double) * 2 * k);
}

// The cached device tables of a term list (built and uploaded on a miss).
focss_status term_plan(Ctx* c, int n_terms, const int32_t* m, const int32_t* n, const double* coef,
                       const TermEntry** out) {
    if (!c->terms) c->terms = new TermCache();
    std::list<TermEntry>& es = c->terms->entries;
    for (auto it = es.begin(); it != es.end(); ++it)
        if (same_terms(*it, n_terms, m, n, coef)) {
            es.splice(es.begin(), es, it);
            *out = &es.front();
            return FOCSS_OK;
        }
    for (int i = 0; i < n_terms; ++i)
        if (std::abs(m[i]) > 4096 || std::abs(n[i]) > 4096)
            return set_error(c, FOCSS_ERR_INVALID_ARG, "triplet: |m|, |n| must be <= 4096");
    Terms t;
    build_terms(n_terms, m, n, coef, t);
    TermEntry p;
    p.ng = (int)t.gm.size();
    p.halo_q = t.halo_q;
    p.halo_a = t.halo_a;
    p.a_lo = t.a_lo;
    p.alen = t.a_hi - t.a_lo;
    p.ksteps = t.ksteps;
    p.exp = t.exp;
    auto up16 = [](size_t v) { return (v + 15) / 16 * 16; };
    p.coef_offset = up16(sizeof(int) * (3 * (size_t)p.ng + 1));
    p.grp_offset = up16(p.coef_offset + sizeof(float2) * t.coef.size());
    p.len_offset = up16(p.grp_offset + sizeof(int4) * t.grp.size());
    p.bmat_offset = up16(p.len_offset + sizeof(int) * p.ng);
    std::vector<char> host(p.bmat_offset, 0);
    int* hi = (int*)host.data();
    std::copy(t.gm.begin(), t.gm.end(), hi);
    std::copy(t.gnlo.begin(), t.gnlo.end(), hi + p.ng);
    std::copy(t.goff.begin(), t.goff.end(), hi + 2 * p.ng);
    std::copy(t.coef.begin(), t.coef.end(), (float2*)(host.data() + p.coef_offset));
    std::copy(t.grp.begin(), t.grp.end(), (int4*)(host.data() + p.grp_offset));
    std::copy(t.len.begin(), t.len.end(), (int*)(host.data() + p.len_offset));
    p.m.assign(m, m + n_terms);
    p.n.assign(n, n + n_terms);
    p.coef.assign(coef, coef + 2 * (size_t)n_terms);
    if (es.size() >= kMaxTermPlans) {  // drop the oldest (in-flight kernels finish first)
        cudaStreamSynchronize(c->stream);
        cudaFree(es.back().dev);
        es.pop_back();
    }
    cudaError_t e = cudaMalloc(&p.dev, p.bmat_offset + t.bmat_bytes);
    if (e != cudaSuccess) return cuda_check(c, e, "triplet tables");
    e = cudaMemcpy(p.dev, host.data(), host.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !t.grp.empty()) {
        // While the context's stream is captured, on a stream of its own: the
        // entry serves calls made before the graph runs, too.
        char* d = (char*)p.dev;
        const bool aside = stream_capturing(c->stream);
        cudaStream_t s = c->stream;
        if (aside) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
        if (e == cudaSuccess) {
            toeplitz_kernel<<<p.ng, 256, 0, s>>>((const float2*)(d + p.coef_offset), (const int*)d + 2 * (size_t)p.ng,
                                                 (const int4*)(d + p.grp_offset), (const int*)(d + p.len_offset),
                                                 std::ldexp(1.f, -p.exp), (__half*)(d + p.bmat_offset));
            count_launch();
            e = cudaGetLastError();
            if (aside) {
                if (e == cudaSuccess) e = cudaStreamSynchronize(s);
                cudaStreamDestroy(s);
            }
        }
    }
    if (e != cudaSuccess) {
        cudaFree(p.dev);
        return cuda_check(c, e, "triplet upload");
    }
    es.push_front(std::move(p));
    *out = &es.front();
    return FOCSS_OK;
}

template <int MODES>
cudaError_t launch_triplet(const TripletArgs& a, size_t smem, bool tensor, dim3 grid, cudaStream_t s) {
    auto kern = tensor ? triplet_tc_kernel<MODES> : triplet_kernel<MODES>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, tensor ? TC_THREADS : NT, smem, s>>>(a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

// The triplet sum over `modes` consecutive rows of each realization of `in`
// (realizations in_bstride apart), written to `out` (batch x modes x N);
// with rx, the equalizer (rx - y) / linear_weight instead.
focss_status run_triplet_rows(Ctx* c, const float2* in, size_t in_bstride, int modes, int samples, int batch,
                              const float2* rx, int radius, int n_terms, const int32_t* m, const int32_t* n,
                              const double* coef, float2 inv_lw, float2* out) {
    if (modes < 1 || modes > 2)
        return set_error(c, FOCSS_ERR_UNSUPPORTED, "triplet: 1 or 2 modes");
    if (n_terms <= 0 || !m || !n || !coef) return set_error(c, FOCSS_ERR_INVALID_ARG, "triplet: empty term list");
    const TermEntry* t = nullptr;
    focss_status st = term_plan(c, n_terms, m, n, coef, &t);
    if (st != FOCSS_OK) return st;
    const size_t ng = (size_t)t->ng;
    const char* d = (const char*)t->dev;
    TripletArgs a{};
    a.in = in;
    a.in_bstride = in_bstride;
    a.rx = rx;
    a.out = out;
    a.inv_lw = inv_lw;
    a.modes = modes;
    a.samples = samples;
    a.radius = radius;
    a.groups = (int)ng;
    a.g_m = (const int*)d;
    a.g_nlo = (const int*)d + ng;
    a.g_off = (const int*)d + 2 * ng;
    a.coef = (const float2*)(d + t->coef_offset);
    a.halo_q = t->halo_q;
    a.halo_a = t->halo_a;
    const int alen = TK + 2 * t->halo_a, qlen = TK + 2 * t->halo_q;
    size_t smem = sizeof(float2) * ((size_t)modes * (alen + alen / 8 + 2) + qlen + qlen / 8 + 2);
    if (smem > 200 * 1024) return set_error(c, FOCSS_ERR_UNSUPPORTED, "triplet: term offsets too large for a tile");
    bool tensor = t->ksteps > 0;
    a.splits = 1;
    if (tensor) {
        a.grp = (const int4*)(d + t->grp_offset);
        a.bmat = (const unsigned char*)(d + t->bmat_offset);
        a.bslot = (int)kStepBytes * t->ksteps;
        a.a_lo = t->a_lo;
        a.alen = t->alen;
        a.qcap = (16 * t->ksteps + TC_K - 16 + 127) / 128 * 128;
        a.coef_exp = t->exp;
        const size_t need = 1024 + (size_t)kSt * (8 * (size_t)a.qcap + a.bslot) + sizeof(int4) * ng +
                            sizeof(float2) * (size_t)modes * (a.alen + a.alen / 16 + 2);
        tensor = need <= 220 * 1024;
        if (tensor) {  // a tile may take the FP32 sum, by as many teams as find room
            a.fp32_pitch = (int)(smem / sizeof(float2));
            a.fp32_units = 4 * smem <= 220 * 1024 ? 4 : 2 * smem <= 220 * 1024 ? 2 : 1;
            smem = std::max(a.fp32_units * smem, need);
        }
    }
    const int tile = tensor ? TC_K : TK;
    dim3 grid((samples + tile - 1) / tile, batch);
    const size_t total = (size_t)batch * modes * samples;
    if (tensor && !stream_capturing(c->stream)) {  // (a graph would hold scratch that a larger call replaces)
        // The groups of a tile can be split over CTAs, whose partial sums a second
        // kernel joins (at least 4 groups each): with fewer tiles than SMs to occupy
        // them, with more to fill the last wave (2^20 symbols are 3.4 waves of
        // tiles, 6.7 of half tiles: 0.694 -> 0.636 ms).  Counted in tiles' times:
        // waves of 1/s tile, each with its set-up (~2 %), and the join.
        const long long tiles = (long long)grid.x * batch, sms = sm_count();
        double best = 1e300;
        for (int s = 1; s <= 32 && (s == 1 || s <= (int)ng / 4); ++s) {
            if (s > 1 && tiles > 16 * sms) break;  // the last wave is a small part
            if (s > 8 && tiles > sms) break;       // partial sums' memory
            const double cost = (double)((tiles * s + sms - 1) / sms) * (1.0 / s + 0.02) + (s > 1 ? 0.02 : 0.0);
            if (cost < best) {
                best = cost;
                a.splits = s;
            }
        }
        if (a.splits > 1) {
            a.part = (float2*)scratch_buffer(c, 7, sizeof(float2) * total * a.splits);
            if (!a.part) a.splits = 1;  // no memory for partial sums: unsplit needs none
            grid.z = a.splits;
        }
    }
    const cudaError_t e = modes == 1 ? launch_triplet<1>(a, smem, tensor, grid, c->stream)
                                     : launch_triplet<2>(a, smem, tensor, grid, c->stream);
    if (e == cudaSuccess && a.splits > 1) {
        triplet_join_kernel<<<(unsigned)std::min<size_t>((total + 255) / 256, (size_t)sm_count() * 8), 256, 0, c->stream>>>(a, total);
        count_launch();
        return cuda_check(c, cudaGetLastError(), "triplet join");
    }
    return cuda_check(c, e, "triplet");
}

namespace {
focss_status run_triplet(Ctx* c, const Field* in, const Field* rx, int radius, int n_terms, const int32_t* m,
                         const int32_t* n, const double* coef, float2 inv_lw, Field* out) {
    return run_triplet_rows(c, in->d, (size_t)in->modes * in->samples, in->modes, in->samples, in->batch,
                            rx ? rx->d : nullptr, radius, n_terms, m, n, coef, inv_lw, out->d);
}
}  // namespace
}  // namespace fg

extern "C" {

FOCSS_API focss_status focss_triplet_apply(focss_ctx* c, const focss_field* in, int radius, int n_terms,
                                           const int32_t* m, const int32_t* n, const double* coef,
                                           focss_field* out) {
    if (!c || !in || !out) return FOCSS_ERR_INVALID_ARG;
    if (in->modes != out->modes || in->samples != out->samples || in->batch != out->batch || in == out)
        return fg::set_error(c, FOCSS_ERR_INVALID_ARG, "triplet_apply: out must be a distinct field of the same shape");
    return fg::run_triplet(c, in, nullptr, radius, n_terms, m, n, coef, make_float2(1.f, 0.f), out);
}

FOCSS_API focss_status focss_sino_equalize(focss_ctx* c, const focss_field* rx, const focss_field* tx, int radius,
                                           int n_terms, const int32_t* m, const int32_t* n, const double* coef,
                                           double lw_re, double lw_im, focss_field* out) {
    if (!c || !rx || !tx || !out) return FOCSS_ERR_INVALID_ARG;
    if (rx->modes != tx->modes || rx->samples != tx->samples || rx->batch != tx->batch ||
        out->modes != rx->modes || out->samples != rx->samples || out->batch != rx->batch || out == tx)
        return fg::set_error(c, FOCSS_ERR_INVALID_ARG, "sino_equalize: shapes");
    const double den = lw_re * lw_re + lw_im * lw_im;
    if (!(den > 0)) return fg::set_error(c, FOCSS_ERR_INVALID_ARG, "sino_equalize: linear weight is zero");
    const float2 inv = make_float2((float)(lw_re / den), (float)(-lw_im / den));
    return fg::run_triplet(c, tx, rx, radius, n_terms, m, n, coef, inv, out);
}

}  // extern "C"
