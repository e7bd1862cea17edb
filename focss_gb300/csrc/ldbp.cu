// ldbp.cu -- learned digital back-propagation: forward and backward kernels.
//
// Model (per realization, field at 2 samples/symbol, N samples):
//   for each span s:   x *= span_scale                         (Amplifier::drop_power)
//     for each step i: x = FIR(x, h[s,i])                       (learned dispersion filter)
//                      x = x * exp(i xi[s,i] |x|^2)             (learned nonlinear gain)
//   y = FIR(x, h_mf);  symbols = y[0::2]                          (learned matched filter)
// FIR(x, h)[n] = sum_{t<T} h[t] x[(n + t - c) mod N], c = (T-1)/2 (circular).
// It replaces the many-step split-step DBP of backward_propagation
// (src/tasks/systems.cpp:73-91) with few learned steps per span; plain DBP is
// its initialisation, its fallback and the yardstick of its Q.
//
// Gradients use the Wirtinger convention g = dL/d(conj z) for complex values;
// for real parameters dL/dxi is returned.  Loss: L = mean_k |symbols_k - t_k|^2.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "fir_tc.cuh"
#include "internal.h"

namespace fg {

constexpr int FIR_MAX_TAPS = 255;

__device__ __forceinline__ int wrap_index(int s, int N) {
    if (s < 0 || s >= N) {
        s %= N;
        if (s < 0) s += N;
    }
    return s;
}

// ---------------------------------------------------------------- chains of layers
// A chain of up to kMaxChain layers, each y = FIR(x, h_l) gain_l and, with xi,
// x' = y exp(i xi_l |y|^2), in one launch.  A CTA takes `owned` samples of one
// realization through all of them: layer l's product (fir_tc.cuh) gives 2048
// outputs, of which the T - 1 at the end are no longer valid inputs' sums, so
// owned = 2048 - (layers - 1)(T - 1), and between layers the samples stay in
// shared memory (split FP16) and registers (FP32).
//
// The input of every layer is scaled by the tile's largest sample (precision:
// fir_tc.cuh).  Tiles in which a layer's input spans more than 2^12 in power
// (largest sample over the mean of the weakest run: of 32 samples of the chain's
// input, of a thread's 8 behind that) or holds samples that are not finite or
// beyond 1e15 run all layers in FP32, so that an overflow stays within the filters' reach.
// 20 x 4 steps of
// 63 taps: relative error of the symbols 1.1e-6 (1.4e-6 with plain FP32 filters).
//
// What bounds it: per tile and layer ~1040 cycles of shared-memory bandwidth
// for the products and ~1200 issue cycles for the epilogue (nonlinear phase,
// splits), with two CTAs per SM (tensor memory) to overlap them.  20 x 4 steps of 63 taps on
// 16 x 65536 samples: 1368 -> 514 us against one FP32 launch per layer.
constexpr int kMaxChain = 8;
struct ChainArgs {
    const float2* x;            // batch x N: samples, or (backward) the gradient
    float2* y;                  // batch x N, or batch x N/2 (decimate: even samples only)
    int dir;                    // layer l's data is at l dir strides: 1, or -1 backward
    float2* keep;               // forward, optional: y of a layer (before the phase); backward: the gradient there
    const float2* act;          // backward: the kept y of the layers
    size_t stride;              // of keep and act
    const unsigned char* bmat;  // Toeplitz matrices of the layers, ks * STEP_BYTES each
    const float* unscale;       // their scales
    const float2* h;            // taps, T per layer (tiles in FP32)
    const float* xi;            // gains of the nonlinear phase, or null
    float* gxi;                 // backward: their gradients (added to)
    float gain[kMaxChain];
    int layers, T, N, owned, decimate;
};

// Gradient through y e^{i phi}, phi = xi |y|^2, from g = dL/dconj of the output:
//   g_y = g e^{-i phi} (1 - i xi p) + conj(g) i xi y^2 e^{i phi},
//   dL/dxi += 2 Re(conj(g) i p y e^{i phi})
// `e` = e^{i phi}, p = |y|^2.
__device__ __forceinline__ float2 phase_grad(float2 g, float2 y, float p, float2 e, float k, float& gxi) {
    const float2 q = cmul(make_float2(g.x, -g.y), cmul(y, e)), b = cmul(q, y), ge = cmulc(g, e);
    const float kp = k * p;
    gxi = -2.f * p * q.y;
    return make_float2(fmaf(-k, b.y, fmaf(kp, ge.y, ge.x)), fmaf(k, b.x, fmaf(-kp, ge.x, ge.y)));
}

// Whether powers of largest value `mx` leave the split's range (infinity and all
// above 1e30 do), `mn` the smallest non-zero sum over a run of `run` samples (both as bits).
__device__ __forceinline__ bool outside_split(unsigned mx, unsigned mn, int run) {
    const float pmax = __uint_as_float(mx);
    return pmax > 0.f && (!(pmax > 1e-36f && pmax <= 1e30f) || pmax > (float)(4096 / run) * __uint_as_float(mn));
}

// The CTA's owned samples of a layer's output `v(i)`, i = 0 .. owned-1, to dst.
template <class V>
__device__ __forceinline__ void chain_store(const ChainArgs& a, float2* dst, int b, int n0, bool last, V v) {
    for (int i = threadIdx.x; i < a.owned; i += firtc::THREADS) {
        const int n = n0 + i;
        if (n >= a.N) break;
        if (last && a.decimate) {
            if (!(n & 1)) dst[(size_t)b * (a.N / 2) + n / 2] = v(i);
        } else {
            dst[(size_t)b * a.N + n] = v(i);
        }
    }
}

// The layers of one tile in FP32 on plain shared-memory buffers.  A thread owns 8
// consecutive outputs and slides a register window along the taps, so that one
// shared load feeds 8 complex multiply-adds (index j at pad8(j): conflict-free).
// 20 x 4 steps of 63 taps on 16 x 65536 samples, every tile out of range: 1.6 ms, 3.0
// with a load for each of them, 1.4 in one FP32 filter launch per layer.
__host__ __device__ constexpr int pad8(int j) { return j + (j >> 3); }
constexpr int kPlainBuf = pad8(firtc::TILE + FIR_MAX_TAPS + 1 + 8);  // windows read up to 8 beyond the last tap
template <bool BWD>
__device__ __noinline__ void chain_tile_fp32(const ChainArgs& a, float2* buf, int b, int n0) {
    const int c = (a.T - 1) / 2, i0 = firtc::OUT * threadIdx.x;
    static_assert(firtc::OUT == 8 && firtc::OUT * firtc::THREADS == firtc::TILE, "8 outputs a thread");
    float2 *cur = buf, *nxt = buf + kPlainBuf;
    int valid = a.owned + a.layers * (a.T - 1);
    const size_t row = (size_t)b * a.N;
    __syncthreads();
    for (int i = threadIdx.x; i < valid; i += firtc::THREADS) cur[pad8(i)] = a.x[row + wrap_index(n0 - a.layers * c + i, a.N)];
    for (int l = 0; l < a.layers; ++l) {
        const ptrdiff_t at = (ptrdiff_t)a.dir * l;
        const float2* h = a.h + at * a.T;
        __syncthreads();
        if (BWD && a.xi) {
            const int first = (a.layers - l) * c;
            float acc = 0.f;
            for (int i = threadIdx.x; i < valid; i += firtc::THREADS) {
                const int n = n0 + i - first;
                const float2 y = a.act[at * (ptrdiff_t)a.stride + row + wrap_index(n, a.N)];
                const float p = cnorm(y), k = a.xi[at];
                float d;
                const float2 g = phase_grad(cur[pad8(i)], y, p, phase_rotation(k * p), k, d);
                cur[pad8(i)] = g;
                if (i >= first && i < first + a.owned && n < a.N) {
                    a.keep[at * (ptrdiff_t)a.stride + row + n] = g;
                    acc += d;
                }
            }
            acc = warp_sum(acc);
            if ((threadIdx.x & 31) == 0) atomicAdd(a.gxi + at, acc);
            __syncthreads();
        }
        const int first = (a.layers - 1 - l) * c;
        valid -= a.T - 1;
        if (i0 < valid) {
            float2 s[8], w[16];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                s[r] = make_float2(0.f, 0.f);
                w[r] = cur[pad8(i0 + r)];
            }
            auto tap = [&](int t) { return BWD ? make_float2(h[a.T - 1 - t].x, -h[a.T - 1 - t].y) : h[t]; };
            auto add = [&](float2 hv, const float2* x) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    s[r].x = fmaf(hv.x, x[r].x, fmaf(-hv.y, x[r].y, s[r].x));
                    s[r].y = fmaf(hv.x, x[r].y, fmaf(hv.y, x[r].x, s[r].y));
                }
            };
            int t = 0;
            for (; t + 8 <= a.T; t += 8) {
                float2 hv[8];
#pragma unroll
                for (int d = 0; d < 8; ++d) hv[d] = tap(t + d);
#pragma unroll
                for (int r = 0; r < 8; ++r) w[8 + r] = cur[pad8(i0 + t + 8 + r)];
#pragma unroll
                for (int d = 0; d < 8; ++d) add(hv[d], w + d);
#pragma unroll
                for (int r = 0; r < 8; ++r) w[r] = w[8 + r];
            }
            for (; t < a.T; ++t) {  // no zero taps: a sample there may be NaN
                add(tap(t), w);
#pragma unroll
                for (int r = 0; r < 7; ++r) w[r] = w[r + 1];
                w[7] = cur[pad8(i0 + t + 8)];
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int i = i0 + r;
                if (i >= valid) break;
                float2 y = cscale(s[r], a.gain[l]);
                if (!BWD) {
                    const int n = n0 + i - first;
                    if (a.keep && i >= first && i < first + a.owned && n < a.N) a.keep[at * (ptrdiff_t)a.stride + row + n] = y;
                    if (a.xi) y = cmul(y, phase_rotation(a.xi[at] * cnorm(y)));
                }
                nxt[pad8(i)] = y;
            }
        }
        __syncthreads();
        float2* t = cur;
        cur = nxt;
        nxt = t;
    }
    chain_store(a, a.y, b, n0, true, [&](int i) { return cur[pad8(i)]; });
}

// BWD: the same chain run backwards on gradients -- per layer the gradient
// through the phase (kept for the tap gradients, and summed for the gain's),
// then the adjoint filter times the gain.  `dir` is then -1 and the matrices
// are the adjoint filters'.
template <bool BWD>
__global__ void __launch_bounds__(firtc::THREADS, 2) ldbp_chain_kernel(const ChainArgs a) {
    using namespace firtc;
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) unsigned long long done, bfull[2];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    // largest |.|^2 and weakest run: of the chain's input, of the filters' inputs
    __shared__ unsigned s_in, s_min_in, s_max[kMaxChain], s_min[kMaxChain];
    __shared__ float s_gxi[kMaxChain];
    __shared__ int s_bad;
    const int ks = ksteps(a.T), cap = qcap(ks), c = (a.T - 1) / 2;
    const uint32_t pitch = 2u * cap, bbytes = STEP_BYTES * ks;
    unsigned char* xs = sm + ((1024u - (tcg::smem_addr(sm) & 1023u)) & 1023u);  // {re hi, im hi, re lo, im lo}
    unsigned char* bs = xs + 4 * (size_t)pitch;                                 // Toeplitz matrices, two for a chain
    float2* stage = reinterpret_cast<float2*>(bs + (a.layers > 1 ? 2 : 1) * (size_t)bbytes);  // CAP_MAX samples, padded
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.y, n0 = blockIdx.x * a.owned;
    const size_t row = (size_t)b * a.N;
    auto load_matrix = [&](int l) {
        tcg::mbar_expect_tx(&bfull[l & 1], bbytes);
        tcg::bulk_load(tcg::smem_addr(bs) + (l & 1) * bbytes, a.bmat + (ptrdiff_t)a.dir * l * (ptrdiff_t)bbytes, bbytes,
                       &bfull[l & 1]);
    };

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < kMaxChain; ++i) {
            s_max[i] = 0u;
            s_min[i] = 0x7F7FFFFFu;
            s_gxi[i] = 0.f;
        }
        s_in = 0u;
        s_min_in = 0x7F7FFFFFu;
        s_bad = 0;
        tcg::mbar_init(&done, 1);
        tcg::mbar_init(&bfull[0], 1);
        tcg::mbar_init(&bfull[1], 1);
        tcg::fence_mbar_init();
    }
    if (warp == 0) tcg::tmem_alloc(&tmem_base, D_COLS);
    pdl_wait();  // nothing in global memory is touched before the launches it depends on are done
    __syncthreads();
    if (threadIdx.x == 0)
        for (int l = 0; l < 2 && l < a.layers; ++l) load_matrix(l);
    // input: element e of the tile is sample n0 - layers c + e, coalesced into
    // the staging buffer, then 8 consecutive per thread
    constexpr int LOADS = 2;  // 8 x 256 x 2 >= CAP_MAX
    constexpr int K = CAP_MAX / THREADS;
    static_assert(CAP_MAX % THREADS == 0 && CAP_MAX >= TILE + FIR_MAX_TAPS - 1 && CAP_MAX <= 8 * LOADS * THREADS, "tile");
    const int base = n0 - a.layers * c, len = TILE + a.T - 1;
    auto stage_in = [&](const float2* src, int first) {
        float2 t[K];
#pragma unroll
        for (int u = 0; u < K; ++u) {
            const int e = threadIdx.x + THREADS * u;
            t[u] = e < len ? src[wrap_index(first + e, a.N)] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < K; ++u) stage[pad(threadIdx.x + THREADS * u)] = t[u];
    };
    float2 v[LOADS][8];
    stage_in(a.x + row, base);
    __syncthreads();
    {
        float mx = 0.f, mn = 3.4e38f;
        bool bad = false;
#pragma unroll
        for (int u = 0; u < LOADS; ++u) {
            const int e0 = 8 * (threadIdx.x + THREADS * u);
            float sum = 0.f;  // 8 samples; four neighbouring lanes hold a run of 32
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[u][j] = e0 < CAP_MAX ? stage[pad(e0 + j)] : make_float2(0.f, 0.f);
                const float p = cnorm(v[u][j]);
                sum += p;
                mx = fmaxf(mx, p);
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            bad = bad || !(sum <= 1e30f);
            if (sum > 0.f) mn = fminf(mn, sum);
        }
        mx = warp_max(mx);
        mn = -warp_max(-mn);
        bad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            atomicMax(&s_in, __float_as_uint(mx));
            if (!BWD || !a.xi) atomicMax(&s_max[0], __float_as_uint(mx));
            atomicMin(&s_min_in, __float_as_uint(mn));
            if (bad) s_bad = 1;
        }
    }
    tcg::fence_before_sync();
    __syncthreads();
    tcg::fence_after_sync();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    bool plain = s_bad || outside_split(s_in, s_min_in, 32);  // the layers run in FP32
    // Largest power and a run of 8 (its sum; whether all of it is valid input) of layer l's filter
    // input; a run beyond 1e30 or not a number counts as infinite.
    auto note_range = [&](int l, float mx, float sum, bool valid) {
        if (valid && !(sum <= 1e30f)) mx = __int_as_float(0x7F800000);
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        const unsigned n = __reduce_min_sync(0xffffffffu, valid && sum > 0.f ? __float_as_uint(sum) : 0x7F7FFFFFu);
        if (lane == 0) {
            atomicMax(&s_max[l], m);
            atomicMin(&s_min[l], n);
        }
    };
    const int o0 = ROW * (32 * (warp & 3) + lane) + OUT * (warp >> 2);  // first output of the thread
    // Backward, before a layer's filter: the gradient through the phase of the
    // thread's 8 samples at tile elements e0 .. (layer l, its y in the staging
    // buffer), with the gain's gradient over the owned samples.
    auto grad8 = [&](float2 (&g)[8], int e0, int l, float& mx, float& sum) {
        const float k = a.xi[(ptrdiff_t)a.dir * l];
        const int first = (a.layers - l) * c, left = min(a.owned, a.N - n0);
        float2 y[8];
        float p[8], d[8], pm = 0.f, acc = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            y[j] = stage[pad(e0 + j)];
            p[j] = cnorm(y[j]);
            pm = fmaxf(pm, p[j]);
        }
        if (fabsf(k) * pm <= kPhaseSmall) {
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = phase_grad(g[j], y[j], p[j], phase_rotation_small(k * p[j]), k, d[j]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = phase_grad(g[j], y[j], p[j], phase_rotation(k * p[j]), k, d[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = e0 + j - first;
            if (i >= 0 && i < left) acc += d[j];
            const float q = cnorm(g[j]);
            sum += q;
            mx = fmaxf(mx, q);
        }
        return acc;
    };
    if (BWD && a.xi && !plain) {
        stage_in(a.act + row, base);
        __syncthreads();
        float acc = 0.f;
#pragma unroll
        for (int u = 0; u < LOADS; ++u) {
            const int e0 = 8 * (threadIdx.x + THREADS * u);
            float mx = 0.f, sum = 0.f;
            if (e0 < CAP_MAX) acc += grad8(v[u], e0, 0, mx, sum);
            note_range(0, mx, sum, e0 + 8 <= len);
        }
        acc = warp_sum(acc);
        if (lane == 0) atomicAdd(&s_gxi[0], acc);
        __syncthreads();
        plain = outside_split(s_max[0], s_min[0], 8);
    }
    if (BWD && a.xi && !plain) {
#pragma unroll
        for (int u = 0; u < LOADS; ++u) {
            const int e0 = 8 * (threadIdx.x + THREADS * u);
            if (e0 < CAP_MAX)
#pragma unroll
                for (int j = 0; j < 8; ++j) stage[pad(e0 + j)] = v[u][j];
        }
        __syncthreads();
        chain_store(a, a.keep, b, n0, false, [&](int i) { return stage[pad(a.layers * c + i)]; });
    }
    if (!plain) {
        const float sc = pow2(-split_exponent(s_max[0]));
#pragma unroll
        for (int u = 0; u < LOADS; ++u) {
            const int e = 8 * (threadIdx.x + THREADS * u);
            if (e < cap) split_store8(xs, pitch, e, v[u], sc);
        }
    }
    int next = 0;  // the first layer that has not run
    for (int l = 0; l < a.layers && !plain; ++l) {
        const bool last = l + 1 == a.layers;
        tcg::fence_async_smem();
        tcg::fence_before_sync();
        __syncthreads();  // the split input is in place, the accumulator read
        if (warp == 0) {
            tcg::fence_after_sync();
            ok = tcg::mbar_wait_warp(&bfull[l & 1], (l >> 1) & 1, &abort_flag);
            if (ok) issue(tmem, tcg::smem_addr(xs), pitch, tcg::smem_addr(bs) + (l & 1) * bbytes, ks, &done);
        }
        // backward: the next layer's y, in flight while the product runs
        float2 ny[BWD ? TILE / THREADS : 1];
        if (BWD && !last) {
            const float2* src = a.act + (ptrdiff_t)a.dir * (l + 1) * (ptrdiff_t)a.stride + row;
#pragma unroll
            for (int u = 0; u < TILE / THREADS; ++u)
                ny[u] = src[wrap_index(base + (l + 1) * c + threadIdx.x + THREADS * u, a.N)];
        }
        ok = ok && tcg::mbar_wait(&done, l & 1, &abort_flag);
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        tcg::fence_after_sync();
        if (threadIdx.x == 0 && l + 2 < a.layers) load_matrix(l + 2);
        float2 y[OUT];
        read_outputs(tmem, warp, pow2(split_exponent(s_max[l])) * a.unscale[(ptrdiff_t)a.dir * l] * a.gain[l], y);
        const int first = (a.layers - 1 - l) * c;  // first owned output
        float mx = 0.f, sum = 0.f;  // powers of the next filter's input
        if (BWD) {
            if (!last) {
#pragma unroll
                for (int u = 0; u < TILE / THREADS; ++u) stage[pad(threadIdx.x + THREADS * u)] = ny[u];
                __syncthreads();
                const float acc = warp_sum(grad8(y, o0, l + 1, mx, sum));
                if (lane == 0) atomicAdd(&s_gxi[l + 1], acc);
                __syncthreads();
            }
        } else {
            if (a.keep) {
#pragma unroll
                for (int r = 0; r < OUT; ++r) stage[pad(o0 + r)] = y[r];
                __syncthreads();
                chain_store(a, a.keep + (ptrdiff_t)a.dir * l * (ptrdiff_t)a.stride, b, n0, false,
                            [&](int i) { return stage[pad(first + i)]; });
            }
            // the phase keeps |y|, whose largest value scales the next layer's input
            float pw[OUT];
#pragma unroll
            for (int r = 0; r < OUT; ++r) {
                pw[r] = cnorm(y[r]);
                sum += pw[r];
                mx = fmaxf(mx, pw[r]);
            }
            if (a.xi) {
                const float k = a.xi[(ptrdiff_t)a.dir * l];
                if (fabsf(k) * mx <= kPhaseSmall) {
#pragma unroll
                    for (int r = 0; r < OUT; ++r) y[r] = cmul(y[r], phase_rotation_small(k * pw[r]));
                } else {
#pragma unroll
                    for (int r = 0; r < OUT; ++r) y[r] = cmul(y[r], phase_rotation(k * pw[r]));
                }
            }
        }
        if (!last) note_range(l + 1, mx, sum, o0 + OUT <= a.owned + first * 2);
        if (last || BWD) {
            // staged: the result, or backward the gradient behind the next phase
            if (a.keep && !BWD) __syncthreads();
#pragma unroll
            for (int r = 0; r < OUT; ++r) stage[pad(o0 + r)] = y[r];
            __syncthreads();
            if (last) {
                chain_store(a, a.y, b, n0, true, [&](int i) { return stage[pad(i)]; });
                break;
            }
            chain_store(a, a.keep + (ptrdiff_t)a.dir * (l + 1) * (ptrdiff_t)a.stride, b, n0, false,
                        [&](int i) { return stage[pad(first + i)]; });
        }
        // the outputs are the next layer's inputs at the same places; the
        // elements behind them (no longer valid) become zero
        if (l == 0)
            for (int e = TILE / 8 + threadIdx.x; e < cap / 8; e += THREADS) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<uint4*>(xs + q * pitch + swz32(16u * e)) = make_uint4(0u, 0u, 0u, 0u);
            }
        __syncthreads();
        next = l + 1;
        plain = outside_split(s_max[next], s_min[next], 8);
        if (!plain) split_store8(xs, pitch, o0, y, pow2(-split_exponent(s_max[next])));
    }
    if (plain) {
        // the matrices on their way land before their buffers are reused
        for (int k = next; k < min(next + 2, a.layers); ++k) ok = tcg::mbar_wait(&bfull[k & 1], (k >> 1) & 1, &abort_flag) && ok;
        tcg::fence_before_sync();
        ok = !__syncthreads_or(!ok);
        tcg::fence_after_sync();
        if (ok) {
            chain_tile_fp32<BWD>(a, reinterpret_cast<float2*>(sm), b, n0);
            if (warp == 0) tcg::tmem_free(tmem, D_COLS);
            return;
        }
    }
    if (!ok) {
        // a wait ran out: the copies and MMAs in flight land (bounded) before
        // the CTA leaves, and its outputs are marked invalid
        if (warp == 0) {
            tcg::mma_commit_warp(&done);
            for (int p = 0; p < 2; ++p) tcg::mbar_wait_warp(&done, p, nullptr);
            for (int p = 0; p < 2; ++p) {
                tcg::mbar_wait_warp(&bfull[0], p, nullptr);
                if (a.layers > 1) tcg::mbar_wait_warp(&bfull[1], p, nullptr);
            }
        }
        __syncthreads();
        const float nan = __int_as_float(0x7fc00000);
        chain_store(a, a.y, b, n0, true, [&](int) { return make_float2(nan, nan); });
        if (threadIdx.x < a.layers) s_gxi[threadIdx.x] = nan;
    }
    pdl_trigger();
    if (BWD && a.xi && threadIdx.x < a.layers) atomicAdd(a.gxi + (ptrdiff_t)a.dir * (int)threadIdx.x, s_gxi[threadIdx.x]);
    tcg::fence_before_sync();
    __syncthreads();
    tcg::fence_after_sync();
    if (warp == 0) tcg::tmem_free(tmem, D_COLS);
}

// ---------------------------------------------------------------- tap gradients
// Of the layers first .. first + gridDim.z - 1 in one launch:
//   g_h[t] += scale sum_n g_y[n] conj(x[(n + t - c) mod N]) over all realizations,
// x = the input for layer 0, else the phase of layer k - 1 applied to its kept
// y again, scale = span_scale in the first layer of a span.
//
// On the tensor cores: with the window w[i] = x[n0 - c + i] and n = n0 + 32 b + r,
//   D[m][r] = sum_b w[32 b + m] g_y[32 b + r],  g_h[t] = sum_r D[t + r][r],
// a product over the 64 blocks b of a 2048-sample tile whose operands are the
// plain arrays w and g_y: element (k = b, m) of an MN-major operand with 64-byte
// rows lies 32 k + m elements from the start, so the Hankel matrix is w itself
// with its 32-element groups along M 64 bytes apart.  M = 128 takes filters of
// up to 97 taps; longer ones take further CTAs (blockIdx.y) 128 samples on.
// Both are split in two FP16 words, the leading ones multiples of 2^-11 (their
// products add up exactly while a sum stays below 4, and truncate by at most
// 2^-19 of the largest product there could be beyond); the columns are
//   (Re w: E0 E1 | Im w: E0 E1) x g re/im x 32,
// E0 = w_hi g_hi and E1 = 2^11 (w_hi g_lo + w_lo g_hi).  Per tile the result is
// rescaled and added to FP32 registers, once per CTA along the diagonals.
// Tiles whose power spans more than 2^10 (largest sample over the weakest
// run of 32's largest) or holds non-finite samples sum in FP32.
//
// What bounds it: issue (~1150 instructions per warp and tile: loads, phase,
// splits, the way back), with the tensor core working on the tile before and
// two CTAs per SM (tensor memory).  With the backward chains' shorter phase
// gradient, loss and gradients of 20 x 4 steps of 63 taps on 16 x 65536 samples
// took 3167 us with FP32 sums of 8 taps x 8 samples per thread (of which these
// 1540), 2122 us so.
struct TapGrad {
    const float2* x0;    // batch x N: the input of layer 0
    const float2* act;   // kept y of all layers, `stride` apart
    const float2* gy;    // gradients of y, from layer `first` on, `stride` apart
    size_t stride;
    const float* xi;     // gains of all layers
    float2* gh;          // T per layer, from layer `first` on
    float span_scale;
    int first, steps, T, N;
    int tiles, chunk;    // tiles in all (tiles per realization x batch), and per CTA
};
namespace tapgrad {
constexpr int TILE = 2048, W = 32, M = 128, THREADS = 256;
constexpr int WIN = TILE - W + M;                    // window elements: 63 x 32 + 128
constexpr int XK = (WIN + THREADS - 1) / THREADS, GK = TILE / THREADS;
constexpr uint32_t XP = 4608, GP = 4096;             // bytes between the words of w, of g_y (multiples of 512)
constexpr int RP = W + 1;                            // pitch of the matrix summed along its diagonals
constexpr uint32_t BUF = 4 * XP + 4 * GP;            // one tile's words; two tiles
constexpr size_t SMEM = 2 * (size_t)BUF + 1024;
constexpr uint32_t D_COLS = 256;
static_assert(2 * WIN <= XP && 2 * TILE <= GP && XP % 512 == 0 && GP % 512 == 0, "words");
static_assert(BUF % 512 == 0 && sizeof(float2) * M * RP <= BUF && sizeof(float2) * (TILE + WIN) <= BUF, "reuse");
// kind::f16, FP32 accumulator, FP16 operands, both MN-major
__host__ __device__ constexpr uint32_t idesc(int n) {
    return (1u << 4) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// One scaled sample as {re hi, im hi, re lo, im lo} at element e, words `pitch` apart.
__device__ __forceinline__ void store(unsigned char* p, uint32_t pitch, int e, float2 v, float sc) {
    const float re = v.x * sc, im = v.y * sc;
    const float rf = (re + 6144.f) - 6144.f, jf = (im + 6144.f) - 6144.f;  // multiples of 2^-11
    const uint32_t o = 2u * (uint32_t)e;
    p += o ^ ((o >> 3) & 0x30u);
    *reinterpret_cast<__half*>(p) = __float2half_rn(rf);
    *reinterpret_cast<__half*>(p + pitch) = __float2half_rn(jf);
    *reinterpret_cast<__half*>(p + 2 * pitch) = __float2half_rn((re - rf) * 2048.f);
    *reinterpret_cast<__half*>(p + 3 * pitch) = __float2half_rn((im - jf) * 2048.f);
}
// One tile in FP32 on plain buffers: the same share of the sums as the CTA's
// product has.  Tap t = off + d takes the sample pairs whose window offset d + r
// (r = sample mod 32, here the lane) lies in this CTA's 0 .. 127; what a filter of
// more than 97 taps has beyond is the share of the CTAs next to it, which may
// find the same tile within the split's range (their windows differ).
__device__ __noinline__ void tile_fp32(float2* buf, const float2* x, const float2* gy, const float* xi, float2* gh,
                                       float scale, int n0, int off, int T, int N) {
    float2 *w = buf, *g = buf + WIN;
    const int c = (T - 1) / 2, lane = threadIdx.x & 31;
    __syncthreads();
    for (int i = threadIdx.x; i < WIN; i += THREADS) {
        const float2 v = x[wrap_index(n0 - c + off + i, N)];
        w[i] = xi ? cmul(v, phase_rotation(*xi * cnorm(v))) : v;
    }
    for (int i = threadIdx.x; i < TILE; i += THREADS) g[i] = n0 + i < N ? gy[n0 + i] : make_float2(0.f, 0.f);
    __syncthreads();
    for (int d = (int)(threadIdx.x >> 5) - (W - 1); d < M && off + d < T; d += THREADS / 32) {
        if (off + d < 0) continue;
        float2 acc = make_float2(0.f, 0.f);
        if (d + lane >= 0 && d + lane < M)
            for (int i = lane; i < TILE; i += W) acc = cadd(acc, cmulc(g[i], w[i + d]));
        acc.x = warp_sum(acc.x) * scale;
        acc.y = warp_sum(acc.y) * scale;
        if (lane == 0) {
            atomicAdd(&gh[off + d].x, acc.x);
            atomicAdd(&gh[off + d].y, acc.y);
        }
    }
    __syncthreads();
}
}  // namespace tapgrad

__global__ void __launch_bounds__(tapgrad::THREADS, 2) tap_grad_kernel(const TapGrad p) {
    using namespace tapgrad;
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) unsigned long long done;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ unsigned s_max[2][2], s_min[2][2];  // of w, g_y; by the tile's parity
    unsigned char* xs = sm + ((1024u - (tcg::smem_addr(sm) & 1023u)) & 1023u);
    const int N = p.N, T = p.T, off = M * blockIdx.y, c = (T - 1) / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = p.first + blockIdx.z;
    const float2* x = k ? p.act + (size_t)(k - 1) * p.stride : p.x0;
    const float* xi = k ? p.xi + (k - 1) : nullptr;
    const float2* gy = p.gy + (size_t)blockIdx.z * p.stride;
    float2* gh = p.gh + (size_t)blockIdx.z * T;
    const float scale = k % p.steps == 0 ? p.span_scale : 1.0f;
    const int per_row = (N + TILE - 1) / TILE;
    const int q0 = blockIdx.x * p.chunk, q1 = min(q0 + p.chunk, p.tiles);

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < 2; ++i)
            for (int j = 0; j < 2; ++j) {
                s_max[i][j] = 0u;
                s_min[i][j] = 0xFFFFFFFFu;
            }
        tcg::mbar_init(&done, 1);
        tcg::fence_mbar_init();
    }
    if (warp == 0) tcg::tmem_alloc(&tmem_base, D_COLS);
    float2 xr[XK], gr[GK];
    auto load = [&](int q) {
        const int b = q / per_row, n0 = (q - b * per_row) * TILE, w0 = n0 - c + off;
        const float2* xb = x + (size_t)b * N;
        const float2* gb = gy + (size_t)b * N;
        if (w0 >= 0 && w0 + WIN <= N && n0 + TILE <= N) {
#pragma unroll
            for (int u = 0; u < XK; ++u) {
                const int e = threadIdx.x + THREADS * u;
                xr[u] = e < WIN ? xb[w0 + e] : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < GK; ++u) gr[u] = gb[n0 + threadIdx.x + THREADS * u];
        } else {
#pragma unroll
            for (int u = 0; u < XK; ++u) {
                const int e = threadIdx.x + THREADS * u;
                xr[u] = e < WIN ? xb[wrap_index(w0 + e, N)] : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < GK; ++u) {
                const int n = n0 + threadIdx.x + THREADS * u;
                gr[u] = n < N ? gb[n] : make_float2(0.f, 0.f);
            }
        }
    };
    load(q0);
    tcg::fence_before_sync();
    __syncthreads();
    tcg::fence_after_sync();
    const uint32_t tmem = tmem_base;
    float2 acc[W / 2];
#pragma unroll
    for (int r = 0; r < W / 2; ++r) acc[r] = make_float2(0.f, 0.f);
    bool ok = true, pending = false;  // pending: the last tile's product
    uint32_t parity = 0;
    float back = 1.f;                 // its scale
    // a tile is split while the tensor core is on the one before
    for (int q = q0; q <= q1; ++q) {
        const int z = (q - q0) & 1;
        unsigned char* buf = xs + z * BUF;
        float sc[2], scale_back = 1.f;
        bool wide = false;
        if (q < q1) {
            if (xi) {
                const float g = *xi;
                float mx = 0.f;
#pragma unroll
                for (int u = 0; u < XK; ++u) mx = fmaxf(mx, cnorm(xr[u]));
                if (fabsf(g) * mx <= kPhaseSmall) {
#pragma unroll
                    for (int u = 0; u < XK; ++u) xr[u] = cmul(xr[u], phase_rotation_small(g * cnorm(xr[u])));
                } else {
#pragma unroll
                    for (int u = 0; u < XK; ++u) xr[u] = cmul(xr[u], phase_rotation(g * cnorm(xr[u])));
                }
            }
            // a warp's 32 samples are one run; non-negative floats order as integers, NaN above infinity
            unsigned mx[2] = {0u, 0u}, mn[2] = {0xFFFFFFFFu, 0xFFFFFFFFu};
#pragma unroll
            for (int u = 0; u < XK; ++u) {
                const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(cnorm(xr[u])) & 0x7FFFFFFFu);
                mx[0] = max(mx[0], m);
                if (m) mn[0] = min(mn[0], m);
            }
#pragma unroll
            for (int u = 0; u < GK; ++u) {
                const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(cnorm(gr[u])) & 0x7FFFFFFFu);
                mx[1] = max(mx[1], m);
                if (m) mn[1] = min(mn[1], m);
            }
            if (lane < 2) {
                atomicMax(&s_max[z][lane], lane ? mx[1] : mx[0]);
                atomicMin(&s_min[z][lane], lane ? mn[1] : mn[0]);
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned m = s_max[z][i];
                const float pmax = __uint_as_float(m), pmin = __uint_as_float(s_min[z][i]);
                wide = wide || !(pmax <= 1e30f) || (m && (!(pmax > 1e-36f) || pmax > 1024.f * pmin));
                const int e = firtc::split_exponent(m);
                sc[i] = firtc::pow2(-e);
                scale_back *= firtc::pow2(e);
            }
            if (wide) {
                const int b = q / per_row;
                tile_fp32(reinterpret_cast<float2*>(buf), x + (size_t)b * N, gy + (size_t)b * N, xi, gh, scale,
                          (q - b * per_row) * TILE, off, T, N);
            } else {
#pragma unroll
                for (int u = 0; u < XK; ++u) {
                    const int e = threadIdx.x + THREADS * u;
                    if (e < WIN) store(buf, XP, e, xr[u], sc[0]);
                }
#pragma unroll
                for (int u = 0; u < GK; ++u) store(buf + 4 * XP, GP, threadIdx.x + THREADS * u, gr[u], sc[1]);
            }
            if (q + 1 < q1) load(q + 1);
        }
        if (pending) {
            ok = tcg::mbar_wait(&done, parity, &abort_flag);
            parity ^= 1;
            tcg::fence_after_sync();
            const uint32_t t = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 16 * (uint32_t)(warp >> 2);
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // (w re/im, g re/im)
                const uint32_t col = t + 128 * (i >> 1) + 32 * (i & 1);
                uint32_t e0[16], e1[16];
                tcg::ld_x16_async(col, e0);
                tcg::ld_x16_async(col + 64, e1);
                tcg::wait_ld(e0);
                tcg::wait_ld(e1);
                const float f = i == 2 ? -back : back;
#pragma unroll
                for (int r = 0; r < W / 2; ++r) {
                    const float v = fmaf(__uint_as_float(e1[r]), 0x1p-11f, __uint_as_float(e0[r]));
                    if (i == 0 || i == 3)
                        acc[r].x = fmaf(v, f, acc[r].x);
                    else
                        acc[r].y = fmaf(v, f, acc[r].y);
                }
            }
        }
        tcg::fence_async_smem();
        tcg::fence_before_sync();
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        pending = q < q1 && !wide;
        back = scale_back;
        if (threadIdx.x < 2) {  // for the tile after the next; read before the barrier above
            s_max[z][threadIdx.x] = 0u;
            s_min[z][threadIdx.x] = 0xFFFFFFFFu;
        }
        if (pending && warp == 0) {
            tcg::fence_after_sync();
            uint64_t a = tcg::smem_desc_sw64_mn(tcg::smem_addr(buf), 2 * W);
            uint64_t g = tcg::smem_desc_sw64_mn(tcg::smem_addr(buf + 4 * XP), GP);
            for (int s = 0; s < TILE / W / 16; ++s) {
                tcg::mma_f16_warp(tmem, a, g, idesc(128), s != 0);
                tcg::mma_f16_warp(tmem + 128, a + XP / 16, g, idesc(128), s != 0);
                tcg::mma_f16_warp(tmem + 64, a + 2 * (XP / 16), g, idesc(64), true);
                tcg::mma_f16_warp(tmem + 192, a + 3 * (XP / 16), g, idesc(64), true);
                a += 1024 / 16;  // 16 blocks of 64 bytes
                g += 1024 / 16;
            }
            tcg::mma_commit_warp(&done);
        }
    }
    if (!ok && warp == 0) {  // a wait ran out: the MMAs in flight end (bounded) before the CTA leaves
        tcg::mma_commit_warp(&done);
        for (int i = 0; i < 2; ++i) tcg::mbar_wait_warp(&done, i, nullptr);
    }
    tcg::fence_before_sync();
    __syncthreads();
    tcg::fence_after_sync();
    if (warp == 0) tcg::tmem_free(tmem, D_COLS);
    float2* mat = reinterpret_cast<float2*>(xs);
#pragma unroll
    for (int r = 0; r < W / 2; ++r) mat[(32 * (warp & 3) + lane) * RP + (W / 2) * (warp >> 2) + r] = acc[r];
    __syncthreads();
    const int d = (int)threadIdx.x - (W - 1), t = off + d;  // m = d + r
    if (d < M && t >= 0 && t < T) {
        float2 s = make_float2(0.f, 0.f);
        for (int r = max(0, -d); r < min(W, M - d); ++r) s = cadd(s, mat[(d + r) * RP + r]);
        if (!ok) s.x = s.y = __int_as_float(0x7fc00000);
        atomicAdd(&gh[t].x, s.x * scale);
        atomicAdd(&gh[t].y, s.y * scale);
    }
}

// loss = mean |sym - t|^2 and the gradient at 2 samples/symbol (0 at odd samples).
__global__ void mse_kernel(const float2* __restrict__ sym, const float2* __restrict__ tx, size_t n_sym_total,
                           float inv_count, float4* __restrict__ gy, double* __restrict__ loss) {
    double acc = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_sym_total; i += (size_t)gridDim.x * blockDim.x) {
        const float2 d = csub(sym[i], tx[i]);
        gy[i] = make_float4(d.x * inv_count, d.y * inv_count, 0.f, 0.f);
        acc += (double)cnorm(d);
    }
    __shared__ double sd[32];
    acc = block_sum_d(acc, sd);
    if (threadIdx.x == 0) atomicAdd(loss, acc * inv_count);
}

// Adam on n real parameters (complex parameters as interleaved pairs; the
// real gradient of a complex z = a + ib is (2 Re g, 2 Im g)).  Parameters in
// [alt_lo, alt_hi) (the nonlinear gains) use the learning rate lr_alt.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m1,
                            float* __restrict__ m2, int n, float lr, float b1, float b2, float eps, float c1,
                            float c2, float gscale, int alt_lo, int alt_hi, float lr_alt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i] * gscale;
        const float a = b1 * m1[i] + (1.f - b1) * gi;
        const float v = b2 * m2[i] + (1.f - b2) * gi * gi;
        m1[i] = a;
        m2[i] = v;
        const float r = (i >= alt_lo && i < alt_hi) ? lr_alt : lr;
        p[i] -= r * (a * c1) / (sqrtf(v * c2) + eps);
    }
}

}  // namespace fg

// ---------------------------------------------------------------- model object
namespace {
struct LdbpModel {
    focss_ctx* ctx = nullptr;
    int spans = 0, steps = 0, taps = 0, mf_taps = 0, samples = 0, batch = 0;
    float span_scale = 1.f;
    int n_params = 0;        // real parameter count
    float* params = nullptr; // [h: spans*steps*taps*2][xi: spans*steps][hmf: mf_taps*2]
    float* grads = nullptr;
    float* m1 = nullptr;
    float* m2 = nullptr;
    int adam_t = 0;
    float2* acts = nullptr;  // per layer y, then per layer the gradient there, of batch*samples
    float2* work = nullptr;  // 2 work buffers of batch*samples
    float2* sym = nullptr;   // batch*samples/2
    double* loss = nullptr;
    unsigned char* bmat = nullptr;  // Toeplitz matrices of the layers, of the matched filter; the adjoints'
    float* unscale = nullptr;       // their scales
    size_t field_n() const { return (size_t)batch * samples; }
    float2* h(int k) const { return (float2*)params + (size_t)k * taps; }
    float* xi(int k) const { return params + (size_t)spans * steps * taps * 2 + k; }
    // the gain section is padded to an even count so the taps after it stay 8-byte aligned
    int xi_count() const { return (spans * steps + 1) & ~1; }
    float2* hmf() const { return (float2*)(params + (size_t)spans * steps * taps * 2 + xi_count()); }
    float2* gh(int k) const { return (float2*)grads + (size_t)k * taps; }
    float* gxi(int k) const { return grads + (size_t)spans * steps * taps * 2 + k; }
    float2* ghmf() const { return (float2*)(grads + (size_t)spans * steps * taps * 2 + xi_count()); }
};

inline int gridn(size_t n) {
    size_t g = (n + 255) / 256;
    return (int)std::max<size_t>(1, std::min<size_t>(g, (size_t)fg::sm_count() * 16));
}
}  // namespace

struct focss_ldbp : LdbpModel {};

using fg::count_launch;

static focss_status ldbp_err(focss_ctx* c, cudaError_t e, const char* what) { return fg::cuda_check(c, e, what); }

// Toeplitz matrices of the current parameters' filters, or of their adjoints.
static size_t layer_bytes(const LdbpModel& M) { return (size_t)fg::firtc::STEP_BYTES * fg::firtc::ksteps(M.taps); }
static size_t matrices_bytes(const LdbpModel& M) {
    return (size_t)M.spans * M.steps * layer_bytes(M) + (size_t)fg::firtc::STEP_BYTES * fg::firtc::ksteps(M.mf_taps);
}
static unsigned char* matrix(const LdbpModel& M, int k, int adjoint) {
    return M.bmat + adjoint * matrices_bytes(M) + k * layer_bytes(M);
}
static float* unscale(const LdbpModel& M, int k, int adjoint) { return M.unscale + adjoint * (M.spans * M.steps + 1) + k; }
// Queued behind every change of the parameters, so that they are current for
// whatever follows on the stream, in a replayed graph too.
static cudaError_t ldbp_matrices(const LdbpModel& M) {
    const int L = M.spans * M.steps;
    for (int adjoint = 0; adjoint < 2; ++adjoint) {
        fg::firtc::toeplitz_kernel<<<L + 1, 256, 0, M.ctx->stream>>>(M.h(0), M.taps, L, M.hmf(), M.mf_taps, adjoint,
                                                                    (__half*)matrix(M, 0, adjoint), unscale(M, 0, adjoint));
        count_launch();
    }
    return cudaGetLastError();
}

// layers per launch: the halo a chain computes twice stays below an eighth
static int chain_length(const LdbpModel& M) {
    return std::max(1, std::min(fg::kMaxChain, 1 + 256 / std::max(1, M.taps - 1)));
}

template <bool BWD>
static cudaError_t launch_chain(const LdbpModel& M, fg::ChainArgs& a) {
    using namespace fg::firtc;
    a.N = M.samples;
    a.dir = BWD ? -1 : 1;
    a.stride = M.field_n();
    a.owned = TILE - (a.layers - 1) * (a.T - 1);
    const int ks = ksteps(a.T);
    const size_t smem = 1024 + 8 * (size_t)qcap(ks) + (a.layers > 1 ? 2 : 1) * (size_t)STEP_BYTES * ks +
                        sizeof(float2) * pad(CAP_MAX);
    // a tile in FP32 takes two plain buffers instead
    const size_t need = std::max(smem, sizeof(float2) * 2 * (size_t)fg::kPlainBuf);
    cudaError_t e = cudaFuncSetAttribute(fg::ldbp_chain_kernel<BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
    if (e != cudaSuccess) return e;
    // programmatic serialization: the next chain's set-up runs while this one
    // ends (as launch_pass; 17 launches of 20 x 4 layers 551 -> 538 us)
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(M.ctx->stream, &cs);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((M.samples + a.owned - 1) / a.owned, M.batch);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = need;
    cfg.stream = M.ctx->stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = cs == cudaStreamCaptureStatusNone ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, fg::ldbp_chain_kernel<BWD>, (const fg::ChainArgs)a);
    count_launch();
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

// All learned steps from `in` (left in M.work), in chains; keep: every
// layer's FIR output (times the span's gain) in M.acts.  Then the matched
// filter's symbols (even samples) into `symbols`.
static cudaError_t ldbp_chains(LdbpModel& M, const float2* in, bool keep, float2* symbols) {
    const size_t n = M.field_n();
    const int L = M.spans * M.steps;
    cudaError_t e = cudaSuccess;
    float2* bufs[2] = {M.work, M.work + n};
    const int F = chain_length(M);
    const float2* src = in;
    int w = 0;
    for (int k = 0; k < L && e == cudaSuccess; k += F) {
        fg::ChainArgs a{};
        a.layers = std::min(F, L - k);
        a.T = M.taps;
        a.x = src;
        a.y = bufs[w];
        a.keep = keep ? M.acts + (size_t)k * n : nullptr;
        a.bmat = matrix(M, k, 0);
        a.unscale = unscale(M, k, 0);
        a.h = M.h(k);
        a.xi = M.xi(k);
        for (int l = 0; l < a.layers; ++l) a.gain[l] = (k + l) % M.steps == 0 ? M.span_scale : 1.0f;
        e = launch_chain<false>(M, a);
        src = bufs[w];
        w ^= 1;
    }
    if (e == cudaSuccess) {
        fg::ChainArgs a{};
        a.layers = 1;
        a.T = M.mf_taps;
        a.x = src;
        a.y = symbols;
        a.decimate = 1;
        a.bmat = matrix(M, L, 0);
        a.unscale = unscale(M, L, 0);
        a.h = M.hmf();
        a.gain[0] = 1.0f;
        e = launch_chain<false>(M, a);
    }
    return e;
}

static cudaError_t launch_tap_grad(const LdbpModel& M, fg::TapGrad& p, int layers) {
    using namespace fg::tapgrad;
    const size_t tiles = (size_t)((M.samples + TILE - 1) / TILE) * M.batch;
    if (tiles > 0x7FFFFFFFu) return cudaErrorInvalidValue;
    const unsigned blocks = (p.T + W - 1 + fg::tapgrad::M - 1) / fg::tapgrad::M;  // window offsets 0 .. T + 30
    p.tiles = (int)tiles;
    // tiles per CTA: the sum along the diagonals once per 16 tiles, fewer where
    // that leaves an SM without its two CTAs
    const size_t slots = 2 * (size_t)fg::sm_count();
    p.chunk = (int)std::min<size_t>(16, (tiles * layers * blocks + slots - 1) / slots);
    cudaError_t e = cudaFuncSetAttribute(fg::tap_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return e;
    fg::tap_grad_kernel<<<dim3((p.tiles + p.chunk - 1) / p.chunk, blocks, layers), THREADS, SMEM, M.ctx->stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

// Gradients of everything from gy, the gradient of the matched filter's output
// (in M.work): the adjoint chains, then the tap gradients from what they and
// the forward pass kept.
static cudaError_t ldbp_backward(LdbpModel& M, const float2* in) {
    const size_t n = M.field_n();
    const int L = M.spans * M.steps;
    float2* bufs[2] = {M.work, M.work + n};
    fg::TapGrad t{in, M.acts, M.work, n, M.xi(0), M.ghmf(), 1.0f, L, M.steps, M.mf_taps, M.samples, 0, 0};
    cudaError_t e = launch_tap_grad(M, t, 1);
    fg::ChainArgs m{};
    m.layers = 1;
    m.T = M.mf_taps;
    m.x = bufs[0];
    m.y = bufs[1];
    m.bmat = matrix(M, L, 1);
    m.unscale = unscale(M, L, 1);
    m.h = M.hmf();
    m.gain[0] = 1.0f;
    if (e == cudaSuccess) e = launch_chain<true>(M, m);
    const int F = chain_length(M);
    int w = 1;
    for (int k = L - 1; k >= 0 && e == cudaSuccess; k -= F) {
        fg::ChainArgs a{};
        a.layers = std::min(F, k + 1);
        a.T = M.taps;
        a.x = bufs[w];
        a.y = bufs[w ^ 1];
        a.keep = M.acts + (size_t)(L + k) * n;
        a.act = M.acts + (size_t)k * n;
        a.bmat = matrix(M, k, 1);
        a.unscale = unscale(M, k, 1);
        a.h = M.h(k);
        a.xi = M.xi(k);
        a.gxi = M.gxi(k);
        for (int l = 0; l < a.layers; ++l) a.gain[l] = (k - l) % M.steps == 0 ? M.span_scale : 1.0f;
        e = launch_chain<true>(M, a);
        w ^= 1;
    }
    // gridDim.z is at most 65535
    for (int k = 0; k < L && e == cudaSuccess; k += 32768) {
        fg::TapGrad a{in, M.acts, M.acts + (size_t)(L + k) * n, n, M.xi(0), M.gh(k), M.span_scale, k, M.steps, M.taps, M.samples, 0, 0};
        e = launch_tap_grad(M, a, std::min(L - k, 32768));
    }
    return e;
}

extern "C" {

FOCSS_API focss_status focss_ldbp_create(focss_ctx* c, int spans, int steps_per_span, int taps, int mf_taps,
                                         int samples, int batch, double span_scale, focss_ldbp** out) {
    if (!c || !out || spans <= 0 || steps_per_span <= 0 || taps <= 0 || mf_taps <= 0 || samples <= 0 || batch <= 0 ||
        samples % 2)
        return FOCSS_ERR_INVALID_ARG;
    if (taps % 2 == 0 || mf_taps % 2 == 0 || taps > fg::FIR_MAX_TAPS || mf_taps > fg::FIR_MAX_TAPS)
        return fg::set_error(c, FOCSS_ERR_INVALID_ARG, "ldbp: tap counts must be odd and <= 255");
    focss_ldbp* m = new (std::nothrow) focss_ldbp();
    if (!m) return FOCSS_ERR_OOM;
    m->ctx = c;
    m->spans = spans;
    m->steps = steps_per_span;
    m->taps = taps;
    m->mf_taps = mf_taps;
    m->samples = samples;
    m->batch = batch;
    m->span_scale = (float)span_scale;
    m->n_params = spans * steps_per_span * 2 * taps + m->xi_count() + 2 * mf_taps;
    const size_t n = m->field_n();
    const size_t n_acts = (size_t)2 * spans * steps_per_span;
    cudaError_t e = cudaMalloc(&m->params, sizeof(float) * 4 * (size_t)m->n_params);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->params, 0, sizeof(float) * 4 * (size_t)m->n_params, c->stream);
    m->grads = m->params + m->n_params;
    m->m1 = m->grads + m->n_params;
    m->m2 = m->m1 + m->n_params;
    if (e == cudaSuccess) e = cudaMalloc(&m->acts, sizeof(float2) * n * n_acts);
    if (e == cudaSuccess) e = cudaMalloc(&m->work, sizeof(float2) * n * 3);
    m->sym = m->work + 2 * n;
    if (e == cudaSuccess) e = cudaMalloc(&m->loss, sizeof(double) * 2);
    const size_t nl = (size_t)spans * steps_per_span;
    if (e == cudaSuccess)
        e = cudaMalloc(&m->bmat, 2 * matrices_bytes(*m));
    if (e == cudaSuccess) e = cudaMalloc(&m->unscale, sizeof(float) * 2 * (nl + 1));
    if (e == cudaSuccess) e = ldbp_matrices(*m);
    if (e != cudaSuccess) {
        cudaFree(m->params);
        cudaFree(m->acts);
        cudaFree(m->work);
        cudaFree(m->loss);
        cudaFree(m->bmat);
        cudaFree(m->unscale);
        delete m;
        return ldbp_err(c, e, "ldbp alloc");
    }
    *out = m;
    return FOCSS_OK;
}

FOCSS_API focss_status focss_ldbp_destroy(focss_ldbp* m) {
    if (!m) return FOCSS_OK;
    cudaStreamSynchronize(m->ctx->stream);
    cudaFree(m->params);
    cudaFree(m->acts);
    cudaFree(m->work);
    cudaFree(m->loss);
    cudaFree(m->bmat);
    cudaFree(m->unscale);
    delete m;
    return FOCSS_OK;
}

FOCSS_API int focss_ldbp_num_params(const focss_ldbp* m) { return m ? m->n_params : 0; }

FOCSS_API focss_status focss_ldbp_set_params(focss_ldbp* m, const float* host, int n) {
    if (!m || !host || n != m->n_params) return FOCSS_ERR_INVALID_ARG;
    cudaError_t e = cudaMemcpyAsync(m->params, host, sizeof(float) * n, cudaMemcpyHostToDevice, m->ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m1, 0, sizeof(float) * 2 * n, m->ctx->stream);
    if (e == cudaSuccess) e = ldbp_matrices(*m);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->ctx->stream);
    m->adam_t = 0;
    return ldbp_err(m->ctx, e, "ldbp set params");
}

FOCSS_API focss_status focss_ldbp_get_params(focss_ldbp* m, float* host, float* grads, int n) {
    if (!m || n != m->n_params) return FOCSS_ERR_INVALID_ARG;
    cudaError_t e = cudaSuccess;
    if (host) e = cudaMemcpyAsync(host, m->params, sizeof(float) * n, cudaMemcpyDeviceToHost, m->ctx->stream);
    if (grads && e == cudaSuccess)
        e = cudaMemcpyAsync(grads, m->grads, sizeof(float) * n, cudaMemcpyDeviceToHost, m->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->ctx->stream);
    return ldbp_err(m->ctx, e, "ldbp get params");
}

FOCSS_API focss_status focss_ldbp_forward(focss_ldbp* m, const focss_field* in, focss_field* symbols) {
    if (!m || !in || !symbols) return FOCSS_ERR_INVALID_ARG;
    if (in->modes != 1 || in->samples != m->samples || in->batch != m->batch || symbols->modes != 1 ||
        symbols->samples != m->samples / 2 || symbols->batch != m->batch)
        return fg::set_error(m->ctx, FOCSS_ERR_INVALID_ARG, "ldbp_forward: shapes");
    return ldbp_err(m->ctx, ldbp_chains(*m, in->d, false, symbols->d), "ldbp forward");
}

// One forward + backward over the batch: gradients into the model (overwritten),
// loss (mean |symbols - tx|^2) returned.
FOCSS_API focss_status focss_ldbp_loss_grad(focss_ldbp* m, const focss_field* in, const focss_field* tx,
                                            double* loss) {
    if (!m || !in || !tx) return FOCSS_ERR_INVALID_ARG;
    if (in->modes != 1 || in->samples != m->samples || in->batch != m->batch || tx->modes != 1 ||
        tx->samples != m->samples / 2 || tx->batch != m->batch)
        return fg::set_error(m->ctx, FOCSS_ERR_INVALID_ARG, "ldbp_loss_grad: shapes");
    cudaStream_t s = m->ctx->stream;
    const size_t ns = (size_t)m->batch * (m->samples / 2);
    cudaError_t e = ldbp_chains(*m, in->d, true, m->sym);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->grads, 0, sizeof(float) * m->n_params, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->loss, 0, sizeof(double), s);
    if (e == cudaSuccess) {
        fg::mse_kernel<<<gridn(ns), 256, 0, s>>>(m->sym, tx->d, ns, 1.f / (float)ns, (float4*)m->work, m->loss);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = ldbp_backward(*m, in->d);
    double h_loss = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_loss, m->loss, sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (loss) *loss = h_loss;
    return ldbp_err(m->ctx, e, "ldbp loss/grad");
}

FOCSS_API focss_status focss_ldbp_adam_step(focss_ldbp* m, double lr, double lr_gain, double beta1, double beta2,
                                            double eps) {
    if (!m) return FOCSS_ERR_INVALID_ARG;
    m->adam_t += 1;
    const float c1 = (float)(1.0 / (1.0 - std::pow(beta1, m->adam_t)));
    const float c2 = (float)(1.0 / (1.0 - std::pow(beta2, m->adam_t)));
    // complex gradients g = dL/dconj(z) -> real gradient 2 g; xi gradients are already real:
    // the factor 2 is applied uniformly (Adam is invariant to gradient scale).
    const int xi_lo = m->spans * m->steps * m->taps * 2;
    fg::adam_kernel<<<gridn(m->n_params), 256, 0, m->ctx->stream>>>(
        m->params, m->grads, m->m1, m->m2, m->n_params, (float)lr, (float)beta1, (float)beta2, (float)eps, c1, c2,
        1.f, xi_lo, xi_lo + m->spans * m->steps, (float)lr_gain);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = ldbp_matrices(*m);
    return ldbp_err(m->ctx, e, "ldbp adam");
}

}  // extern "C"
