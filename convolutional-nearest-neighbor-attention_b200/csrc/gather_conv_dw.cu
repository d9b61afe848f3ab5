// Depthwise gather + conv for any number of taps: o[m, c] = sum_j w[j, c] * p[m, j] * v[neighbour(m, j), c].
//
// Tokens m = (b, h, t) are dealt out flat, TT per CTA, so the grid follows the number of tokens and not the number of
// (batch, head) slices.  A CTA turns its tokens' values into weights once (exponentials by all threads, each token's
// sum in tap order by one), keeps (row offset, weight) pairs in shared memory, and then every thread works on one
// 16-byte channel group of TPT tokens at a time: a tap's weights are loaded and unpacked once for the TPT tokens,
// whose neighbour rows are TPT independent 16-byte loads in flight.
//
// Reads K x the size of V, most of it from L2 and L1: at 131072 tokens of 768 channels and 25 taps 5.0 GB against
// 0.2 GB of values.  There L2 is 42 % busy and the ALU, which unpacks, 50 %: bound by the latency of the neighbour rows, so
// what counts is how many of them an SM has in flight: four tokens side by side, one tap at a time and three CTAs (80
// registers), whose (row, weight) pairs of a tap lie together: 131072 x 768 x 25 501 -> 477 us (two taps and two CTAs, 104
// registers, before), 32768 x 768 x 9 66.2 -> 58.4, 32768 x 384 x 9 35.4 -> 32.6; one token: four taps, four CTAs.  (The bounds
// leave the bfloat16 forms spills of 4 to 20 bytes.)
#include "common.cuh"
#include "f32x2.cuh"

namespace convnn {
namespace {

constexpr int THREADS = 256;

struct DwParams {
    const void* v;
    const int32_t* idx;
    const float* val;
    const void* w;
    void* o;
    int M, T, H, Cp, K, maximum, softmax;
    int C;          // taps per neighbour (row stride of w)
    int groups;     // channel groups of VEC per token; the output row holds groups * VEC values
    int wvec;       // taps can be read VEC at a time
};

// Channel values as packed fp32 pairs.
template <typename T, int VEC> struct Channels;
template <> struct Channels<__nv_bfloat16, 8> {
    typedef uint4 raw;
    static __device__ __forceinline__ void unpack(const raw& r, f32x2 (&x)[4]) { bf16x8_to_f32x2(r, x); }
};
template <> struct Channels<float, 4> {
    typedef ulonglong2 raw;
    static __device__ __forceinline__ void unpack(const raw& r, f32x2 (&x)[2]) { x[0] = r.x; x[1] = r.y; }
};

__device__ __forceinline__ void store_group(__nv_bfloat16* o, const f32x2 (&a)[4]) {
    *reinterpret_cast<uint4*>(o) = f32x2_to_bf16x8(a);
}
template <int N>
__device__ __forceinline__ void store_group(float* o, const f32x2 (&a)[N]) {
#pragma unroll
    for (int q = 0; q < N; q += 2) *reinterpret_cast<ulonglong2*>(o + 2 * q) = make_ulonglong2(a[q], a[q + 1]);
}

// (neighbour row in units of VEC channels, weight) pairs of tokens m0 ... m0 + nt - 1 into shared memory, the TPT tokens of
// a set side by side per tap.  The exponentials are taken by all threads; a token's maximum and its sum in tap order by
// one, so the weights are those of a serial loop.  Threads go along shared memory (along a token's taps, with four tokens per
// set, their stores met in the same banks: 830000 tokens of 16 float32 channels, 25 taps 250 us).  The places behind the last
// token hold its pairs again.
template <int VEC, int TPT>
__device__ __forceinline__ void token_pairs(const DwParams& p, int m0, int nt, int2* pairs, float* red) {
    const int n_up = (nt + TPT - 1) / TPT * TPT * p.K;
    const long long nbase = (long long)m0 * p.K;
    auto at = [&](int t, int j) { return ((t / TPT) * p.K + j) * TPT + t % TPT; };
    // token and tap of place e
    auto whose = [&](int e, int& t, int& j) {
        const int per_set = p.K * TPT, set = e / per_set, in = e - set * per_set;
        t = min(set * TPT + in % TPT, nt - 1);
        j = in / TPT;
    };
    for (int e = threadIdx.x; e < n_up; e += THREADS) {
        int t, j;
        whose(e, t, j);
        const long long ne = nbase + t * p.K + j;
        const int bh = (m0 + t) / p.T, b = bh / p.H, h = bh - b * p.H;
        const float x = p.val[ne];
        pairs[e] = make_int2(((b * p.T + p.idx[ne]) * p.H + h) * (p.Cp / VEC), __float_as_int(p.maximum ? x : -x));
    }
    __syncthreads();
    // f(weight, token) over all of them
    auto each = [&](auto f) {
        for (int e = threadIdx.x; e < n_up; e += THREADS) {
            int t, j;
            whose(e, t, j);
            pairs[e].y = __float_as_int(f(__int_as_float(pairs[e].y), t));
        }
    };
    if (p.softmax) {
        for (int t = threadIdx.x; t < nt; t += THREADS) {
            float m = -3.402823466e38f;
#pragma unroll 8
            for (int j = 0; j < p.K; ++j) m = fmaxf(m, __int_as_float(pairs[at(t, j)].y));
            red[t] = m;
        }
        __syncthreads();
        each([&](float x, int t) { return expf(x - red[t]); });
        __syncthreads();
        for (int t = threadIdx.x; t < nt; t += THREADS) {
            float s = 0.f;
#pragma unroll 8
            for (int j = 0; j < p.K; ++j) s += __int_as_float(pairs[at(t, j)].y);
            red[t] = s;
        }
        __syncthreads();
        each([&](float x, int t) { return x / red[t]; });
    } else if (!p.maximum) {
        each([](float x, int) { return 1.0f / (-x + 1e-8f); });
    }
    __syncthreads();
}

// Rows in flight: TPT tokens side by side per tap, UNROLL taps; more of either leaves fewer warps (MINB CTAs per SM).
template <typename T, typename TO, int VEC, int TPT, int UNROLL, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) gather_conv_dw_kernel(const DwParams p, const int TT) {
    chain_begin_for<TO>();
    typedef Channels<T, VEC> Ch;
    extern __shared__ __align__(16) unsigned char dw_smem[];
    int2* pairs = reinterpret_cast<int2*>(dw_smem);           // [TT / TPT][K][TPT]
    float* red = reinterpret_cast<float*>(pairs + TT * p.K);  // [TT]
    const int m0 = blockIdx.x * TT, nt = min(TT, p.M - m0);
    token_pairs<VEC, TPT>(p, m0, nt, pairs, red);

    const typename Ch::raw* v = static_cast<const typename Ch::raw*>(p.v);
    const T* w = static_cast<const T*>(p.w);
    const int sets = (nt + TPT - 1) / TPT;
    for (int item = threadIdx.x; item < sets * p.groups; item += THREADS) {
        const int set = item / p.groups, cg = item - set * p.groups, c = cg * VEC;
        const typename Ch::raw* vc = v + cg;
        const int2* pr = pairs + set * p.K * TPT;
        f32x2 acc[TPT][VEC / 2];
#pragma unroll
        for (int q = 0; q < TPT; ++q)
#pragma unroll
            for (int e = 0; e < VEC / 2; ++e) acc[q][e] = 0ull;
#pragma unroll UNROLL
        for (int j = 0; j < p.K; ++j) {
            typename Ch::raw raw[TPT];
            float pj[TPT];
            if constexpr (TPT == 1) {
                const int2 e = pr[j];
                raw[0] = vc[e.x];
                pj[0] = __int_as_float(e.y);
            } else {
#pragma unroll
                for (int q = 0; q < TPT; q += 2) {
                    const int4 e = *reinterpret_cast<const int4*>(pr + j * TPT + q);
                    raw[q] = vc[e.x];
                    raw[q + 1] = vc[e.z];
                    pj[q] = __int_as_float(e.y);
                    pj[q + 1] = __int_as_float(e.w);
                }
            }
            f32x2 w2[VEC / 2];
            if (p.wvec) {
                Ch::unpack(*reinterpret_cast<const typename Ch::raw*>(w + j * p.C + c), w2);
            } else {
                float ws[VEC];
#pragma unroll
                for (int e = 0; e < VEC; ++e) ws[e] = c + e < p.C ? to_f32<T>(w[j * p.C + c + e]) : 0.f;
#pragma unroll
                for (int e = 0; e < VEC / 2; ++e) w2[e] = pack2(ws[2 * e], ws[2 * e + 1]);
            }
#pragma unroll
            for (int q = 0; q < TPT; ++q) {
                f32x2 x[VEC / 2];
                Ch::unpack(raw[q], x);
                const f32x2 p2 = pack2(pj[q], pj[q]);
#pragma unroll
                for (int e = 0; e < VEC / 2; ++e) acc[q][e] = fma2(w2[e], mul2(p2, x[e]), acc[q][e]);
            }
        }
        TO* o = static_cast<TO*>(p.o) + (long long)(m0 + set * TPT) * p.groups * VEC + c;
#pragma unroll
        for (int q = 0; q < TPT; ++q)
            if (set * TPT + q < nt) store_group(o + (long long)q * p.groups * VEC, acc[q]);
    }
}

// Weighted neighbour block of the tensor-core standard conv: P[m, j * C + c] = bf16(weight(m, j) * v[neighbour(m, j), c]),
// the A operand of a GEMM with the (d_k, K * C) tap weights; four independent rows in flight per thread.
__global__ void __launch_bounds__(THREADS) gather_weighted_kernel(const DwParams p, const int TT) {
    chain_begin();
    constexpr int U = 4;
    extern __shared__ __align__(16) unsigned char dw_smem[];
    int2* pairs = reinterpret_cast<int2*>(dw_smem);
    float* red = reinterpret_cast<float*>(pairs + TT * p.K);
    const int m0 = blockIdx.x * TT, nt = min(TT, p.M - m0);
    token_pairs<8, 1>(p, m0, nt, pairs, red);
    const uint4* v = static_cast<const uint4*>(p.v);
    uint4* o = static_cast<uint4*>(p.o) + (long long)m0 * p.K * p.groups;
    const int n = nt * p.K * p.groups;                        // output vectors, consecutive in memory
    for (int i0 = threadIdx.x; i0 < n; i0 += THREADS * U) {
        uint4 raw[U];
        float w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * THREADS;
            if (i < n) {
                const int e = i / p.groups;
                const int2 pr = pairs[e];
                w[u] = __int_as_float(pr.y);
                raw[u] = v[pr.x + (i - e * p.groups)];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * THREADS;
            if (i < n) {
                f32x2 x[4];
                bf16x8_to_f32x2(raw[u], x);
                const f32x2 w2 = pack2(w[u], w[u]);
#pragma unroll
                for (int q = 0; q < 4; ++q) x[q] = mul2(w2, x[q]);
                o[i] = f32x2_to_bf16x8(x);
            }
        }
    }
}

template <typename T, typename TO, int VEC>
int launch(const DwParams& p, cudaStream_t st) {
    // Four tokens per thread where that still leaves every SM two CTAs' worth of threads, else one.  Tokens per CTA: one
    // item (token set, channel group) per thread on small grids; on large ones up to eight, as long as six CTAs per SM
    // remain, so that a CTA's prologue (its tokens' weights) is spread over more rows (131072 x 768, 25 taps: 641 us
    // with one item per thread where eight took 501).
    const long long items = (long long)p.M * p.groups;
    const int tpt = items >= 4LL * device_sms() * 512 ? 4 : 1;
    int TT = (THREADS * tpt + p.groups - 1) / p.groups;
    const long long mult = p.M / ((long long)TT * device_sms() * 6);
    if (mult > 1) TT *= mult < 8 ? (int)mult : 8;
    // A grid that leaves SMs idle: fewer tokens per CTA, whose weights come first, at the price of idle threads (us; 2 x 65 x 96, 25 taps
    // 7.4 -> 4.7, 10 x 197 x 192 8.4 -> 6.3, 14 x 65 x 192, 16 taps 6.5 -> 4.2, 3 x 65 x 96, 9 taps 5.0 -> 3.9).
    const int spread = (p.M + 2 * device_sms() - 1) / (2 * device_sms());
    if (tpt == 1 && TT > spread) TT = spread;
    if (TT > 4096 / p.K) TT = 4096 / p.K;                 // 32 KB of (row, weight) pairs
    TT = TT / tpt * tpt;
    if (TT < tpt) TT = tpt;
    const size_t smem = (size_t)TT * p.K * 8 + TT * 4;
    const int grid = (p.M + TT - 1) / TT;
    // The form by the rounds of CTAs per SM it needs: with four tokens per thread three CTAs of one tap in flight, or two of two
    // taps where both need two rounds (3 x 1611 tokens x 10, 96 channels, 25 taps 36.1, 32.7 us); with one token four CTAs of four
    // taps while that is one round (two CTAs of eight, of more than twelve taps: 2 x 65 x 96, 25 taps 8.9, 7.4; unless that leaves four or
    // more to be taken one by one: 17 x 65 x 2 heads of 64, float32, 13 taps 4.1, 4.6, 115 x 79 x 16, 20 taps 4.2, 4.7), then five or six of
    // two taps, which fit in one (71 x 34 x 2 heads of 128, float32, 3 taps 5.4, 4.1; 9 x 701 x 2 heads of 64 6.6, 5.3).
    const int sms = device_sms(), per_sm = (grid + sms - 1) / sms;
    auto go = [&](auto kern) { launch_chained(kern, grid, THREADS, smem, st, p, TT); };
    if (tpt == 4 && per_sm != 4) go(gather_conv_dw_kernel<T, TO, VEC, 4, 1, 3>);
    else if (tpt == 4) go(gather_conv_dw_kernel<T, TO, VEC, 4, 2, 2>);
    else if (per_sm <= 2 && p.K > 12 && p.K % 8 < 4) go(gather_conv_dw_kernel<T, TO, VEC, 1, 8, 2>);
    else if (per_sm <= 4) go(gather_conv_dw_kernel<T, TO, VEC, 1, 4, 4>);
    else if (per_sm == 6) go(gather_conv_dw_kernel<T, TO, VEC, 1, 2, 6>);
    else go(gather_conv_dw_kernel<T, TO, VEC, 1, 2, 5>);
    CONVNN_CHECK_LAUNCH("gather_conv_dw");
    return CONVNN_OK;
}

DwParams params_of(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                   const void* w_conv, void* o) {
    DwParams p{};
    p.v = v; p.idx = idx; p.val = val; p.w = w_conv; p.o = o;
    p.M = dm.B * dm.H * dm.T; p.T = dm.T; p.H = dm.H; p.Cp = dm.Cp; p.K = dm.K;
    p.maximum = d->metric != CONVNN_EUCLIDEAN; p.softmax = d->softmax;
    return p;
}

}  // namespace

// P rows of K * C bfloat16 values; C a multiple of eight, no coordinate channel.
int launch_gather_weighted(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val, void* P,
                           cudaStream_t st) {
    DwParams p = params_of(d, dm, v, idx, val, nullptr, P);
    p.groups = dm.C / 8;
    // about eight 16-byte vectors per thread; a token alone has K * C / 8 of them (a fixed 64 tokens per CTA left two
    // images of 65 tokens, 768 channels, 25 taps on four CTAs: 245 us)
    int TT = 8 * THREADS / (p.K * p.groups);
    TT = TT < 1 ? 1 : (TT > 64 ? 64 : TT);
    launch_chained(gather_weighted_kernel, (p.M + TT - 1) / TT, THREADS, (size_t)TT * p.K * 8 + TT * 4, st, p, TT);
    CONVNN_CHECK_LAUNCH("gather_weighted");
    return CONVNN_OK;
}

// out_f32: rows of Cp unrounded values (the separable conv's intermediate with the coordinate channel); otherwise rows
// of d_k values in the storage type.  Returns CONVNN_E_UNSUPPORTED (last_error untouched) where rows are no multiple of
// 16 bytes.
int try_launch_gather_conv_dw(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                              const void* w_conv, void* o, bool out_f32, cudaStream_t st) {
    const bool f32 = d->dtype == CONVNN_F32;
    const int vec = f32 ? 4 : 8, channels = out_f32 ? dm.Cp : dm.dk;
    if (channels % vec != 0 || dm.Cp % vec != 0 || !aligned16(v) || !aligned16(o)) return CONVNN_E_UNSUPPORTED;
    DwParams p = params_of(d, dm, v, idx, val, w_conv, o);
    p.C = out_f32 ? dm.C : dm.dk; p.groups = channels / vec;
    p.wvec = p.C % vec == 0 && aligned16(w_conv);
    if (f32) return launch<float, float, 4>(p, st);
    return out_f32 ? launch<__nv_bfloat16, float, 8>(p, st) : launch<__nv_bfloat16, __nv_bfloat16, 8>(p, st);
}

}  // namespace convnn
