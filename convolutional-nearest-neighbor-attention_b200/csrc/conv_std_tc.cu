// Standard conv over the neighbours on the tensor cores, bfloat16 heads of 16, 32 or 64 channels (reference layers.py:345-406,
// 313):   o[b, h, t, oc] = sum_{j, c} w[oc, j, c] * bf16(p[t, j] * v[b, n(t, j), h, c])
//
// The weighted neighbour block is the A operand of a GEMM and never leaves the SM: sixteen producer warps (eight tokens of a
// 128-token tile each) turn their tokens' values into weights, fetch the neighbour rows of a few taps ahead, and write them
// weighted and rounded into a ring of swizzled [128 x d_k] blocks; the tap weights stay in shared memory for the
// CTA's life.  Rounding and the order of the sums are those of gather_weighted_kernel + gemm_tc, to which K times the size of
// v went through memory twice.  A CTA owns whole (batch, head) slices, so with several heads the result can leave in the
// flat reinterpretation the output projection reads (layers.py:247-259), without a kernel of its own.
//
// Bound by the instructions that fetch, weigh and store the neighbour rows (0.57 per cycle and scheduler, shared-memory wavefronts 51 %)
// and their latency on sixteen warps.  128 images x 197 tokens x 12 heads of 32, 9
// taps: 78 us, with the reinterpretation; 98 + 11 us before (block 174 MB written and read).  64 images, 3 heads: 17 (17.5 + 4).
//
// Warps: 0 MMA issuer and TMA of the taps, 1-16 producers, 17-20 epilogue (lane quarters).
#include "common.cuh"
#include "f32x2.cuh"
#include "sm100.cuh"

namespace convnn {

__device__ int g_conv_std_status = 0;

namespace {

using namespace sm100;

constexpr int BM = 128;
constexpr int NP = 16;                  // producer warps
constexpr int TPW = BM / NP;            // tokens of a tile per producer warp
constexpr int NT = 32 * (1 + NP + 4);
constexpr int MAX_SLOTS = 4;
constexpr size_t SMEM_MAX = 226 * 1024;

struct ConvStdParams {
    const uint4* v;             // (B, T, H, d_k)
    const int32_t* idx;
    const float* val;           // (B, H, T, K)
    __nv_bfloat16* o;
    int T, H, K, maximum, softmax, merged;
    int n_units, n_tiles;       // (batch, head) slices, 128-token tiles of one
    int slots;                  // groups of tap blocks in flight
    uint32_t slab;              // bytes of one collected slice
    int acc_cols;
};

__device__ __forceinline__ void fail(volatile int* abort_flag, int code) {
    *abort_flag = 1;
    atomicCAS(&g_conv_std_status, 0, code);
}

// Taps whose rows are requested, and handed to the MMA, together (one each, and values requested
// when they are needed: 145 us at the shape above).
__host__ __device__ constexpr int taps_per_slot(int groups) { return groups <= 4 ? 5 : 3; }

// GROUPS: 16-byte channel groups of a head (d_k / 8).
template <int GROUPS>
__global__ void __launch_bounds__(NT, 1) conv_std_tc_kernel(const __grid_constant__ CUtensorMap tmW, const ConvStdParams p) {
    constexpr int DK = GROUPS * 8;
    constexpr uint32_t PITCH = DK * 2, BLOCK = BM * PITCH;
    constexpr int U = GROUPS <= 4 ? 1 : 2;                          // vectors per lane and tap
    constexpr int AHEAD = taps_per_slot(GROUPS);
    constexpr uint32_t SLOT = AHEAD * BLOCK;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t w_tap = DK * PITCH, slots = p.slots;
    uint8_t* sW = smem + slots * SLOT;                             // [K][d_k x d_k]
    __nv_bfloat16* slab = reinterpret_cast<__nv_bfloat16*>(sW + p.K * w_tap);
    float2* pairs_all = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(slab) + p.slab);      // [NP][TPW][K] weight, row of v
    uint64_t* full = reinterpret_cast<uint64_t*>(pairs_all + BM * p.K);
    uint64_t* empty = full + MAX_SLOTS;
    uint64_t* tfull = empty + MAX_SLOTS;
    uint64_t* tempty = tfull + 2;
    uint64_t* wfull = tempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wfull + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_SLOTS; ++s) {
            mbar_init(&full[s], NP);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 4);
        }
        mbar_init(wfull, 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmW);
    }
    const uint32_t ncols = 2u * p.acc_cols;
    if (warp == 0) {
        tmem_alloc(tmem_slot, ncols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_begin();

    if (warp == 0) {
        if (lane < p.K) {                            // lane j loads the weights of tap j
            const uint32_t mask = p.K == 32 ? 0xffffffffu : (1u << p.K) - 1u;
            if (lane == 0) mbar_expect_tx_a(smem_u32(wfull), p.K * w_tap);
            __syncwarp(mask);
            tma_load_2d_a(smem_u32(sW) + lane * w_tap, &tmW, smem_u32(wfull), lane * DK, 0);
        }
        __syncwarp();
        if (lane == 0) {
            const uint32_t idesc = make_idesc_bf16_f32(BM, DK);
            const uint64_t dhi = kmajor_desc_hi(PITCH);
            auto desc = [&](const void* at) { return dhi | (uint64_t)((smem_u32(at) & 0x3FFFFu) >> 4); };
            bool ok = mbar_wait(wfull, 0, abort_flag);
            if (!ok) fail(abort_flag, 112);
            uint32_t s = 0, ph = 0, n = 0;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x) {
                for (int i = 0; i < p.n_tiles && ok; ++i, ++n) {
                    const uint32_t a = n & 1u;
                    if (!mbar_wait(&tempty[a], ((n >> 1) & 1u) ^ 1u, abort_flag)) { fail(abort_flag, 113); ok = false; break; }
                    tc_fence_after_sync();
                    for (int j0 = 0; j0 < p.K; j0 += AHEAD) {
                        if (!mbar_wait(&full[s], ph, abort_flag)) { fail(abort_flag, 114); ok = false; break; }
                        tc_fence_after_sync();
                        for (int j = j0; j < min(j0 + AHEAD, p.K); ++j)
                            mma_chunk(tmem_base + a * p.acc_cols, desc(smem + s * SLOT + (j - j0) * BLOCK), desc(sW + j * w_tap), idesc,
                                      DK / 16, j != 0);
                        mma_commit(&empty[s]);
                        if (++s == slots) { s = 0; ph ^= 1u; }
                    }
                    if (ok) mma_commit(&tfull[a]);
                }
            }
        }
    } else if (warp <= NP) {
        const int w = warp - 1;
        float2* pairs = pairs_all + w * TPW * p.K;
        // this lane's vector(s) of a tap block: token tok, channel group grp
        const int tok = lane / GROUPS % TPW, grp = lane % GROUPS;
        uint32_t at[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = w * TPW + tok + u * (32 / GROUPS);         // row of the block; the hardware's swizzle of 32, 64, 128 bytes
            const int x = GROUPS == 2 ? (r >> 2) & 1 : (GROUPS == 4 ? (r >> 1) & 3 : r & 7);
            at[u] = (uint32_t)r * PITCH + (uint32_t)((grp ^ x) << 4);
        }
        const bool writes = GROUPS > 2 || lane < 2 * TPW;            // (16 channels: eight tokens are sixteen vectors)
        // the values and neighbours of a tile's tokens are requested a tile ahead: lane l those at l, l + 32, ...
        float xv[TPW];
        int xi[TPW];
        auto request = [&](int unit, int i) {
            const int t0 = i * BM + w * TPW, n = min(TPW, p.T - t0) * p.K;
            const long long nbase = ((long long)unit * p.T + t0) * p.K + lane;
#pragma unroll
            for (int q = 0; q < TPW; ++q) {
                xv[q] = lane + 32 * q < n ? p.val[nbase + 32 * q] : 0.f;
                xi[q] = lane + 32 * q < n ? p.idx[nbase + 32 * q] : 0;
            }
        };
        if ((int)blockIdx.x < p.n_units) request(blockIdx.x, 0);
        bool ok = true;
        uint32_t s = 0, ph = 0;
        for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x) {
            const int b = unit / p.H, h = unit - b * p.H;
            const int vbase = (b * p.T * p.H + h) * GROUPS, vstride = p.H * GROUPS;     // (B T D < 2^31)
            for (int i = 0; i < p.n_tiles && ok; ++i) {
                const int nt = min(TPW, p.T - i * BM - w * TPW);
#pragma unroll
                for (int q = 0; q < TPW; ++q)
                    if (lane + 32 * q < nt * p.K)
                        pairs[lane + 32 * q] = make_float2(p.maximum || !p.softmax ? xv[q] : -xv[q], __int_as_float(vbase + xi[q] * vstride));
                __syncwarp();
                if (i + 1 < p.n_tiles) request(unit, i + 1);
                else if (unit + (int)gridDim.x < p.n_units) request(unit + gridDim.x, 0);
                // weights over the values as in token_weights.cuh (exponentials by all lanes, sums in tap order): sixteen lanes
                // per token, up to 32 values, four pairs of tokens side by side
                const int j = lane & 15;
                if (nt > 0 && p.softmax) {
                    constexpr int M = TPW / 2;
                    float e[M][2], mx[M], sum[M];
                    bool in[M][2];
#pragma unroll
                    for (int c = 0; c < M; ++c) {
                        const int m = 2 * c + (lane >> 4);
                        mx[c] = -3.402823466e38f;
                        sum[c] = 0.f;
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            in[c][q] = m < nt && j + 16 * q < p.K;
                            e[c][q] = in[c][q] ? pairs[m * p.K + j + 16 * q].x : 0.f;
                            if (in[c][q]) mx[c] = fmaxf(mx[c], e[c][q]);
                        }
                    }
#pragma unroll
                    for (int d = 8; d >= 1; d /= 2)
#pragma unroll
                        for (int c = 0; c < M; ++c) mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], d));
#pragma unroll
                    for (int c = 0; c < M; ++c)
#pragma unroll
                        for (int q = 0; q < 2; ++q) e[c][q] = in[c][q] ? expf(e[c][q] - mx[c]) : 0.f;
                    for (int k = 0; k < min(p.K, 16); ++k)
#pragma unroll
                        for (int c = 0; c < M; ++c) sum[c] += __shfl_sync(0xffffffffu, e[c][0], k, 16);
                    for (int k = 16; k < p.K; ++k)
#pragma unroll
                        for (int c = 0; c < M; ++c) sum[c] += __shfl_sync(0xffffffffu, e[c][1], k - 16, 16);
#pragma unroll
                    for (int c = 0; c < M; ++c)
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            if (in[c][q]) pairs[(2 * c + (lane >> 4)) * p.K + j + 16 * q].x = e[c][q] / sum[c];
                } else if (!p.softmax && !p.maximum) {
                    for (int e = lane; e < nt * p.K; e += 32) pairs[e].x = 1.0f / (pairs[e].x + 1e-8f);
                }
                __syncwarp();
                for (int j0 = 0; j0 < p.K; j0 += AHEAD) {
                    uint4 raw[AHEAD][U];
                    float wt[AHEAD][U];
#pragma unroll
                    for (int j = 0; j < AHEAD; ++j)
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int m = tok + u * (32 / GROUPS);
                            raw[j][u] = make_uint4(0u, 0u, 0u, 0u);              // rows past the sequence: zeros
                            wt[j][u] = 0.f;
                            if (j0 + j < p.K && m < nt && writes) {
                                const float2 e = pairs[m * p.K + j0 + j];
                                wt[j][u] = e.x;
                                raw[j][u] = __ldg(p.v + __float_as_int(e.y) + grp);
                            }
                        }
                    ok = mbar_wait(&empty[s], ph ^ 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { if (lane == 0) fail(abort_flag, 115); break; }
#pragma unroll
                    for (int j = 0; j < AHEAD; ++j) {
                        if (j0 + j >= p.K) break;
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            f32x2 x[4];
                            bf16x8_to_f32x2(raw[j][u], x);
                            const f32x2 w2 = pack2(wt[j][u], wt[j][u]);
#pragma unroll
                            for (int q = 0; q < 4; ++q) x[q] = mul2(w2, x[q]);
                            if (writes) *reinterpret_cast<uint4*>(smem + s * SLOT + j * BLOCK + at[u]) = f32x2_to_bf16x8(x);
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[s]);
                    if (++s == slots) { s = 0; ph ^= 1u; }
                }
                __syncwarp();
            }
        }
    } else {
        // Every epilogue warp makes the same passes and meets both barriers of a unit, also after a wait has expired.
        const int lq = warp & 3, tid = threadIdx.x - 32 * (1 + NP);
        uint32_t n = 0;
        for (int unit = blockIdx.x; unit < p.n_units; unit += gridDim.x) {
            const int b = unit / p.H, h = unit - b * p.H;
            for (int i = 0; i < p.n_tiles; ++i, ++n) {
                const uint32_t a = n & 1u;
                bool ok = mbar_wait(&tfull[a], (n >> 1) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { if (lane == 0) fail(abort_flag, 116); continue; }
                tc_fence_after_sync();
                const int t = i * BM + lq * 32 + lane;
#pragma unroll
                for (int c = 0; c < DK; c += 16) {
                    uint32_t r[16], x[8];
                    tmem_ld_x16(tmem_base + ((uint32_t)(lq * 32) << 16) + a * p.acc_cols + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const __nv_bfloat162 f = __floats2bfloat162_rn(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
                        x[e] = *reinterpret_cast<const uint32_t*>(&f);
                    }
                    if (t < p.T) {
                        uint4* dst = reinterpret_cast<uint4*>(slab + t * DK + c);
                        dst[0] = make_uint4(x[0], x[1], x[2], x[3]);
                        dst[1] = make_uint4(x[4], x[5], x[6], x[7]);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[a]);
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");           // the slice is complete
            if (p.merged) {
                // y[b, t, h d_k + c] = flat(slice)[c T + t]; neighbouring threads share an output row
                __nv_bfloat16* out = p.o + (long long)b * p.T * p.H * DK + h * DK;
                for (int e = tid; e < p.T * GROUPS; e += 128) {
                    const int t = e / GROUPS, g = e % GROUPS;
                    const __nv_bfloat16* src = slab + g * 8 * p.T + t;
                    uint32_t x[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        x[q] = (uint32_t)__bfloat16_as_ushort(src[2 * q * p.T]) | ((uint32_t)__bfloat16_as_ushort(src[(2 * q + 1) * p.T]) << 16);
                    *reinterpret_cast<uint4*>(out + (long long)t * p.H * DK + g * 8) = make_uint4(x[0], x[1], x[2], x[3]);
                }
            } else {
                uint4* out = reinterpret_cast<uint4*>(p.o + (long long)unit * p.T * DK);
                for (int e = tid; e < p.T * GROUPS; e += 128) out[e] = reinterpret_cast<const uint4*>(slab)[e];
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");           // and may be overwritten
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // a wait expired: give copies still in flight time to land before the CTA's shared memory is released
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, ncols);
    }
}

template <int GROUPS>
int launch(const ConvStdParams& p, size_t smem, const CUtensorMap& tmW, cudaStream_t st) {
    auto kern = conv_std_tc_kernel<GROUPS>;
    CONVNN_ENSURE_SMEM(kern, smem);
    const int sms = device_sms();
    launch_chained(kern, p.n_units < sms ? p.n_units : sms, NT, smem, st, tmW, p);
    CONVNN_CHECK_LAUNCH("conv_std_tc");
    return CONVNN_OK;
}

}  // namespace

// Where this kernel is faster than gather_weighted_kernel + gemm_tc (+ merge_heads).  Its time goes by the 128-token tiles of the
// busiest CTA (3.6 us and 2.5 to 6.5 a tile), the others' by rows (0.1 to 0.5 ns) from a floor of 7 to 16 us.  One tile per
// CTA always wins.  Beyond that `fill` counts, the share of those tiles that holds rows: short sequences and ragged ends
// waste tiles, many taps make the others write more.  us, others -> this kernel, slices x tokens x channels, nine taps unless noted:
//   1 tile     8 x 65 x 32 10.2 -> 6.9     148 x 100 x 64 13.5 -> 9.5
//   one slice  8 x 197 x 64 11.0 -> 14.5, 74 x 256 x 64, 5 taps 11.3 -> 12.9 (not taken)     148 x 197 x 64 20.9 -> 15.0, 148 x 2000 x 16 81.8 -> 59.0
//   several    600 x 17 x 32 11.1 -> 17.9, 600 x 197 x 64, 5 taps 40.7 -> 45.2, 300 x 1000 x 16, 5 taps 53.2 -> 65.2 (not taken)
//              600 x 197 x 32 44.5 -> 37.5     600 x 256 x 64 85.3 -> 60.5     1536 x 256 x 16 104.7 -> 79.5
// Merged, the reinterpretation's own kernel (2.5 us and more) is saved as well.  Whole layers of two or four heads, us:
//   148 slices x 197 x 64 54.3 -> 45.1, 600 x 197 x 32 127.7 -> 117.4     8 x 256 x 64 31.1 -> 34.0, 600 x 17 x 16 43.5 -> 49.9 (not taken)
// (captured; call by call the saved launches count too: ViT-Tiny of three heads, 16 images 749 -> 719)
static bool conv_std_wanted(const Dims& dm, bool merged) {
    const int sms = device_sms();
    const long long units = (long long)dm.B * dm.H, tiles = (units + sms - 1) / sms * ((dm.T + BM - 1) / BM);
    if (dm.T > 2 * BM && units < sms) return false;      // (one slice of 600 tokens: 10 us before, 21 here)
    if (tiles == 1) return true;
    const double fill = (double)units * dm.T / ((double)tiles * BM * sms), taps = dm.K;
    if (merged) {
        // (tokens a multiple of 32 apart lie in one bank for the reinterpreted store: 2 x 256 x 64 30.4 -> 33.2, 2 x 197 x 64 29.7 -> 30.6)
        if (tiles == 2 && (fill >= 0.4 || dm.K * dm.dk <= 288 || dm.T % 32 != 0)) return true;
    } else if (units <= sms) {
        if ((tiles == 2 || dm.K >= 5) && (dm.dk == 32 ? units * 3 >= sms * 2 : units * 5 >= sms * 4)) return true;
    } else if (tiles == 2 && fill >= 0.5) {
        return true;
    }
    double need;
    if (dm.dk == 16) need = merged ? 0.45 + 1.25 / taps : dm.K > 16 ? 0.34 : 0.42 + 2.25 / taps;
    else if (dm.dk == 32) need = (merged ? 0.1 : 0.21) + 2. / taps;
    else need = 0.25 + (merged ? 1.5 : 2.25) / taps;
    // sixteen taps of sixteen channels: the weights that a warp's tokens read lie in the same banks (300 x 2000: 226 -> 253)
    if (dm.dk == 16 && dm.K == 16 && !merged) need += 0.12;
    return fill >= need;
}

// merged: o is (B, T, H d_k) in the flat reinterpretation, else (B, H, T, d_k).  CONVNN_E_UNSUPPORTED (last_error untouched)
// where heads are of another width, where the other kernels are faster (above), or where the tap weights, two slots and a
// slice do not fit in shared memory (64 channels: from 14 taps on).
int try_launch_conv_std_tc(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                           const void* w_conv, void* o, bool merged, cudaStream_t st) {
    if (d->dtype != CONVNN_BF16 || d->conv_type != CONVNN_STANDARD || d->coord || force_simt() ||
        (dm.dk != 16 && dm.dk != 32 && dm.dk != 64) ||
        !conv_std_wanted(dm, merged) || !aligned16(v) || !aligned16(w_conv) || !aligned16(o))
        return CONVNN_E_UNSUPPORTED;
    ConvStdParams p{};
    p.v = static_cast<const uint4*>(v); p.idx = idx; p.val = val; p.o = static_cast<__nv_bfloat16*>(o);
    p.T = dm.T; p.H = dm.H; p.K = dm.K; p.maximum = d->metric != CONVNN_EUCLIDEAN; p.softmax = d->softmax;
    p.merged = merged ? 1 : 0;
    p.n_units = dm.B * dm.H; p.n_tiles = (dm.T + BM - 1) / BM;
    p.acc_cols = dm.dk < 32 ? 32 : dm.dk;
    const size_t slab = ((size_t)dm.T * dm.dk * 2 + 15) / 16 * 16;
    const size_t fixed = 1024 + (size_t)dm.K * dm.dk * dm.dk * 2 + slab + (size_t)BM * dm.K * 8 + (2 * MAX_SLOTS + 8) * 8;
    const size_t slot = (size_t)taps_per_slot(dm.dk / 8) * BM * dm.dk * 2;
    if (fixed + 2 * slot > SMEM_MAX) return CONVNN_E_UNSUPPORTED;
    const size_t fit = (SMEM_MAX - fixed) / slot;
    p.slots = fit < (size_t)MAX_SLOTS ? (int)fit : MAX_SLOTS;
    p.slab = (uint32_t)slab;
    CUtensorMap tmW;
    const uint64_t dims[2] = {(uint64_t)dm.K * dm.dk, (uint64_t)dm.dk}, str[1] = {(uint64_t)dm.K * dm.dk * 2};
    const uint32_t box[2] = {(uint32_t)dm.dk, (uint32_t)dm.dk};
    if (!encode_tensor_map_bf16(&tmW, w_conv, 2, dims, str, box, dm.dk * 2)) return CONVNN_E_CUDA;
    size_t smem = fixed + p.slots * slot;
    if (smem < 116 * 1024) smem = 116 * 1024;
    if (dm.dk == 16) return launch<2>(p, smem, tmW, st);
    if (dm.dk == 32) return launch<4>(p, smem, tmW, st);
    return launch<8>(p, smem, tmW, st);
}

int read_conv_std_status(int* out) {
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_conv_std_status, sizeof(int));
    if (e != cudaSuccess) return set_error(CONVNN_E_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    *out = v;
    return CONVNN_OK;
}

}  // namespace convnn
