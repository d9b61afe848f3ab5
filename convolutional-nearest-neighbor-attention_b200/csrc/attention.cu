// Softmax attention  o = softmax(q k^T / sqrt(d_k)) v  per (batch, head): the other half of the
// reference's MultiHeadBranchingAttention (MultiHeadAttention.forward, layers.py:105-130).
//
// bfloat16, up to 256 tokens, d_k a multiple of 16 up to 128 -- the tensor-core kernel.  A work
// unit is 128 query rows of one (batch, head); the whole key range is one MMA tile:
//   warp 0     TMA producer: Q rows (128 x d_k) and K rows (BN x d_k) as K-major swizzled chunks,
//              V rows (BN x d_k) token-major.
//   warp 1     MMA issuer.  MMA 1: S = Q K^T (M = 128, N = BN = tokens rounded up to 16) into
//              TMEM.  MMA 2: O = P V with P (bfloat16, written by the softmax warps) as the
//              K-major A operand and V^T as the K-major B operand; O lands in the first d_k
//              columns of the same accumulator once every row of S has been consumed.
//   warps 2-5  a thread owns one query row (its TMEM lane): row maximum, p = exp2((s - max) *
//              log2(e)/sqrt(d_k)), row sum; p goes to shared memory in the 128-byte-swizzled
//              operand layout.  Before that the four warps transpose V (token-major, as the
//              projection stores it) into the K-major V^T chunks MMA 2 needs.  Finally O / sum is
//              read back from TMEM, rounded and stored.
// P and the Q / K chunks share one shared-memory region (Q and K are dead once S is complete), so two
// CTAs fit on an SM at ViT shapes and cover each other's serial phases.
// Every mbarrier wait is bounded; on expiry the CTA latches a code and drains.
//
// Anything else (float32, longer sequences, other head widths) is computed on the fp32 pipes, a tile of rows per CTA.
#include <math_constants.h>

#include "common.cuh"
#include "sm100.cuh"
#include "f32x2.cuh"

namespace convnn {

__device__ int g_attention_status = 0;

namespace {

using namespace sm100;

constexpr int BM = 128;
constexpr int NTHREADS = 192;      // TMA warp, MMA warp, 4 softmax warps
constexpr int CW = 16;

struct AttnParams {
    __nv_bfloat16* o;              // (B, T, H * dk)
    int T, H, dk, D;
    int KCH, KC;                   // channels per chunk / chunks of the Q K^T reduction
    int BN, BNpad;                 // key columns of the score tile, TMEM columns
    int NKC2;                      // 64-token chunks of the P V reduction
    int n_row_tiles, n_units;
    uint32_t p_region_bytes;       // shared by P and the Q / K chunks
    float scale_log2;              // log2(e) / sqrt(dk)
};

__device__ __forceinline__ void fail(volatile int* abort_flag, int code) {
    *abort_flag = 1;
    atomicCAS(&g_attention_status, 0, code);
}

__device__ __forceinline__ void tmem_ld_wait_on(uint32_t (&r)[CW]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

template <bool BESIDE>                    // see chain_leave()
__global__ void __launch_bounds__(NTHREADS, 2)
attention_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t pitch = p.KCH * 2;
    const uint32_t a_bytes = BM * pitch, b_bytes = p.BN * pitch;
    const uint32_t v_bytes = (uint32_t)p.BN * p.dk * 2;
    const uint32_t vt_chunk = (uint32_t)p.dk * 128;            // one V^T chunk: d_k rows of 64 tokens
    uint8_t* sP = smem;                                        // [NKC2][128 rows x 128 B]; aliases sQ | sK
    uint8_t* sQ = smem;                                        // [KC][128 x pitch]
    uint8_t* sK = smem + p.KC * a_bytes;                       // [KC][BN x pitch]
    uint8_t* sVt = smem + p.p_region_bytes;                    // [NKC2][dk rows x 128 B]
    uint8_t* sV = sVt + p.NKC2 * vt_chunk;                     // [BN][dk] token-major
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + ((v_bytes + 15) & ~15u));
    uint64_t* qk_full = bars;
    uint64_t* v_full = bars + 1;
    uint64_t* v_empty = bars + 2;
    uint64_t* s_full = bars + 3;
    uint64_t* p_ready = bars + 4;
    uint64_t* o_full = bars + 5;
    uint64_t* t_empty = bars + 6;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t ncols = (uint32_t)p.BNpad;

    if (threadIdx.x == 0) {
        mbar_init(qk_full, 1);
        mbar_init(v_full, 1);
        mbar_init(v_empty, 4);
        mbar_init(s_full, 1);
        mbar_init(p_ready, 4);
        mbar_init(o_full, 1);
        mbar_init(t_empty, 4);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmQ);
        prefetch_tensormap(&tmK);
        prefetch_tensormap(&tmV);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, ncols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_wait_unless(BESIDE);
    chain_next();

    if (warp == 0) {
        {
            uint32_t it = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x, ++it) {
                const uint32_t ph = it & 1u;
                const int bh = unit / p.n_row_tiles, rt = unit - bh * p.n_row_tiles;
                const int b = bh / p.H, h = bh - b * p.H;
                // Q / K land where the previous unit's P was: MMA 2 must have finished reading it
                if (it > 0 && !mbar_wait_warp(smem_u32(o_full), ph ^ 1u, abort_flag)) { fail(abort_flag, 61); ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(qk_full, p.KC * (a_bytes + b_bytes));
                    for (int kc = 0; kc < p.KC; ++kc) {
                        tma_load_4d(sQ + kc * a_bytes, &tmQ, qk_full, kc * p.KCH, h, rt * BM, b);
                        tma_load_4d(sK + kc * b_bytes, &tmK, qk_full, kc * p.KCH, h, 0, b);
                    }
                }
                if (!mbar_wait_warp(smem_u32(v_empty), ph ^ 1u, abort_flag)) { fail(abort_flag, 62); ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(v_full, v_bytes);
                    tma_load_4d(sV, &tmV, v_full, 0, h, 0, b);
                }
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc1 = make_idesc_bf16_f32(BM, p.BN);
            const uint32_t idesc2 = make_idesc_bf16_f32(BM, p.dk);
            const uint64_t dhi = kmajor_desc_hi(pitch), dhi128 = kmajor_desc_hi(128);
            const int nk16 = p.KCH / 16;
            const uint32_t sQ0 = smem_u32(sQ), sK0 = smem_u32(sK), sP0 = smem_u32(sP), sVt0 = smem_u32(sVt);
            uint32_t it = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x, ++it) {
                const uint32_t ph = it & 1u;
                if (!mbar_wait_warp(smem_u32(t_empty), ph ^ 1u, abort_flag)) { fail(abort_flag, 63); ok = false; break; }
                if (!mbar_wait_warp(smem_u32(qk_full), ph, abort_flag)) { fail(abort_flag, 64); ok = false; break; }
                tc_fence_after_sync();
                if (elect_one()) {
                    for (int kc = 0; kc < p.KC; ++kc) {
                        const uint64_t ad = dhi | (uint64_t)(((sQ0 + kc * a_bytes) & 0x3FFFFu) >> 4);
                        const uint64_t bd = dhi | (uint64_t)(((sK0 + kc * b_bytes) & 0x3FFFFu) >> 4);
                        mma_chunk(tmem_base, ad, bd, idesc1, nk16, kc != 0);
                    }
                    mma_commit(s_full);
                }
                if (!mbar_wait_warp(smem_u32(p_ready), ph, abort_flag)) { fail(abort_flag, 65); ok = false; break; }
                tc_fence_after_sync();
                if (elect_one()) {
                    uint32_t acc = 0;
                    for (int kc2 = 0; kc2 < p.NKC2; ++kc2) {
                        const uint64_t ad = dhi128 | (uint64_t)(((sP0 + kc2 * 16384u) & 0x3FFFFu) >> 4);
                        const uint64_t bd = dhi128 | (uint64_t)(((sVt0 + kc2 * vt_chunk) & 0x3FFFFu) >> 4);
                        for (int k16 = 0; k16 < 4; ++k16) {
                            if (kc2 * 64 + k16 * 16 >= p.BN) break;
                            mma_bf16_ss(tmem_base, ad + 2 * k16, bd + 2 * k16, idesc2, acc);
                            acc = 1;
                        }
                    }
                    mma_commit(o_full);
                }
            }
        }
    } else {
        const int lq = warp & 3;
        const int r = lq * 32 + lane;            // query row within the tile = TMEM lane
        const int st = threadIdx.x - 64;         // 0 .. 127 among the softmax threads
        const uint32_t taddr = tmem_base + ((uint32_t)(lq * 32) << 16);
        const uint32_t sP_row = smem_u32(sP) + r * 128;
        uint32_t it = 0;
        bool ok = true;
        for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x, ++it) {
            const uint32_t ph = it & 1u;
            const int bh = unit / p.n_row_tiles, rt = unit - bh * p.n_row_tiles;
            const int b = bh / p.H, h = bh - b * p.H;
            const int row = rt * BM + r;
            // ---- V (token-major) -> V^T chunks: [channel][64 tokens], 16-byte segments swizzled ------
            ok = mbar_wait(v_full, ph, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) { if (lane == 0) fail(abort_flag, 66); break; }
            {
                // item i = (segment of 8 tokens sg, channel c), i = sg * dk + c, visited with stride 128:
                // (sg, c) advance by (128 / dk, 128 % dk) with a carry, no division in the loop
                const int nseg = p.BN / 8;
                const int dsg = 128 / p.dk, dc = 128 - dsg * p.dk;
                int sg = st / p.dk, c = st - sg * p.dk;
                const unsigned short* v16 = reinterpret_cast<const unsigned short*>(sV);
                while (sg < nseg) {
                    const int t0 = sg * 8;
                    const unsigned short* src = v16 + t0 * p.dk + c;
                    uint32_t w[4];
#pragma unroll
                    for (int e2 = 0; e2 < 4; ++e2) {
                        const uint32_t lo = src[(2 * e2) * p.dk], hi = src[(2 * e2 + 1) * p.dk];
                        w[e2] = lo | (hi << 16);
                    }
                    const int kc2 = t0 >> 6, seg = (t0 & 63) >> 3;
                    uint8_t* dst = sVt + kc2 * vt_chunk + c * 128 + ((seg ^ (c & 7)) << 4);
                    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                    sg += dsg;
                    c += dc;
                    if (c >= p.dk) { c -= p.dk; ++sg; }
                }
            }
            fence_proxy_async();                 // the transposed tile is read by the MMA (async proxy)
            __syncwarp();
            if (lane == 0) mbar_arrive(v_empty);
            // ---- scores -> probabilities -----------------------------------------------------------
            ok = mbar_wait(s_full, ph, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) { if (lane == 0) fail(abort_flag, 67); break; }
            tc_fence_after_sync();
            // row maximum; only the last chunk can hold columns past the sequence
            float m = -CUDART_INF_F;
#pragma unroll 1
            for (int c = 0; c < p.BN; c += CW) {
                uint32_t acc[CW];
                tmem_ld_x16(taddr + c, acc);
                tmem_ld_wait_on(acc);
                if (c + CW > p.T) {
#pragma unroll
                    for (int j = 0; j < CW; ++j)
                        if (c + j >= p.T) acc[j] = 0xff800000u;          // -inf
                }
                float m4[4];
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4)
                    m4[q4] = fmaxf(fmaxf(__uint_as_float(acc[4 * q4]), __uint_as_float(acc[4 * q4 + 1])),
                                   fmaxf(__uint_as_float(acc[4 * q4 + 2]), __uint_as_float(acc[4 * q4 + 3])));
                m = fmaxf(m, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])));
            }
            // p = 2^(s * scale - m * scale): one fused multiply-add and one hardware exp2 per score
            const float ms = -m * p.scale_log2;
            f32x2 sum2 = 0ull;
#pragma unroll 1
            for (int c = 0; c < p.BN; c += CW) {
                uint32_t acc[CW];
                tmem_ld_x16(taddr + c, acc);
                tmem_ld_wait_on(acc);
                if (c + CW > p.T) {
#pragma unroll
                    for (int j = 0; j < CW; ++j)
                        if (c + j >= p.T) acc[j] = 0xff800000u;          // -inf: probability 0
                }
                uint32_t pk[8];
#pragma unroll
                for (int j2 = 0; j2 < 8; ++j2) {
                    float p0, p1;
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p0) : "f"(fmaf(__uint_as_float(acc[2 * j2]), p.scale_log2, ms)));
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p1) : "f"(fmaf(__uint_as_float(acc[2 * j2 + 1]), p.scale_log2, ms)));
                    sum2 = add2(sum2, pack2(p0, p1));
                    __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
                    pk[j2] = *reinterpret_cast<uint32_t*>(&hh);
                }
                const int kc2 = c >> 6, seg = (c & 63) >> 3;
                const uint32_t base = sP_row + kc2 * 16384u;
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(base + (((seg) ^ (r & 7)) << 4)), "r"(pk[0]),
                             "r"(pk[1]), "r"(pk[2]), "r"(pk[3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(base + (((seg + 1) ^ (r & 7)) << 4)), "r"(pk[4]),
                             "r"(pk[5]), "r"(pk[6]), "r"(pk[7]) : "memory");
            }
            float sum_lo, sum_hi;
            unpack2(sum2, sum_lo, sum_hi);
            const float sum = sum_lo + sum_hi;
            fence_proxy_async();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
            // ---- O / sum ---------------------------------------------------------------------------------
            ok = mbar_wait(o_full, ph, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) { if (lane == 0) fail(abort_flag, 68); break; }
            tc_fence_after_sync();
            const float inv = 1.0f / sum;
            __nv_bfloat16* orow = p.o + ((long long)b * p.T + row) * p.D + h * p.dk;
#pragma unroll 1
            for (int c = 0; c < p.dk; c += CW) {
                uint32_t acc[CW];
                tmem_ld_x16(taddr + c, acc);
                tmem_ld_wait_on(acc);
                uint32_t pk[8];
#pragma unroll
                for (int j2 = 0; j2 < 8; ++j2) {
                    __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(acc[2 * j2]) * inv,
                                                              __uint_as_float(acc[2 * j2 + 1]) * inv);
                    pk[j2] = *reinterpret_cast<uint32_t*>(&hh);
                }
                if (row < p.T) {
                    *reinterpret_cast<uint4*>(orow + c) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    *reinterpret_cast<uint4*>(orow + c + 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(t_empty);
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, ncols);
    }
    chain_leave(BESIDE);
}

// R = 8 TR query rows of one (batch, head) per CTA, for float32 and head widths that the tensor-core kernel does not take.
//
//   scores   a thread owns TR rows x up to seven keys (lane, lane + 32, ...); q and K pass through shared memory in chunks of 32
//            channels, the next chunk in registers meanwhile
//   softmax  a warp per row
//   output   a thread owns TR rows x up to seven channels; V passes in chunks of 32 tokens
//
// Columns (keys, channels) that one pass has no room for are spread evenly over several.  Every sum runs in the order of the kernel for
// longer sequences below (channels, tokens and the lanes' partial sums ascending), so that both give the same bits.  What bounds it:
// shared-memory reads, a word per column and a broadcast per row for TR multiply-adds each, and at few rows the chain of chunks.
// us with the four projections, one warp per row reading K a word at a time -> this kernel: 6 x 65 x 192, one head, bfloat16 98 -> 26; 64
// x 197 x 192 2090 -> 115; 8 x 197 x 384 806 -> 84; float32, 8 x 197, 3 heads of 32 171 -> 39; 16 x 197, 12 heads of 32 1113 -> 229.
constexpr int AT_CH = 32, AT_THREADS = 256, AT_COLS = 7, AT_QP = AT_CH + 4;

// Values first .. first + 7 of a row of n, zeros past its end.
template <typename T>
__device__ __forceinline__ void load_eight(float (&x)[8], const T* row, int first, int n, bool vec) {
    if (vec && first + 8 <= n) {
        if constexpr (sizeof(T) == 2) {
            const uint4 u = *reinterpret_cast<const uint4*>(row + first);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[2 * e] = __uint_as_float(w[e] << 16);
                x[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
            }
        } else {
            const float4 u = *reinterpret_cast<const float4*>(row + first), v = *reinterpret_cast<const float4*>(row + first + 4);
            x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
            x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = first + e < n ? to_f32(row[first + e]) : 0.f;
    }
}

// acc[r][g] += a[r][i] * tile[i][32 g + lane] for i = 0 .. n - 1, in that order, G groups of columns; rows of the tile are 32 G + PAD apart.
template <int TR, int G, int PAD>
__device__ __forceinline__ void times_tile(float (&acc)[TR][AT_COLS], const float* a, int pitch, const float* tile, int n) {
    constexpr int V = TR > 5 ? 2 : 4;                // values of a row at once (registers)
    int i = 0;
#pragma unroll 1
    for (; i + V <= n; i += V) {
        float x[TR][V];
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            if (V == 4) {
                const float4 w = *reinterpret_cast<const float4*>(a + r * pitch + i);
                x[r][0] = w.x; x[r][1] = w.y; x[r][V - 2] = w.z; x[r][V - 1] = w.w;
            } else {
                const float2 w = *reinterpret_cast<const float2*>(a + r * pitch + i);
                x[r][0] = w.x; x[r][1] = w.y;
            }
        }
#pragma unroll
        for (int u = 0; u < V; ++u) {
            float t[G];
#pragma unroll
            for (int g = 0; g < G; ++g) t[g] = tile[(i + u) * (32 * G + PAD) + 32 * g];
#pragma unroll
            for (int r = 0; r < TR; ++r)
#pragma unroll
                for (int g = 0; g < G; ++g) acc[r][g] = fmaf(x[r][u], t[g], acc[r][g]);
        }
    }
#pragma unroll 1
    for (; i < n; ++i) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float t = tile[i * (32 * G + PAD) + 32 * g];
#pragma unroll
            for (int r = 0; r < TR; ++r) acc[r][g] = fmaf(a[r * pitch + i], t, acc[r][g]);
        }
    }
}
template <int TR, int PAD>
__device__ __forceinline__ void times_groups(float (&acc)[TR][AT_COLS], const float* a, int pitch, const float* tile, int n, int groups) {
    switch (groups) {
        case 1: times_tile<TR, 1, PAD>(acc, a, pitch, tile, n); break;
        case 2: times_tile<TR, 2, PAD>(acc, a, pitch, tile, n); break;
        case 3: times_tile<TR, 3, PAD>(acc, a, pitch, tile, n); break;
        case 4: times_tile<TR, 4, PAD>(acc, a, pitch, tile, n); break;
        case 5: times_tile<TR, 5, PAD>(acc, a, pitch, tile, n); break;
        case 6: times_tile<TR, 6, PAD>(acc, a, pitch, tile, n); break;
        default: times_tile<TR, 7, PAD>(acc, a, pitch, tile, n); break;
    }
}

// Passes over `cols` columns and groups of 32 per pass.
__host__ __device__ inline int tile_passes(int cols) { return (cols + 32 * AT_COLS - 1) / (32 * AT_COLS); }
__host__ __device__ inline int tile_groups(int cols) { return ((cols + 31) / 32 + tile_passes(cols) - 1) / tile_passes(cols); }

template <typename T, int TR>
__global__ void __launch_bounds__(AT_THREADS, 2)
attention_tile_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ o, int Tn, int H, int dk,
                      float scale, int vec) {
    constexpr int R = 8 * TR;
    chain_begin_for<T>();
    extern __shared__ float sm[];
    const int kp = tile_passes(Tn), kg = tile_groups(Tn), vp = tile_passes(dk), vg = tile_groups(dk);
    const int pitch = (Tn + 3) / 4 * 4 + 4;              // of a row of scores
    float* qs = sm;                                      // [R][AT_QP]
    float* prob = qs + R * AT_QP;                        // [R][pitch]
    float* inv = prob + R * pitch;                       // [R]
    float* tile = inv + R;                               // scores: [32 channels][32 kg + 1 keys], output: [32 tokens][32 vg channels]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bh = blockIdx.y, b = bh / H, h = bh - b * H, row0 = blockIdx.x * R;
    const long long D = (long long)H * dk, base = (long long)b * Tn * D + h * dk;
    const int n_rows = min(R, Tn - row0);
    const int rg = warp * TR;                            // first row of this warp (its lanes read their values as broadcasts)
    float acc[TR][AT_COLS];
    auto clear = [&] {
#pragma unroll
        for (int r = 0; r < TR; ++r)
#pragma unroll
            for (int g = 0; g < AT_COLS; ++g) acc[r][g] = 0.f;
    };
    // ---- scores ----
    const T* kb = k + base;
    const int n_ch = (dk + AT_CH - 1) / AT_CH, keys = 32 * kg;
    // a thread's part of a chunk: eight channels 8 (tid % 4) .. of keys tid / 4, + 64, ... (four lanes read 64 or 128 bytes of a row; the
    // tile's rows are a word longer than they need be, so that they meet in no bank)
    const int lk = tid >> 2, lc = (tid & 3) * 8;
    float next[(32 * AT_COLS + 63) / 64][8], qnext[(R + 31) / 32 * 4];
    auto fetch_k = [&](int pass, int ch) {
        const int c = min(ch * AT_CH + lc, dk);
#pragma unroll
        for (int i = 0; i < (32 * AT_COLS + 63) / 64; ++i)
            if (lk + 64 * i < keys) load_eight<T>(next[i], kb + (long long)min(pass * keys + lk + 64 * i, Tn - 1) * D, c, dk, vec);
        // (four channels 4 (tid % 8) .. of rows tid / 8, + 32)
#pragma unroll
        for (int i = 0; i < (R + 31) / 32; ++i) {
            const int r = (tid >> 3) + 32 * i, c4 = ch * AT_CH + (tid & 7) * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                qnext[4 * i + e] = r < n_rows && c4 + e < dk ? to_f32(q[base + (row0 + r) * D + c4 + e]) * scale : 0.f;
        }
    };
    fetch_k(0, 0);
    for (int pass = 0; pass < kp; ++pass) {
        clear();
        for (int ch = 0; ch < n_ch; ++ch) {
            __syncthreads();                             // the chunk before has been read
#pragma unroll
            for (int i = 0; i < (32 * AT_COLS + 63) / 64; ++i)
                if (lk + 64 * i < keys) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) tile[(lc + e) * (keys + 1) + lk + 64 * i] = next[i][e];
                }
#pragma unroll
            for (int i = 0; i < (R + 31) / 32; ++i) {
                const int r = (tid >> 3) + 32 * i;
                if (r < R)
                    *reinterpret_cast<float4*>(qs + r * AT_QP + (tid & 7) * 4) =
                        make_float4(qnext[4 * i], qnext[4 * i + 1], qnext[4 * i + 2], qnext[4 * i + 3]);
            }
            __syncthreads();
            if (ch + 1 < n_ch) fetch_k(pass, ch + 1);
            else if (pass + 1 < kp) fetch_k(pass + 1, 0);
            times_groups<TR, 1>(acc, qs + rg * AT_QP, AT_QP, tile + lane, min(AT_CH, dk - ch * AT_CH), kg);
        }
#pragma unroll
        for (int r = 0; r < TR; ++r)
#pragma unroll
            for (int g = 0; g < AT_COLS; ++g) {
                const int key = pass * keys + 32 * g + lane;
                if (g < kg && key < Tn) prob[(rg + r) * pitch + key] = acc[r][g];
            }
    }
    // ---- softmax: the rows of this warp, whose scores it has written itself ----
    const T* vb = v + base;
    const int n_jt = (Tn + AT_CH - 1) / AT_CH, chans = 32 * vg;
    // a thread's part of a chunk: eight channels 8 (tid % 8 + 8 i) .. of token tid / 8
    const int lj = tid >> 3;
    auto fetch_v = [&](int pass, int jt) {
        const T* vr = vb + (long long)min(jt * AT_CH + lj, Tn - 1) * D;
#pragma unroll
        for (int i = 0; i < (32 * AT_COLS + 63) / 64; ++i) {
            const int c = 8 * ((tid & 7) + 8 * i);
            if (c < chans) load_eight<T>(next[i], vr, min(pass * chans + c, dk), dk, vec);
        }
    };
    fetch_v(0, 0);
    __syncwarp();
#pragma unroll 1
    for (int r = 0; r < TR; ++r) {
        float* pr = prob + (rg + r) * pitch;
        float m = -3.402823466e38f;
        for (int j = lane; j < Tn; j += 32) m = fmaxf(m, pr[j]);
        for (int off = 16; off; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
        float sum = 0.f;
        for (int j = lane; j < Tn; j += 32) {
            const float e = expf(pr[j] - m);
            pr[j] = e;
            sum += e;
        }
        for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) inv[rg + r] = 1.0f / sum;
    }
    // ---- output ----
    for (int pass = 0; pass < vp; ++pass) {
        clear();
        for (int jt = 0; jt < n_jt; ++jt) {
            __syncthreads();
#pragma unroll
            for (int i = 0; i < (32 * AT_COLS + 63) / 64; ++i) {
                const int c = 8 * ((tid & 7) + 8 * i);
                if (c < chans) {
                    float* to = tile + lj * chans + c;
                    *reinterpret_cast<float4*>(to) = make_float4(next[i][0], next[i][1], next[i][2], next[i][3]);
                    *reinterpret_cast<float4*>(to + 4) = make_float4(next[i][4], next[i][5], next[i][6], next[i][7]);
                }
            }
            __syncthreads();
            if (jt + 1 < n_jt) fetch_v(pass, jt + 1);
            else if (pass + 1 < vp) fetch_v(pass + 1, 0);
            times_groups<TR, 0>(acc, prob + rg * pitch + jt * AT_CH, pitch, tile + lane, min(AT_CH, Tn - jt * AT_CH), vg);
        }
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            if (rg + r < n_rows) {
                T* to = o + base + (row0 + rg + r) * D;
                const float s = inv[rg + r];
#pragma unroll
                for (int g = 0; g < AT_COLS; ++g) {
                    const int c = pass * chans + 32 * g + lane;
                    if (g < vg && c < dk) to[c] = from_f32<T>(acc[r][g] * s);
                }
            }
        }
    }
}

size_t tile_smem(int Tn, int dk, int R) {
    const int groups = tile_groups(Tn) > tile_groups(dk) ? tile_groups(Tn) : tile_groups(dk);
    return ((size_t)R * AT_QP + (size_t)R * ((Tn + 3) / 4 * 4 + 4) + R + (size_t)AT_CH * (32 * groups + 1)) * sizeof(float);
}

template <typename T, int TR>
int launch_tile(const void* q, const void* k, const void* v, void* o, int B, int Tn, int H, int dk, float scale, cudaStream_t st) {
    const size_t smem = tile_smem(Tn, dk, 8 * TR);
    auto kern = attention_tile_kernel<T, TR>;
    CONVNN_ENSURE_SMEM(kern, smem);
    const int vec = dk % 8 == 0 && aligned16(k) && aligned16(v);         // (rows of a multiple of eight values)
    launch_chained(kern, dim3((Tn + 8 * TR - 1) / (8 * TR), B * H), AT_THREADS, smem, st, static_cast<const T*>(q),
                   static_cast<const T*>(k), static_cast<const T*>(v), static_cast<T*>(o), Tn, H, dk, scale, vec);
    CONVNN_CHECK_LAUNCH("attention_tile");
    return CONVNN_OK;
}

// One warp per query row; scores in shared memory.  Sequences too long for a tile of rows, and short ones of many heads.
template <typename T>
__global__ void attention_simt_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                                      T* __restrict__ o, int Tn, int H, int dk, float scale) {
    chain_begin_for<T>();
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    float* prob = sm + warp * (Tn + dk);
    float* qrow = prob + Tn;
    const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
    const long long D = (long long)H * dk;
    const T* kb = k + (long long)b * Tn * D + h * dk;
    const T* vb = v + (long long)b * Tn * D + h * dk;
    for (int row = blockIdx.x * nw + warp; row < Tn; row += gridDim.x * nw) {
        const T* qr = q + ((long long)b * Tn + row) * D + h * dk;
        for (int c = lane; c < dk; c += 32) qrow[c] = to_f32(qr[c]) * scale;
        __syncwarp();
        float m = -3.402823466e38f;
        for (int j = lane; j < Tn; j += 32) {
            const T* kr = kb + (long long)j * D;
            float s = 0.f;
            for (int c = 0; c < dk; ++c) s = fmaf(qrow[c], to_f32(kr[c]), s);
            prob[j] = s;
            m = fmaxf(m, s);
        }
        for (int off = 16; off; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
        float sum = 0.f;
        for (int j = lane; j < Tn; j += 32) {
            const float e = expf(prob[j] - m);
            prob[j] = e;
            sum += e;
        }
        for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        __syncwarp();
        const float inv = 1.0f / sum;
        T* orow = o + ((long long)b * Tn + row) * D + h * dk;
        for (int c = lane; c < dk; c += 32) {
            float acc = 0.f;
            for (int j = 0; j < Tn; ++j) acc = fmaf(prob[j], to_f32(vb[(long long)j * D + c]), acc);
            orow[c] = from_f32<T>(acc * inv);
        }
        __syncwarp();
    }
}

int pow2_at_least(int v, int lo) {
    int r = lo;
    while (r < v) r <<= 1;
    return r;
}

bool attention_tc_ok(int dtype, const void* q, const void* k, const void* v, const void* o, int Tn, int D, int H) {
    const int dk = D / H;
    return dtype == CONVNN_BF16 && !force_simt() && Tn <= 256 && dk % 16 == 0 && dk <= 128 && aligned16(q) &&
           aligned16(k) && aligned16(v) && aligned16(o);
}

int launch_attention_tc(const void* q, const void* k, const void* v, void* o, int B, int Tn, int D, int H,
                        cudaStream_t st, bool beside) {
    AttnParams p{};
    p.o = static_cast<__nv_bfloat16*>(o);
    p.T = Tn; p.H = H; p.dk = D / H; p.D = D;
    p.KCH = p.dk % 64 == 0 ? 64 : (p.dk % 32 == 0 ? 32 : 16);
    p.KC = p.dk / p.KCH;
    p.BN = (Tn + 15) / 16 * 16;
    p.BNpad = pow2_at_least(p.BN > p.dk ? p.BN : p.dk, 32);
    p.NKC2 = (p.BN + 63) / 64;
    p.n_row_tiles = (Tn + BM - 1) / BM;
    p.n_units = B * H * p.n_row_tiles;
    p.scale_log2 = (float)(1.4426950408889634 / sqrt((double)p.dk));
    const int pitch = p.KCH * 2;
    const size_t qk_bytes = (size_t)p.KC * (BM + p.BN) * pitch, pp_bytes = (size_t)p.NKC2 * 16384;
    p.p_region_bytes = (uint32_t)(((qk_bytes > pp_bytes ? qk_bytes : pp_bytes) + 1023) & ~(size_t)1023);
    const size_t smem = 1024 + p.p_region_bytes + (size_t)p.NKC2 * p.dk * 128 + (((size_t)p.BN * p.dk * 2 + 15) & ~(size_t)15) +
                        7 * 8 + 16;
    if (smem > 227 * 1024) return set_error(CONVNN_E_UNSUPPORTED, "attention_tc: shape needs %zu bytes of shared memory", smem);

    CUtensorMap tmQ, tmK, tmV;
    const uint64_t dims[4] = {(uint64_t)p.dk, (uint64_t)H, (uint64_t)Tn, (uint64_t)B};
    const uint64_t str[3] = {(uint64_t)p.dk * 2, (uint64_t)D * 2, (uint64_t)Tn * D * 2};
    const uint32_t boxQ[4] = {(uint32_t)p.KCH, 1, (uint32_t)BM, 1};
    const uint32_t boxK[4] = {(uint32_t)p.KCH, 1, (uint32_t)p.BN, 1};
    const uint32_t boxV[4] = {(uint32_t)p.dk, 1, (uint32_t)p.BN, 1};
    if (!encode_tensor_map_bf16(&tmQ, q, 4, dims, str, boxQ, pitch)) return CONVNN_E_CUDA;
    if (!encode_tensor_map_bf16(&tmK, k, 4, dims, str, boxK, pitch)) return CONVNN_E_CUDA;
    if (!encode_tensor_map_bf16(&tmV, v, 4, dims, str, boxV, 0)) return CONVNN_E_CUDA;

    const int sms = device_sms();
    const int per_sm = smem <= 113 * 1024 && p.BNpad <= 256 ? 2 : 1;
    const int ctas = sms * per_sm;
    const int grid = p.n_units < ctas ? p.n_units : ctas;
    if (beside) {
        CONVNN_ENSURE_SMEM(attention_tc_kernel<true>, smem);
        launch_chained(attention_tc_kernel<true>, grid, NTHREADS, smem, st, tmQ, tmK, tmV, p);
    } else {
        CONVNN_ENSURE_SMEM(attention_tc_kernel<false>, smem);
        launch_chained(attention_tc_kernel<false>, grid, NTHREADS, smem, st, tmQ, tmK, tmV, p);
    }
    CONVNN_CHECK_LAUNCH("attention_tc");
    return CONVNN_OK;
}

// Sequences of up to 20 tokens (28 of many narrow bfloat16 heads): a tile of `rows` rows takes its chain of chunks whatever it holds,
// two at a time on an SM, while a warp per row waits for one row's dot products and shares the SM with many.  us of both, fits to 190
// and 221 shapes of 2 to 40 tokens (rms 10 %) and 150 of up to 26 (18 %); the choice costs 0.3 % over the better of the two on average.
// Tile -> row per warp, us of the attention alone: 4854 heads of 2 tokens x 8 70.9 -> 6.9, 1551 x 2 x 24 24.9 -> 4.1, 5904 x 2 x 192 225 -> 39,
// 3730 x 4 x 40 71 -> 13.7, 3978 x 7 x 24 60 -> 22, 4608 x 9 x 24 91 -> 37; few heads, 120 x 2 x 8 5.0 -> 2.9; bfloat16 with the projections 4205 x 20 x
// 24 170 -> 114, 1188 x 26 x 8 55 -> 43.  The other way 108 x 9 x 256 29 -> 18, 1440 x 10 x 160 115 -> 60, 585 x 15 x 160 116 -> 25, float32 3600 x 20
// x 32 190 -> 105.  (One token of few heads has the tile whatever it costs: 4 us.)
bool row_per_warp(int heads, int Tn, int dk, int rows, bool bf16) {
    if (rows == 0) return false;
    const long long tiles = (long long)heads * ((Tn + rows - 1) / rows), at_once = 2ll * device_sms();
    const bool narrow = bf16 && dk <= 64;
    if (Tn > (narrow && tiles > 3 * at_once ? 28 : 20) || (Tn == 1 && tiles <= at_once)) return false;
    const double round = rows == 8 ? 3.9 + 0.042 * dk : rows == 16 ? 4.5 + 0.048 * dk + 0.04 * Tn : 6.5 + 0.059 * dk + 0.077 * Tn;
    const double tile = round * ((tiles + at_once - 1) / at_once);
    const double chain = 2.7 + dk * (0.017 + 0.0077 * Tn);
    const double work = (narrow ? 0.65 : 1.0) * heads * Tn / device_sms() * (0.03 + dk * (0.0021 + 0.0004 * Tn));
    return chain * chain + work * work < (tiles <= at_once ? 0.8 : 1.1) * tile * tile;
}

template <typename T>
int launch_attention_simt_t(const void* q, const void* k, const void* v, void* o, int B, int Tn, int D, int H,
                            cudaStream_t st) {
    const int dk = D / H, nw = 4;
    const float scale = (float)(1.0 / sqrt((double)dk));
    // Rows per CTA: the fewest multiply-adds on the busiest SM, where a CTA costs its rows and, staging its chunks, twelve more, and a
    // round of two CTAs their chain of chunks.
    int rows = 0;
    long long least = 0;
    for (const int R : {56, 40, 16, 8}) {
        const long long n = ((long long)B * H * ((Tn + R - 1) / R) + device_sms() - 1) / device_sms(), cost = n * (R + 12) + (n + 1) / 2 * 32;
        if (tile_smem(Tn, dk, R) <= 200 * 1024 && (!rows || cost < least)) {
            rows = R;
            least = cost;
        }
    }
    if (row_per_warp(B * H, Tn, dk, rows, sizeof(T) == 2)) rows = 0;
    if (rows == 8) return launch_tile<T, 1>(q, k, v, o, B, Tn, H, dk, scale, st);
    if (rows == 16) return launch_tile<T, 2>(q, k, v, o, B, Tn, H, dk, scale, st);
    if (rows == 40) return launch_tile<T, 5>(q, k, v, o, B, Tn, H, dk, scale, st);
    if (rows == 56) return launch_tile<T, 7>(q, k, v, o, B, Tn, H, dk, scale, st);
    const size_t smem = (size_t)nw * (Tn + dk) * sizeof(float);
    if (smem > 200 * 1024)
        return set_error(CONVNN_E_UNSUPPORTED, "softmax attention over %d tokens is outside this build", Tn);
    auto kern = attention_simt_kernel<T>;
    CONVNN_ENSURE_SMEM(kern, smem);
    int gx = (Tn + nw - 1) / nw;
    if (gx > 64) gx = 64;
    launch_chained(kern, dim3(gx, B * H), nw * 32, smem, st, static_cast<const T*>(q), static_cast<const T*>(k),
                                                 static_cast<const T*>(v), static_cast<T*>(o), Tn, H, dk, scale);
    CONVNN_CHECK_LAUNCH("attention_simt");
    return CONVNN_OK;
}

}  // namespace

// q, k, v, o: (B, T, H, d_k) = (B*T, D) row-major in `dtype`.
int launch_attention(int dtype, const void* q, const void* k, const void* v, void* o, int B, int Tn, int D, int H,
                     cudaStream_t st, bool beside) {
    if (attention_tc_ok(dtype, q, k, v, o, Tn, D, H)) return launch_attention_tc(q, k, v, o, B, Tn, D, H, st, beside);
    if (dtype == CONVNN_F32) return launch_attention_simt_t<float>(q, k, v, o, B, Tn, D, H, st);
    return launch_attention_simt_t<__nv_bfloat16>(q, k, v, o, B, Tn, D, H, st);
}

int read_attention_status(int* out) {
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_attention_status, sizeof(int));
    if (e != cudaSuccess) return set_error(CONVNN_E_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    *out = v;
    return CONVNN_OK;
}

}  // namespace convnn
