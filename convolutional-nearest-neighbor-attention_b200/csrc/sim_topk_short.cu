// Similarity + top-K for short candidate lists (S <= 256): a row's whole similarity vector is one accumulator in tensor
// memory, so the selection can read it twice.
//
//   pass 1  a bound: the maxima of 32 groups of columns (lists of up to twelve: sixteen per half of a row, column modulo 16) or 64
//           (longer lists) are sorted by networks; the nsel-th largest of them is a key that at least nsel columns reach.
//   pass 2  the columns whose key reaches the bound (of 197 about 10 for K = 9, 29 for K = 25) are appended, in column order, to the
//           row's entries in shared memory, without a branch on how many there are.
//   rank    a network sorts the entries (packed_rank.cuh); the earlier column wins ties.
//           A row with more entries than it has room for takes, if its list is long, the nsel-th largest of those it has as its bound
//           and repeats pass 2 (some 47 of 256 columns reach the first bound for K = 32, 3 more or less, where there is room for 51);
//           where that does not do either (ties), and short lists at once, the columns above the bound chunk by chunk, 15 us more.
//
// The results are the streaming kernels' bit for bit.
//
// What bounds it (128 images of 12 heads, 197 x 197 x 32, K = 9, 79 us; the streaming kernel 136): instructions, half of them on the half-rate
// pipe, and their fetch: with the entries inserted into a sorted list and written a word at a time 93; a chunk loop unrolled once more 125 for 106,
// the metric known at compile time 96 for 106, tensor-memory reads one chunk ahead nothing.  (18 warps of 96 registers:
// one thread per row spills 16 to 64 bytes.)  Lists of more than twelve have one thread per row, eight warps, and wait as much as they
// issue (0.31 instructions per cycle and scheduler); us, a sorted list of values as the bound or the streaming kernel -> groups and a
// network: 57 x 12 heads of 197 x 197 x 32, K = 25 171 -> 85; 256 x 197 x 197 x 192, K = 25 70 -> 36, K = 16 50 -> 26; 256 x 577 x 150 x 384,
// K = 16 107 -> 67.  Streaming -> this kernel, K = 9: 256 images of 197 x 192 30.5 -> 20.9 (K = 4: 22.8 -> 15.8), 6 heads of 64 126 -> 82,
// 65 x 65 x 192 12.5 -> 9.2, 1024 x 65 x 65, 3 heads of 64 94 -> 41, 64 x 1000 x 200 x 256 33 -> 25, 256 x 197 x 64 x 384 17.8 -> 15.9.
//
// A persistent CTA per SM: warp 0 TMA producer (128 key rows + all candidate rows of one (batch, head), 64-channel chunks,
// ring), warp 1 MMA issuer (M = 128, N = S rounded to 16), then selection warps (thread = row).  G accumulators of 512 / G
// columns, G = 4 for S <= 128 (narrow heads only, lists of up to nine), else 2, so the next units' MMAs run under the selection.  With NH = 2 two warps share a row
// block of an accumulator, a column half each: the bound follows from their two sorted lists (the n-th largest of
// a and b is the largest min(a[i], b[n-2-i])), their entries grow towards each other, and they take turns at ranking.
#include "common.cuh"
#include "sm100.cuh"
#include "toplist.cuh"
#include "sim_topk_select.cuh"
#include "packed_rank.cuh"

namespace convnn {

__device__ int g_sim_short_status = 0;

namespace {

using namespace sm100;

constexpr int BM = 128;
constexpr int MAX_STAGES = 6;

struct ShortParams {
    const float* qstat;
    const float* kstat;
    const int32_t* cand;
    int32_t* idx;
    float* val;
    int T, S, H, K, nsel, metric, sampled;
    int KCH, KC;      // channels per shared-memory chunk, chunks per unit
    int BN;           // S rounded up to 16
    int stages, n_row_tiles, n_units;
    float sqrt_dk;
};

__device__ __forceinline__ void fail(volatile int* abort_flag, int code) {
    *abort_flag = 1;
    atomicCAS(&g_sim_short_status, 0, code);
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_x32(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld_x16(taddr, r); }

// Ranking keys of W accumulator columns from `col0` on; -inf past the last candidate.
// METRIC < 0: p.metric.  CLOSED: the statistics past the last candidate are NaN, and so are the keys (MATMUL has none).
template <int W, int METRIC = -1, bool CLOSED = false>
__device__ __forceinline__ void make_keys(float (&key)[W], const uint32_t (&acc)[W], const float* qs, const int* cs, int col0,
                                          const ShortParams& p, int row, float sentinel) {
    const int metric = METRIC < 0 ? p.metric : METRIC;
    if (metric != CONVNN_MATMUL) {
        const f32x2 two = pack2(2.0f, 2.0f);
#pragma unroll
        for (int j4 = 0; j4 < W / 4; ++j4) {
            const float4 s4 = *reinterpret_cast<const float4*>(qs + col0 + 4 * j4);
            const f32x2 d01 = pack2(__uint_as_float(acc[4 * j4]), __uint_as_float(acc[4 * j4 + 1]));
            const f32x2 d23 = pack2(__uint_as_float(acc[4 * j4 + 2]), __uint_as_float(acc[4 * j4 + 3]));
            f32x2 k01, k23;
            if (metric == CONVNN_COSINE) {
                k01 = mul2(d01, pack2(s4.x, s4.y));
                k23 = mul2(d23, pack2(s4.z, s4.w));
            } else {
                k01 = fma2(two, d01, pack2(-s4.x, -s4.y));
                k23 = fma2(two, d23, pack2(-s4.z, -s4.w));
            }
            unpack2(k01, key[4 * j4], key[4 * j4 + 1]);
            unpack2(k23, key[4 * j4 + 2], key[4 * j4 + 3]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < W; ++j) key[j] = __uint_as_float(acc[j]);
    }
    if (p.sampled) {
#pragma unroll
        for (int j4 = 0; j4 < W / 4; ++j4) {
            const int4 c4 = *reinterpret_cast<const int4*>(cs + col0 + 4 * j4);
            if (c4.x == row) key[4 * j4] = sentinel;
            if (c4.y == row) key[4 * j4 + 1] = sentinel;
            if (c4.z == row) key[4 * j4 + 2] = sentinel;
            if (c4.w == row) key[4 * j4 + 3] = sentinel;
        }
    }
    if (CLOSED && metric != CONVNN_MATMUL) return;
    const int left = p.S - col0;
    if (left < W) {
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j >= left) key[j] = -CUDART_INF_F;
    }
}

// Lists of more than twelve are ranked by a network (one thread per row); the entries a row has room for (checked every eight columns).
// 59 leave the ring two stages of 64 channels with 256 candidates, 60 one (us, one stage and no second bound -> two and a second bound:
// 87 images of 256 x 256 x 128, K = 30 38.8 -> 25.4, 105 x 2 x 242 x 242 x 192, K = 26 45 -> 41; 68 x 243 x 243 x 192, K = 32 40 -> 27, 10 x 6 heads of 239 x
// 239 x 128 38 -> 26; sorted lists of values 33).
template <int NSEL>
constexpr bool networked = NSEL > 12;
template <int NSEL, int NH>
constexpr int slots_of = NSEL <= 12 ? (NH == 2 ? 28 : 32) : NSEL <= 16 ? 36 : NSEL <= 25 ? 52 : 59;

template <int NSEL, int G, int NH, int METRIC, Way WAY>
__global__ void __launch_bounds__(64 + 128 * G * NH, 1)
sim_topk_short_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ, const ShortParams p) {
    constexpr int MAXC = 512 / G;                  // tensor-memory columns of one accumulator
    constexpr int NT = 128 * G * NH;               // selection threads
    constexpr int W = G == 4 ? 16 : 32;            // columns per read of a long list's first pass (18 warps leave 96 registers per thread)
    constexpr uint32_t ENTRY = 32 * 8;             // bytes between a row's successive entries
    constexpr int SLOTS = slots_of<NSEL, NH>;
    constexpr bool NETWORK = networked<NSEL>;
    static_assert(!NETWORK || NH == 1, "rows of long lists are one thread's");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t pitch = p.KCH * 2;
    const uint32_t a_bytes = BM * pitch, b_bytes = p.BN * pitch, stage_bytes = a_bytes + b_bytes;
    const uint32_t STAGES = p.stages;
    float2* hits = reinterpret_cast<float2*>(smem + STAGES * stage_bytes);       // [4 G blocks of rows][SLOTS][32] (key, column)
    float* statbuf = reinterpret_cast<float*>(hits + SLOTS * 128 * G);      // [warps][MAXC] column statistics
    int* cs = reinterpret_cast<int*>(statbuf + NT / 32 * MAXC);                  // [MAXC] candidate tokens
    float* lists = reinterpret_cast<float*>(cs + MAXC);                          // short lists: [NSEL][NT] sorted keys
    int* counts = reinterpret_cast<int*>(lists + (NETWORK ? 0 : NSEL * NT));       // NH = 2: [NT] entries
    uint64_t* full = reinterpret_cast<uint64_t*>(counts + (NH == 2 ? NT : 0));
    uint64_t* empty = full + MAX_STAGES;
    uint64_t* tfull = empty + MAX_STAGES;
    uint64_t* tempty = tfull + G;
    uint64_t* xlist = tempty + G;                  // NH = 2, per (accumulator, lane quarter): both lists written
    uint64_t* xhits = xlist + 4 * G;               //                                          both sets of entries written
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xhits + 4 * G);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < G; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 4 * NH);
        }
        for (int b = 0; b < 4 * G; ++b) {
            mbar_init(&xlist[b], 2);
            mbar_init(&xhits[b], 2);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmK);
        prefetch_tensormap(&tmQ);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_begin();

    const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), st0 = smem_u32(smem);
    if (warp == 0) {
        {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x) {
                const int bh = unit / p.n_row_tiles, rt = unit - bh * p.n_row_tiles;
                const int b = bh / p.H, h = bh - b * p.H;
                for (int kc = 0; kc < p.KC; ++kc) {
                    ok = mbar_wait_warp(empty0 + 8 * s, ph ^ 1u, abort_flag);
                    if (!ok) { if (lane == 0) fail(abort_flag, 71); break; }
                    const uint32_t st = st0 + s * stage_bytes, fb = full0 + 8 * s;
                    if (elect_one()) {
                        mbar_expect_tx_a(fb, stage_bytes);
                        tma_load_4d_a(st, &tmK, fb, kc * p.KCH, h, rt * BM, b);
                        tma_load_4d_a(st + a_bytes, &tmQ, fb, kc * p.KCH, h, 0, b);
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc = make_idesc_bf16_f32(BM, p.BN);
            const uint64_t dhi = kmajor_desc_hi(pitch);
            const int nk16 = p.KCH / 16;
            const uint32_t tfull0 = smem_u32(tfull), tempty0 = smem_u32(tempty);
            uint32_t s = 0, ph = 0, buf = 0, use = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x) {
                if (!mbar_wait_warp(tempty0 + 8 * buf, (use & 1u) ^ 1u, abort_flag)) { fail(abort_flag, 72); break; }
                tc_fence_after_sync();
                for (int kc = 0; kc < p.KC; ++kc) {
                    if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag)) { fail(abort_flag, 73); ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t sa = st0 + s * stage_bytes;
                    if (elect_one()) {
                        mma_chunk(tmem_base + buf * MAXC, dhi | (uint64_t)(sa >> 4), dhi | (uint64_t)((sa + a_bytes) >> 4), idesc, nk16,
                                  kc != 0);
                        mma_commit_a(empty0 + 8 * s);
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
                if (ok && elect_one()) mma_commit_a(tfull0 + 8 * buf);
                if (++buf == G) { buf = 0; ++use; }
            }
        }
    } else {
        const int g = (warp - 2) / (4 * NH);         // accumulator this warp serves
        const int half = NH == 2 ? ((warp - 2) >> 2) & 1 : 0;
        const int lq = warp & 3;                     // TMEM lane quarter it may read
        const int r = lq * 32 + lane;
        const int tid = threadIdx.x - 64, peer = NH == 2 ? (tid ^ 128) : tid;   // the other half's thread of this row
        const int xb = g * 4 + lq;
        float* qs = statbuf + (warp - 2) * MAXC;
        // entries of a row: the lower half's upwards from slot 0, the upper half's downwards from the last; more than there are
        // slots are marked with a count that no row has room for.
        float2* own = hits + (g * 4 + lq) * (SLOTS * 32) + lane;
        const uint32_t hit0 = smem_u32(own), block0 = hit0 - lane * 8u;
        const int c_begin = half ? ((p.S + 1) / 2 + 15) / 16 * 16 : 0;
        const int c_end = NH == 2 && !half ? min(((p.S + 1) / 2 + 15) / 16 * 16, p.S) : p.S;
        const uint32_t taddr = tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)g * MAXC;
        if (p.sampled)                               // (every warp writes the same values)
            for (int c = lane; c < MAXC; c += 32) cs[c] = c < p.S ? p.cand[c] : -1;
        uint32_t use = 0, use_of_pair = 0;           // (a row block past the sequence takes no part in an exchange)
        bool ok = true;
        for (int unit = blockIdx.x + g * gridDim.x; unit < p.n_units && ok; unit += G * gridDim.x, ++use) {
            const int bh = unit / p.n_row_tiles, rt = unit - bh * p.n_row_tiles;
            const int row = rt * BM + r;
            const bool row_ok = row < p.T;
            const bool warp_live = rt * BM + lq * 32 < p.T;
            const bool ranks = NH == 1 || (int)(use & 1u) == half;
            float kst = 1.0f;
            if (row_ok && p.metric != CONVNN_MATMUL) kst = p.kstat[(long long)bh * p.T + row];
            const float sentinel = p.sampled ? self_sentinel(p.metric, kst, p.sqrt_dk) : 0.f;
            __syncwarp();
            if (p.metric != CONVNN_MATMUL) {
                const float* qrow = p.qstat + (long long)bh * p.S;
#pragma unroll
                for (int c = 0; c < MAXC; c += 32) qs[c + lane] = c + lane < p.S ? qrow[c + lane] : CUDART_NAN_F;
            }
            __syncwarp();
            ok = mbar_wait(&tfull[g], use & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) { if (lane == 0) fail(abort_flag, 74); break; }
            tc_fence_after_sync();
            if constexpr (!NETWORK) {
                bool insert = false;
                int n_low = 0, cnt = 0;
                if (warp_live) {
                    // Pass 1: maxima of column groups, sixteen per half of a row (NH = 1: of the even and the odd chunks).
                    float v[16], w[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = w[j] = -CUDART_INF_F;
                    auto into = [&](float (&m)[16], int c) {
                        uint32_t acc[16];
                        tmem_ld_x16(taddr + c, acc);
                        tmem_ld_wait();
                        float key[16];
                        make_keys<16, METRIC, true>(key, acc, qs, cs, c, p, row, sentinel);
#pragma unroll
                        for (int j = 0; j < 16; ++j) m[j] = fmaxf(m[j], key[j]);
                    };
#pragma unroll 1
                    for (int c = c_begin; c < c_end; c += NH == 2 ? 16 : 32) {
                        into(v, c);
                        if (NH == 1 && c + 16 < c_end) into(w, c + 16);
                    }
                    sort_descending(v);
                    if (NH == 1) sort_descending(w);
#pragma unroll
                    for (int s = 0; s < NSEL; ++s) lists[s * NT + tid] = NH == 1 ? w[s] : v[s];
                    if (NH == 2) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&xlist[xb]);
                        ok = mbar_wait(&xlist[xb], use_of_pair & 1u, abort_flag);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) { if (lane == 0) fail(abort_flag, 75); break; }
                    }
                    // the nsel-th largest of both lists
                    float thr = v[0];
#pragma unroll
                    for (int s = 1; s < NSEL; ++s) thr = fminf(thr, s < p.nsel ? v[s] : CUDART_INF_F);
                    thr = fmaxf(thr, lists[(p.nsel - 1) * NT + peer]);
#pragma unroll
                    for (int i = 0; i < NSEL - 1; ++i)
                        if (i < p.nsel - 1) thr = fmaxf(thr, fminf(v[i], lists[(p.nsel - 2 - i) * NT + peer]));
                    insert = !(thr > -CUDART_INF_F) || !(fmaxf(v[0], lists[peer]) < CUDART_INF_F);
                    // Pass 2: the columns that reach it.
                    constexpr int ROOM = SLOTS - 8;
                    const uint32_t first = half ? hit0 + (SLOTS - 1) * ENTRY : hit0;
                    const uint32_t step = half ? 0u - ENTRY : ENTRY;
                    uint32_t at = first;
                    bool over = false;
#pragma unroll 1
                    for (int c = c_begin; c < c_end; c += 16) {
                        uint32_t acc[16];
                        tmem_ld_x16(taddr + c, acc);
                        tmem_ld_wait();
                        float key[16];
                        make_keys<16, METRIC, true>(key, acc, qs, cs, c, p, row, sentinel);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            if (j % 8 == 0) {
                                const bool full_up = (half ? first - at : at - first) > ROOM * ENTRY;
                                over = over || full_up;
                                at = full_up ? first + ROOM * step : at;
                            }
                            if (key[j] >= thr) {
                                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(__float_as_uint(key[j])), "r"(c + j)
                                             : "memory");
                                at += step;
                            }
                        }
                    }
                    cnt = (int)((half ? first - at : at - first) / ENTRY);
                    if (over) cnt = SLOTS + 1;
                    n_low = cnt;
                    if (NH == 2) {
                        counts[tid] = cnt;
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&xhits[xb]);
                        if (ranks) {
                            ok = mbar_wait(&xhits[xb], use_of_pair & 1u, abort_flag);
                            ok = __all_sync(0xffffffffu, ok);
                            if (!ok) { if (lane == 0) fail(abort_flag, 76); break; }
                            const int other = counts[peer];
                            n_low = half ? other : cnt;
                            cnt += other;
                        }
                        ++use_of_pair;
                    }
                    if (!row_ok) cnt = 0;
                    const bool redo = cnt > SLOTS;
                    if (ranks && __any_sync(0xffffffffu, redo)) {
                        // More columns reach the bound than a row has room for: chunk by chunk into the list.
                        TopList<NSEL> top;
                        top.init();
                        const float floor = just_below(thr);
#pragma unroll 1
                        for (int c = 0; c < p.S; c += 16) {
                            uint32_t acc[16];
                            tmem_ld_x16(taddr + c, acc);
                            tmem_ld_wait();
                            float key[16];
                            make_keys<16, METRIC, true>(key, acc, qs, cs, c, p, row, sentinel);
                            const float low = fmaxf(top.worst(), floor);
                            uint32_t mask = 0;
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                mask |= key[j] > low ? 1u << j : 0u;
                                if (redo) own[j * 32].x = key[j];
                            }
                            if (!redo) mask = 0;
                            const int steps = __reduce_max_sync(0xffffffffu, __popc(mask));
                            for (int it = 0; it < steps; ++it) {
                                const int j = mask ? __ffs(mask) - 1 : 0;
                                const float kc = own[j * 32].x;
                                if (mask && kc > top.worst()) top.insert_sorted(kc, c + j);
                                mask &= mask - 1;
                            }
                        }
                        if (redo) {                  // its list is its entries
#pragma unroll
                            for (int s = 0; s < NSEL; ++s)
                                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(hit0 + s * ENTRY),
                                             "r"(__float_as_uint(top.v[s])), "r"(top.i[s]) : "memory");
                            n_low = cnt = p.nsel;
                            insert = true;
                        }
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[g]);
                if (ranks && warp_live) {
                    // The n-th entry in column order.
                    auto entry = [&](int n) { return hit0 + (NH == 1 || n < n_low ? n : SLOTS - 1 + n_low - n) * ENTRY; };
                    TopList<NSEL> top;
                    rank_entries<NSEL>(top, entry, cnt, p.nsel, insert);
                    write_rows<NSEL, WAY>(top, p, cs, block0, ((long long)bh * p.T + rt * BM + lq * 32) * p.K,
                                     min(32, p.T - rt * BM - lq * 32), row, kst);
                }
            } else {
                uint32_t at = hit0;
                bool redo = false;
                if (warp_live) {
                    // Pass 1: maxima of 64 column groups, 32 of the even chunks of 32 columns and 32 of the odd ones.
                    float thr = -CUDART_INF_F, largest = -CUDART_INF_F;
                    {
                        float v[32];
#pragma unroll 1
                        for (int odd = 0; odd < 2; ++odd) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = -CUDART_INF_F;
#pragma unroll 1
                            for (int c = 32 * odd; c < p.S; c += 64) {
#pragma unroll
                                for (int w = 0; w < 32; w += W) {
                                    uint32_t acc[W];
                                    tmem_ld(taddr + c + w, acc);
                                    tmem_ld_wait();
                                    float key[W];
                                    make_keys<W, METRIC, true>(key, acc, qs, cs, c + w, p, row, sentinel);
#pragma unroll
                                    for (int j = 0; j < W; ++j) v[w + j] = fmaxf(v[w + j], key[j]);
                                }
                            }
                            sort_descending(v);
                            largest = fmaxf(largest, v[0]);
                            if (odd) break;
#pragma unroll
                            for (int s = 0; s < NSEL; ++s)       // (into the row's own, still empty slots)
                                asm volatile("st.shared.f32 [%0], %1;" ::"r"(hit0 + s * ENTRY), "f"(v[s]) : "memory");
                        }
                        // the nsel-th largest of both
                        thr = v[0];
#pragma unroll
                        for (int s = 1; s < NSEL; ++s) thr = fminf(thr, s < p.nsel ? v[s] : CUDART_INF_F);
                        auto of_even = [&](int s) {
                            float x;
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(hit0 + s * ENTRY) : "memory");
                            return x;
                        };
                        thr = fmaxf(thr, of_even(p.nsel - 1));
#pragma unroll
                        for (int i = 0; i < NSEL - 1; ++i)
                            if (i < p.nsel - 1) thr = fmaxf(thr, fminf(v[i], of_even(p.nsel - 2 - i)));
                    }
                    // Pass 2: the columns that reach it.  A row that has no room for them all takes the nsel-th largest of those it has
                    // room for as its bound, which nsel columns reach too, and once more the columns that reach that.
                    constexpr int FULL = SLOTS - 8;
                    constexpr uint32_t ROOM = FULL * ENTRY;
                    bool over;
#pragma unroll 1
                    for (int attempt = 0;; ++attempt) {
                        over = false;
                        at = hit0;
#pragma unroll 1
                        for (int c = 0; c < p.S; c += 16) {
                            uint32_t acc[16];
                            tmem_ld_x16(taddr + c, acc);
                            tmem_ld_wait();
                            float key[16];
                            make_keys<16, METRIC, true>(key, acc, qs, cs, c, p, row, sentinel);
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                if (j % 8 == 0) {
                                    over = over || at > hit0 + ROOM;
                                    at = min(at, hit0 + ROOM);
                                }
                                if (key[j] >= thr) {
                                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(__float_as_uint(key[j])), "r"(c + j)
                                                 : "memory");
                                    at += ENTRY;
                                }
                            }
                        }
                        over = over || at > hit0 + ROOM;
                        if (attempt == 1 || !__any_sync(0xffffffffu, over && row_ok)) break;
                        float q[FULL];
#pragma unroll
                        for (int n = 0; n < FULL; ++n) q[n] = lds_key(hit0 + n * ENTRY);
                        sort_descending(q);
                        float tight = q[0];
#pragma unroll
                        for (int s = 1; s < NSEL; ++s) tight = fminf(tight, s < p.nsel ? q[s] : CUDART_INF_F);
                        if (over) thr = fmaxf(thr, tight);
                    }
                    // Too many of them (ties), fewer than nsel keys above -inf (NaN inputs), keys of +inf: the row takes the columns
                    // above the bound chunk by chunk.
                    redo = row_ok && (over || !(thr > -CUDART_INF_F) || !(largest < CUDART_INF_F));
                    if (!row_ok) at = hit0;
                    if (__any_sync(0xffffffffu, redo)) {
                        TopList<NSEL> top;
                        top.init();
                        const float floor = just_below(thr);
#pragma unroll 1
                        for (int c = 0; c < p.S; c += 16) {
                            uint32_t acc[16];
                            tmem_ld_x16(taddr + c, acc);
                            tmem_ld_wait();
                            float key[16];
                            make_keys<16, METRIC, true>(key, acc, qs, cs, c, p, row, sentinel);
                            const float low = fmaxf(top.worst(), floor);
                            uint32_t mask = 0;
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                mask |= key[j] > low ? 1u << j : 0u;
                                if (redo) own[j * 32].x = key[j];
                            }
                            if (!redo) mask = 0;
                            const int steps = __reduce_max_sync(0xffffffffu, __popc(mask));
                            for (int it = 0; it < steps; ++it) {
                                const int j = mask ? __ffs(mask) - 1 : 0;
                                const float kc = own[j * 32].x;
                                if (mask && kc > top.worst()) top.insert_sorted(kc, c + j);
                                mask &= mask - 1;
                            }
                        }
                        if (redo) {                  // its list is its entries
#pragma unroll
                            for (int s = 0; s < NSEL; ++s)
                                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(hit0 + s * ENTRY),
                                             "r"(__float_as_uint(top.v[s])), "r"(top.i[s]) : "memory");
                            at = hit0 + p.nsel * ENTRY;
                        }
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[g]);
                if (warp_live) {
                    TopList<NSEL> top;
                    rank_entries<NSEL>(top, [&](int n) { return hit0 + n * ENTRY; }, (int)((at - hit0) / ENTRY), p.nsel, redo);
                    write_rows<NSEL, WAY>(top, p, cs, block0, ((long long)bh * p.T + rt * BM + lq * 32) * p.K,
                                     min(32, p.T - rt * BM - lq * 32), row, kst);
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // a wait expired: give copies still in flight time to land before the CTA's shared memory is released
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int NSEL, int G, int NH, int METRIC, Way WAY>
int launch_metric(const Dims& dm, ShortParams& p, const CUtensorMap& tmK, const CUtensorMap& tmQ, cudaStream_t st) {
    constexpr int MAXC = 512 / G;
    const size_t stage = (size_t)(BM + p.BN) * p.KCH * 2;
    constexpr int NT = 128 * G * NH;
    const size_t fixed = 1024 + (size_t)slots_of<NSEL, NH> * 128 * G * 8 + (size_t)(NT / 32 + 1) * MAXC * 4 +
                         (networked<NSEL> ? 0 : (size_t)(NSEL + 1) * NT * 4) + (2 * MAX_STAGES + 10 * G) * 8 + 16;
    p.stages = (int)((226 * 1024 - fixed) / stage);
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    if (p.stages > 2 * p.KC) p.stages = 2 * p.KC;            // deeper than two units' chunks serves nothing
    size_t smem = fixed + p.stages * stage;
    if (smem < 116 * 1024) smem = 116 * 1024;                // a CTA takes all of an SM's TMEM: never two on one SM
    const int sms = device_sms();
    auto kern = sim_topk_short_kernel<NSEL, G, NH, METRIC, WAY>;
    CONVNN_ENSURE_SMEM(kern, smem);
    launch_chained(kern, p.n_units < sms ? p.n_units : sms, 64 + NT, smem, st, tmK, tmQ, p);
    CONVNN_CHECK_LAUNCH("sim_topk_short");
    return CONVNN_OK;
}

template <int NSEL, int G, int NH, Way WAY>
int launch_way(const Dims& dm, ShortParams& p, const CUtensorMap& tmK, const CUtensorMap& tmQ, cudaStream_t st) {
    if (p.metric == CONVNN_COSINE) return launch_metric<NSEL, G, NH, CONVNN_COSINE, WAY>(dm, p, tmK, tmQ, st);
    if (p.metric == CONVNN_MATMUL) return launch_metric<NSEL, G, NH, CONVNN_MATMUL, WAY>(dm, p, tmK, tmQ, st);
    return launch_metric<NSEL, G, NH, CONVNN_EUCLIDEAN, WAY>(dm, p, tmK, tmQ, st);
}

// Short lists a word at a time cost a sector per word, by lines a pass through shared memory and code that few rows do not repay:
// K = 9, 128 x 12 x 197 x 197 x 32 91.5 -> 82.8 us, 64 x 1000 x 200 x 256 27.3 -> 24.8, 1024 x 3 x 65 x 65 x 64 46.7 -> 43.6; but 256 x 197 x
// 197 x 192 20.2 -> 20.4, 256 x 65 x 65 x 192 9.8 -> 10.3, K = 5, 700 x 197 x 197 x 32 35.4 -> 37.3.  Long ones, skewed: K = 25, 64 x 3 x 197 x 197 x 64 33.5 -> 29.4; 57 x 12 x 197 x
// 197 x 32 84 (by lines 85 to 87); K = 16, 256 x 577 x 150 x 384 75.7 -> 67.
template <int NSEL, int G, int NH>
int launch_short(const Dims& dm, ShortParams& p, const CUtensorMap& tmK, const CUtensorMap& tmQ, cudaStream_t st) {
    if constexpr (networked<NSEL>) {
        return launch_way<NSEL, G, NH, SKEWED>(dm, p, tmK, tmQ, st);
    } else {
        if constexpr (NSEL == 8 || NSEL == 9)
            if (dm.K % 2 == 1 && dm.K >= 9 && (long long)dm.B * dm.H * dm.T >= 384ll * device_sms())
                return launch_way<NSEL, G, NH, LINES>(dm, p, tmK, tmQ, st);
        return launch_way<NSEL, G, NH, WORDS>(dm, p, tmK, tmQ, st);
    }
}

}  // namespace

// What the warp-per-row kernel leaves to it.  Anything of up to one unit per SM (48 x 197 x 197 x 192, K = 25 33.8, 23.0); lists of more
// than twelve (streaming 256 x 577 x 150 x 384, K = 16 129, here 67; 57 x 12 x 197 x 197 x 32, K = 25 171, 84) except, beyond sixteen, where they hold most of up
// to 40 candidates and about half as many rounds of units stream (streaming, this kernel: 94 x 153 x 23 x 768, K = 20 13.8, 21.5; 143 x 172 x 38 x 32, K =
// 28 16.4, 19.4; 20 x 187 x 28 x 6 x 96, K = 28 14.5, 18.7; 32 x 574 x 18 x 3 x 512, K = 18 22.6, 30.7; 32 x 175 x 39 x 12 x 384, K = 27 44.7, 69.3; 316 x 131 x 27 x
// 256, K = 27 30, 36; but 77 x 685 x 47 x 32, K = 17 25.3, 15.8; 84 x 654 x 31 x 64, K = 17 21.1, 15.9; 47 x 886 x 36 x 256, K = 25 32, 28); lists of up to twelve except where the streaming kernel's 256-row units are fewer and the bound saves little (us, streaming, this kernel):
//   * few candidates: of sequences that fill more than one unit here (512 x 197 x 16 x 192, K = 4 10.8, 14.4; 256 x 197 x 32 x 768, K = 3
//     19.6, 21.9), and of others where heads are wide, lists long or the second round of units thin (1000 x 17 x 17 x 512, K = 2 19.5, 23.6;
//     200 x 100 x 20 x 384, K = 5 8.6, 9.6; 163 x 65 x 65 x 128, K = 12 13.4, 14.6; but 1000 x 17 x 17 x 64 0.65 of the time, 340 x 25 x 25 x 192 0.85, and
//     heads above 512 channels, which leave the streaming kernel one CTA per SM, 0.85)
//   * heads above 640 channels with so many candidates that the ring has two stages, while the streaming kernel's units fill most of
//     one round (141 x 256 x 256 x 768, K = 5 26.2, 32.6; 100 images 25.2, 22.1; 200 50.6, 42.6)
bool sim_topk_short_wanted(const Dims& dm) {
    if (dm.S > 256) return false;
    const long long sms = device_sms(), bh = (long long)dm.B * dm.H, units = bh * ((dm.T + BM - 1) / BM);
    if (units <= sms) return true;
    if (dm.nsel > 12) {
        const long long streaming = bh * ((dm.T + 2 * BM - 1) / (2 * BM));
        const long long here = (units + sms - 1) / sms, there = (streaming + sms - 1) / sms;
        const bool half = here >= 2 * there || (dm.T <= BM + 32 && 5 * here >= 8 * there);
        return !(dm.nsel > 16 && dm.S <= 40 && dm.T > BM && half && (there == 1 ? 2 : 1) * dm.nsel * 3 >= 2 * dm.S);
    }
    if (dm.T > BM && dm.S <= 32) return false;
    if (dm.T <= BM && dm.S <= 40) {
        if (dm.Cp > 512) return true;
        if (dm.nsel > 9) return false;
        return dm.Cp <= 128 || (units > 2 * sms && dm.Cp <= (dm.nsel > 4 ? 384 : dm.S > 32 ? 256 : 192));
    }
    if (dm.T <= BM && dm.S <= 80 && dm.nsel > 9 && dm.Cp <= 128 && 2 * units <= 3 * sms) return false;
    const long long streaming = bh * ((dm.T + 2 * BM - 1) / (2 * BM));
    return !(dm.Cp > 640 && dm.S > 224 && streaming <= sms && 5 * streaming > 4 * sms);
}

int launch_sim_topk_short(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                          const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
    ShortParams p{};
    p.qstat = qstat; p.kstat = kstat; p.cand = cand; p.idx = idx; p.val = val;
    p.T = dm.T; p.S = dm.S; p.H = dm.H; p.K = dm.K; p.nsel = dm.nsel; p.metric = d->metric; p.sampled = d->sampled;
    p.KCH = dm.Cp <= 16 ? 16 : (dm.Cp <= 32 ? 32 : 64);      // (the copies fill what lies past a head with zeros)
    p.KC = (dm.Cp + p.KCH - 1) / p.KCH;
    p.BN = (dm.S + 15) / 16 * 16;
    p.n_row_tiles = (dm.T + BM - 1) / BM;
    p.n_units = dm.B * dm.H * p.n_row_tiles;
    p.sqrt_dk = (float)sqrt((double)dm.dk);

    CUtensorMap tmK, tmQ;
    const uint64_t dimsK[4] = {(uint64_t)dm.Cp, (uint64_t)dm.H, (uint64_t)dm.T, (uint64_t)dm.B};
    const uint64_t dimsQ[4] = {(uint64_t)dm.Cp, (uint64_t)dm.H, (uint64_t)dm.S, (uint64_t)dm.B};
    const uint64_t strK[3] = {(uint64_t)dm.Cp * 2, (uint64_t)dm.H * dm.Cp * 2, (uint64_t)dm.T * dm.H * dm.Cp * 2};
    const uint64_t strQ[3] = {(uint64_t)dm.Cp * 2, (uint64_t)dm.H * dm.Cp * 2, (uint64_t)dm.S * dm.H * dm.Cp * 2};
    const uint32_t boxK[4] = {(uint32_t)p.KCH, 1, (uint32_t)BM, 1};
    const uint32_t boxQ[4] = {(uint32_t)p.KCH, 1, (uint32_t)p.BN, 1};
    if (!encode_tensor_map_bf16(&tmK, k, 4, dimsK, strK, boxK, p.KCH * 2)) return CONVNN_E_CUDA;
    if (!encode_tensor_map_bf16(&tmQ, q, 4, dimsQ, strQ, boxQ, p.KCH * 2)) return CONVNN_E_CUDA;

    const int n = dm.nsel;
    // One thread per row and four accumulators for up to 128 candidates, if many units follow one another and the heads are
    // narrow: its entries leave the ring two stages (us, this form, the other: 256 x 197 x 64, K = 9, three heads of 64 29.3, 33.6;
    // 1024 x 65 x 65, three heads of 64 42, 58; 256 x 197 x 64 x 384 19.3, 17.2; 1024 x 64 x 64 x 384 37, 25).
    const bool narrow = dm.S <= 128 && dm.Cp <= 256 && p.n_units > device_sms();
#define CONVNN_SHORT(N)                                                     \
    do {                                                                    \
        if (narrow) return launch_short<N, 4, 1>(dm, p, tmK, tmQ, st);    \
        return launch_short<N, 2, 2>(dm, p, tmK, tmQ, st);                     \
    } while (0)
    if (n <= 4) CONVNN_SHORT(4);
    if (n <= 8) CONVNN_SHORT(8);
    if (n == 9) CONVNN_SHORT(9);
    if (n <= 12) return launch_short<12, 2, 2>(dm, p, tmK, tmQ, st);
    if (n <= 16 && dm.S <= 128) return launch_short<16, 4, 1>(dm, p, tmK, tmQ, st);
    if (n <= 16) return launch_short<16, 2, 1>(dm, p, tmK, tmQ, st);
    if (n <= 25) return launch_short<25, 2, 1>(dm, p, tmK, tmQ, st);
    return launch_short<32, 2, 1>(dm, p, tmK, tmQ, st);
#undef CONVNN_SHORT
}

int read_sim_short_status(int* out) {
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_sim_short_status, sizeof(int));
    if (e != cudaSuccess) return set_error(CONVNN_E_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    *out = v;
    return CONVNN_OK;
}

}  // namespace convnn
