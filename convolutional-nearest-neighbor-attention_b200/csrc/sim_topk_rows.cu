// Similarity + top-K for candidate lists that fit one accumulator (S <= 256), a WARP per key row.
//
// A thread per row (the TMEM layout) leaves at most 256 rows in flight per SM and chains of dependent comparisons.  Here the
// accumulator is copied once to shared memory as ranking keys, row by row, and sixteen warps take rows from there: lane l
// holds columns l, l + 32, ..., two rows are interleaved, nothing diverges and no lane idles on a ragged sequence end (topk_rows.cuh).
//
// A persistent CTA per SM owns an equal share of the flattened (batch, head, row) range, in segments of up to 128 rows of
// one (batch, head), wherever they start.  Warp 0: TMA producer (128 key rows from the segment's first, all
// candidate rows, 64-channel chunks, ring); warp 1: MMA issuer (M = 128, N = S rounded to 16), two accumulators; warps 2-17:
// copy and selection.
#include "common.cuh"
#include "f32x2.cuh"
#include "sim_topk_select.cuh"
#include "sm100.cuh"
#include "topk_rows.cuh"

namespace convnn {

__device__ int g_sim_rows_status = 0;

namespace {

using namespace sm100;
using namespace topk_rows;

constexpr int BM = 128;
constexpr int MAX_STAGES = 6;
constexpr int NW = 16;                  // selection warps
constexpr int WR = BM / NW;             // most rows of a segment per warp
constexpr int NT = 64 + 32 * NW;

struct RowsParams {
    const float *qstat, *kstat;
    const int32_t* cand;
    int32_t* idx;
    float* val;
    int T, S, H, K, nsel, metric, sampled;
    // GATHER: the depthwise conv over the neighbours instead of their lists (reference layers.py:345-406)
    const uint4* v;     // (B, T, H, 8 groups)
    const uint4* w;     // taps (K, 8 groups)
    uint4* o;           // (B, H, T, 8 groups)
    int groups, softmax;
    int KCH, KC;        // channels per shared-memory chunk, chunks per segment
    int BN, pitch;      // S rounded up to 16; words between the rows of the key buffer (4 mod 8: 16-byte stores of eight
                        // consecutive rows fall into different banks)
    int acc_cols;       // TMEM columns of one accumulator
    int seg_rows;       // most rows of a segment (rows of the key buffer)
    int inv_K;
    int stages;
    int rows_total, rows_per_cta, per_head;
    float sqrt_dk;
    int box_rows;                  // key rows fetched per segment
};

__device__ __forceinline__ void fail(volatile int* abort_flag, int code) {
    *abort_flag = 1;
    atomicCAS(&g_sim_rows_status, 0, code);
}

// A CTA's range of flattened rows, cut into segments of one (batch, head).  Ranges follow each other; with `per_head` set they
// start anew in every (batch, head), `per_head` of them.
struct Segment {
    int g, end;          // first flattened row, end of the CTA's range
    int bh, row, n;
    __device__ __forceinline__ Segment(const RowsParams& p) {
        if (p.per_head) {
            bh = blockIdx.x / p.per_head;
            row = (blockIdx.x - bh * p.per_head) * p.rows_per_cta;
            g = bh * p.T + row;
            end = g + min(p.rows_per_cta, p.T - row);
        } else {
            g = blockIdx.x * p.rows_per_cta;
            end = min(g + p.rows_per_cta, p.rows_total);
            bh = g / p.T;
            row = g - bh * p.T;
        }
        n = min(min(p.T - row, end - g), p.seg_rows);
    }
    __device__ __forceinline__ bool valid() const { return g < end; }
    __device__ __forceinline__ void next(const RowsParams& p) {
        g += n;
        row += n;
        if (row == p.T) { row = 0; ++bh; }
        n = min(min(p.T - row, end - g), p.seg_rows);
    }
};

__device__ __forceinline__ void selection_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory"); }

// Depthwise conv of the warp's rows, whose (value, token) lists lie in `list` (pairs: .x value, .y token): weights over the
// values as in token_weights.cuh (sums in tap order), then a 16-byte channel group of a row per lane.
constexpr int TAPS = 5;                 // neighbour rows in flight per lane (nine spill: 504 -> 496 us per ViT-Tiny image)
__device__ __forceinline__ void conv_rows(const RowsParams& p, float2* list, const uint4* taps, int w, int n, int g, int bh) {
    const int lane = threadIdx.x & 31, b = bh / p.H, h = bh - b * p.H;
    const bool maximum = p.metric != CONVNN_EUCLIDEAN;
    const int vbase = (b * p.T * p.H + h) * p.groups, vstride = p.H * p.groups;      // (B T D < 2^31)
    // the lane's first neighbour rows are on their way while the weights are made
    uint4 raw[TAPS];
    if (lane < n * p.groups) {
        const int m = lane / p.groups, cg = lane - m * p.groups;
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
            if (j < p.K) raw[j] = __ldg(p.v + vbase + __float_as_int(list[m * p.K + j].y) * vstride + cg);
    }
    __syncwarp();                                   // (the entries are rewritten below)
    for (int m0 = 0; m0 < n; m0 += 2) {             // two rows, sixteen lanes each (K <= 17: a lane more holds the last)
        const int j = lane & 15, m = m0 + (lane >> 4);
        const bool in = m < n && j < p.K, last = p.K > 16 && m < n && j == 15;
        float2* e0 = list + m * p.K;
        float x = in ? e0[j].x : 0.f, x16 = last ? e0[16].x : 0.f;
        float wt, wt16 = 0.f;
        if (p.softmax) {
            if (!maximum) { x = -x; x16 = -x16; }
            float mx = in ? fmaxf(x, -3.402823466e38f) : -3.402823466e38f;
            if (last) mx = fmaxf(mx, x16);
#pragma unroll
            for (int d = 8; d >= 1; d /= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
            const float ex = in ? expf(x - mx) : 0.f, ex16 = last ? expf(x16 - mx) : 0.f;
            float s = 0.f;
            for (int i = 0; i < min(p.K, 16); ++i) s += __shfl_sync(0xffffffffu, ex, i, 16);
            if (p.K > 16) s += __shfl_sync(0xffffffffu, ex16, 15, 16);
            wt = ex / s;
            wt16 = ex16 / s;
        } else {
            wt = maximum ? x : 1.0f / (x + 1e-8f);
            wt16 = maximum ? x16 : 1.0f / (x16 + 1e-8f);
        }
        if (in) e0[j] = make_float2(wt, __int_as_float(vbase + __float_as_int(e0[j].y) * vstride));
        if (last) e0[16] = make_float2(wt16, __int_as_float(vbase + __float_as_int(e0[16].y) * vstride));
    }
    __syncwarp();
    for (int e = lane; e < n * p.groups; e += 32) {
        const int m = e / p.groups, cg = e - m * p.groups;
        const float2* l = list + m * p.K;
        f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
        for (int j0 = 0; j0 < p.K; j0 += TAPS) {
            if (e != lane || j0 != 0) {
#pragma unroll
                for (int j = 0; j < TAPS; ++j)
                    if (j0 + j < p.K) raw[j] = __ldg(p.v + __float_as_int(l[j0 + j].y) + cg);
            }
#pragma unroll
            for (int j = 0; j < TAPS; ++j)
                if (j0 + j < p.K) {
                    f32x2 x[4], tw[4];
                    bf16x8_to_f32x2(raw[j], x);
                    bf16x8_to_f32x2(taps[(j0 + j) * p.groups + cg], tw);
                    const float pj = l[j0 + j].x;
                    const f32x2 p2 = pack2(pj, pj);
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[q] = fma2(tw[q], mul2(p2, x[q]), acc[q]);
                }
        }
        p.o[(long long)(g + w + m * NW) * p.groups + cg] = f32x2_to_bf16x8(acc);
    }
    __syncwarp();
}

template <int J, int NS, bool GATHER>          // NS as in select_lists()
__global__ void __launch_bounds__(NT, 1)
sim_topk_rows_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ,
                     const __grid_constant__ RowsParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t pitch = p.KCH * 2;
    const uint32_t a_bytes = BM * pitch, b_bytes = p.BN * pitch, stage_bytes = a_bytes + b_bytes;
    const uint32_t landing = p.box_rows * pitch + b_bytes;    // (rows past the CTA's range stay whatever they were: no sum uses them)
    const uint32_t STAGES = p.stages;
    float* keybuf = reinterpret_cast<float*>(smem + STAGES * stage_bytes);      // [seg_rows][pitch]
    float2* lists = reinterpret_cast<float2*>(keybuf + p.seg_rows * p.pitch);   // [NW][WR][K] key, column
    float2* found = lists + NW * WR * p.K;                                      // [NW][found_pairs] survivors: key, column
    float* qs = reinterpret_cast<float*>(found + NW * found_pairs(NS));         // [BN] column statistics
    int* cs = reinterpret_cast<int*>(qs + p.BN);                                // [BN] candidate tokens
    float* kst_s = reinterpret_cast<float*>(cs + p.BN);                         // [BM] row statistics
    uint64_t* full = reinterpret_cast<uint64_t*>(kst_s + BM);
    uint64_t* empty = full + MAX_STAGES;
    uint64_t* tfull = empty + MAX_STAGES;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint4* taps = reinterpret_cast<uint4*>(tempty + 4);                         // GATHER: [K][groups]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], NW);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmK);
        prefetch_tensormap(&tmQ);
    }
    const uint32_t ncols = 2u * p.acc_cols;
    if (warp == 1) {
        tmem_alloc(tmem_slot, ncols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // (every role waits for the predecessor before its own first access to global memory)

    const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), st0 = smem_u32(smem);
    if (warp == 0) {
        Segment sg(p);
        chain_wait();
        {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (; sg.valid() && ok; sg.next(p)) {
                const int b = sg.bh / p.H, h = sg.bh - b * p.H;
                for (int kc = 0; kc < p.KC; ++kc) {
                    ok = mbar_wait_warp(empty0 + 8 * s, ph ^ 1u, abort_flag);
                    if (!ok) { if (lane == 0) fail(abort_flag, 81); break; }
                    const uint32_t st = st0 + s * stage_bytes, fb = full0 + 8 * s;
                    if (elect_one()) {
                        mbar_expect_tx_a(fb, landing);
                        tma_load_4d_a(st, &tmK, fb, kc * p.KCH, h, sg.row, b);
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
            chain_wait();                            // (the budgets of its waits are for this kernel's work)
            for (Segment sg(p); sg.valid() && ok; sg.next(p)) {
                if (!mbar_wait_warp(tempty0 + 8 * buf, (use & 1u) ^ 1u, abort_flag)) { fail(abort_flag, 82); break; }
                tc_fence_after_sync();
                for (int kc = 0; kc < p.KC; ++kc) {
                    if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag)) { fail(abort_flag, 83); ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t sa = st0 + s * stage_bytes;
                    if (elect_one()) {
                        mma_chunk(tmem_base + buf * p.acc_cols, dhi | (uint64_t)(sa >> 4),
                                  dhi | (uint64_t)((sa + a_bytes) >> 4), idesc, nk16, kc != 0);
                        mma_commit_a(empty0 + 8 * s);
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
                if (ok && elect_one()) mma_commit_a(tfull0 + 8 * buf);
                if (++buf == 2) { buf = 0; ++use; }
            }
        }
    } else {
        const int w = warp - 2;
        const int tid = threadIdx.x - 64;
        const int lq = warp & 3;                     // TMEM lane quarter it may read
        const int sub = w >> 2;                      // its share of that quarter's columns
        const int r = lq * 32 + lane;
        float2* list = lists + w * WR * p.K;
        const uint32_t found0 = smem_u32(found + w * found_pairs(NS));
        const RowsTask task{kst_s, cs, p.idx, p.val, p.pitch, p.BN, p.nsel, p.K, p.inv_K, p.metric, p.sampled, p.sqrt_dk};
        const bool stats = p.metric != CONVNN_MATMUL;
        uint32_t buf = 0, use = 0;
        const float none = __int_as_float(0x7fffffff);           // columns past the last candidate: their keys become NaN
        // Every selection warp makes the same number of passes and meets every barrier, also after a wait has expired
        // anywhere in the CTA (it then skips the work): none is left waiting for another.
        Segment sg(p);
        float q_next = none, kst_next = 1.f;
        auto fetch = [&] {
            if (tid < p.S) q_next = stats ? p.qstat[(long long)sg.bh * p.S + tid] : 1.f;
            if (stats && r < sg.n) kst_next = p.kstat[sg.g + r];
        };
        chain_wait();
        chain_next();
        if (sg.valid()) fetch();
        if (p.sampled)                               // (this and the taps are read behind the barriers of the first segment)
            for (int c = tid; c < p.BN; c += 32 * NW) cs[c] = c < p.S ? p.cand[c] : -1;
        if (GATHER)
            for (int c = tid; c < p.K * p.groups; c += 32 * NW) taps[c] = p.w[c];
        while (sg.valid()) {
            const float kst = kst_next;
            if (tid < p.BN) qs[tid] = q_next;
            const Segment cur = sg;
            sg.next(p);
            if (sg.valid()) fetch();
            bool ok = mbar_wait(&tfull[buf], use & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok && lane == 0) fail(abort_flag, 84);
            selection_barrier();                     // the key buffer is free, the column statistics are there
            if (ok && lq * 32 < cur.n) {
                tc_fence_after_sync();
                if (sub == 0) kst_s[r] = kst;
                const int row = cur.row + r;
                const float sentinel = p.sampled ? self_sentinel(p.metric, kst, p.sqrt_dk) : 0.f;
                float* out = keybuf + (r < p.seg_rows ? r : 0) * p.pitch;
                const bool mine = r < cur.n;
                const uint32_t taddr = tmem_base + ((uint32_t)(lq * 32) << 16) + buf * p.acc_cols;
                auto store_keys = [&](const uint32_t (&acc)[16], int c) {
#pragma unroll
                    for (int j4 = 0; j4 < 4; ++j4) {
                        const float4 s4 = *reinterpret_cast<const float4*>(qs + c + 4 * j4);
                        const f32x2 d01 = pack2(__uint_as_float(acc[4 * j4]), __uint_as_float(acc[4 * j4 + 1]));
                        const f32x2 d23 = pack2(__uint_as_float(acc[4 * j4 + 2]), __uint_as_float(acc[4 * j4 + 3]));
                        f32x2 k01, k23;
                        if (p.metric != CONVNN_EUCLIDEAN) {      // (matmul: statistics of 1)
                            k01 = mul2(d01, pack2(s4.x, s4.y));
                            k23 = mul2(d23, pack2(s4.z, s4.w));
                        } else {
                            const f32x2 two = pack2(2.0f, 2.0f);
                            k01 = fma2(two, d01, pack2(-s4.x, -s4.y));
                            k23 = fma2(two, d23, pack2(-s4.z, -s4.w));
                        }
                        float4 k;
                        unpack2(k01, k.x, k.y);
                        unpack2(k23, k.z, k.w);
                        if (p.sampled) {
                            const int4 c4 = *reinterpret_cast<const int4*>(cs + c + 4 * j4);
                            if (c4.x == row) k.x = sentinel;
                            if (c4.y == row) k.y = sentinel;
                            if (c4.z == row) k.z = sentinel;
                            if (c4.w == row) k.w = sentinel;
                        }
                        if (mine) *reinterpret_cast<float4*>(out + c + 4 * j4) = k;
                    }
                };
                for (int c = sub * 16; c < p.BN; c += 128) {     // two blocks in flight
                    uint32_t a0[16], a1[16];
                    const bool two = c + 64 < p.BN;
                    tmem_ld_x16(taddr + c, a0);
                    if (two) tmem_ld_x16(taddr + c + 64, a1);
                    tmem_ld_wait();
                    store_keys(a0, c);
                    if (two) store_keys(a1, c + 64);
                }
                tc_fence_before_sync();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[buf]);
            selection_barrier();                     // the keys are there
            if (!*abort_flag) {
                if constexpr (GATHER) {
                    const int n = select_lists<J, NS, NW>(task, keybuf, list, found0, w, cur.n, cur.row,
                        [&](int m, int slot, int tok, float s) { list[m * p.K + slot] = make_float2(s, __int_as_float(tok)); });
                    conv_rows(p, list, taps, w, n, cur.g, cur.bh);
                } else {
                    select_and_write<J, NS, NW>(task, keybuf, list, found0, w, cur.n, cur.g, cur.row);
                }
            }
            if (++buf == 2) { buf = 0; ++use; }
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
        tmem_dealloc(tmem_base, ncols);
    }
}

template <int J, int NS, bool GATHER>
int launch_rows(RowsParams& p, size_t smem, int grid, const CUtensorMap& tmK, const CUtensorMap& tmQ, cudaStream_t st) {
    auto kern = sim_topk_rows_kernel<J, NS, GATHER>;
    CONVNN_ENSURE_SMEM(kern, smem);
    launch_chained(kern, grid, NT, smem, st, tmK, tmQ, p);
    CONVNN_CHECK_LAUNCH("sim_topk_rows");
    return CONVNN_OK;
}

template <int J>
int launch_rows_j(RowsParams& p, size_t smem, int grid, const CUtensorMap& tmK, const CUtensorMap& tmQ, cudaStream_t st) {
    if (p.o) {
        if (p.nsel == 9) return launch_rows<J, 9, true>(p, smem, grid, tmK, tmQ, st);
        if (p.nsel <= 12) return launch_rows<J, 0, true>(p, smem, grid, tmK, tmQ, st);
        return launch_rows<J, -3, true>(p, smem, grid, tmK, tmQ, st);
    }
    if (p.nsel == 8) return launch_rows<J, 8, false>(p, smem, grid, tmK, tmQ, st);
    if (p.nsel == 9) return launch_rows<J, 9, false>(p, smem, grid, tmK, tmQ, st);
    if (p.nsel <= 12) return launch_rows<J, 0, false>(p, smem, grid, tmK, tmQ, st);
    if (p.nsel <= 16) return launch_rows<J, -3, false>(p, smem, grid, tmK, tmQ, st);
    if (p.nsel <= 25) return launch_rows<J, -1, false>(p, smem, grid, tmK, tmQ, st);
    return launch_rows<J, -2, false>(p, smem, grid, tmK, tmQ, st);
}

}  // namespace

static int rows_per_sm(const Dims& dm) {
    const int sms = device_sms();
    return (int)(((long long)dm.B * dm.H * dm.T + sms - 1) / sms + NW - 1) / NW * NW;
}

// Rows per CTA; ranges that do not cross from one (batch, head) to the next, where they need be no longer: a segment less each.
struct Ranges {
    int rows, per_head, grid;
};
static Ranges ranges_of(const Dims& dm) {
    const long long total = (long long)dm.B * dm.H * dm.T;
    Ranges r{rows_per_sm(dm), 0, 0};
    const int parts = device_sms() / (dm.B * dm.H);
    if (parts > 0) {
        const int rows = ((dm.T + parts - 1) / parts + NW - 1) / NW * NW;
        if (rows <= r.rows + NW) {
            r.rows = rows;
            r.per_head = (dm.T + rows - 1) / rows;
        }
    }
    r.grid = r.per_head ? dm.B * dm.H * r.per_head : (int)((total + r.rows - 1) / r.rows);
    return r;
}

// What bounds it: warp instructions, ~310 per row of 197 keys with the copy, at 0.44 per cycle and scheduler (148 images; copying
// the accumulator and selecting do not overlap).  A row costs about the same wherever it runs, while the two-pass kernel works in whole 128-row units and the streaming kernel
// needs many rows per SM to hide its chains.  us, others -> this kernel, 192 channels unless noted:
//   197 x 197, K = 9         1 image 14.9 -> 6.5    37: 15.2 -> 8.8    148: 21.9 -> 17.1    220: 30.4 -> 26.2    256: 30.4 -> 30.2 (not taken)
//   12 heads of 64           1 image 14.8 -> 6.6    16: 27.5 -> 22.3    32: 40.4 -> 37.8 (not taken)
//   197 x 64 x 384, K = 9    1 image 9.2 -> 6.5     16: 9.5 -> 7.1      74: 9.8 -> 12.2 (not taken)
//   (two batches in flight lose 0.6 % with it at 256 images: a CTA of this kernel fills its SM)
//   1000 x 256 x 768, K = 5  1 image 18.0 -> 9.9    4: 18.2 -> 11.1     16: 18.9 -> 21.5 (not taken)
// These figures are against the two-pass kernel's sorted lists of values.  Since that bounds its rows by group maxima, and this kernel
// bounds lists of more than twelve by two maxima per lane (two-pass, this kernel, us):
//   197 x 197, one head of 96, K = 9   20 images 9.3, 7.1   38: 9.4, 9.2   64: 9.7, 10.6   150: 17.6, 21.0;  3 heads of 32   64: 17.4, 22.1
//   K = 5   20: 8.4, 7.0   38: 8.6, 8.8   64: 8.8, 10.2        K = 16   20: 12.7, 8.1   38: 13.3, 12.0   64 x 3 heads of 64: 23.5, 36.6
//   197 x 197 x 192, K = 25   1 image 16.8, 8.2   20: 16.8, 10.0   34: 17.8, 13.9      65 x 65 x 192   80: 13.0, 13.5   100: 14.2, 13.5
// Row tiles of 128 pad longer sequences, and candidates that are not the rows themselves cost the two-pass kernel more: lists of up to twelve
// keep this kernel longer beyond 256 tokens (two-pass, this kernel, us).
//   K = 9    13 x 969 x 254 x 64 13.3, 9.9   35 x 330 x 206 x 32 12.0, 9.4   18 x 893 x 253 x 32 13.0, 10.6   14 x 677 x 210, two heads of 64 12.0, 13.5
//            12 x 843 x 188 x 256 11.5, 9.6   20 x 680 x 207 x 256 12.5, 14.7
// (Rows whose survivors overflow cost this kernel 5 us and a launch has them or not.  For lists of 13 to 16 that decides between 64 and 112
// rows per SM, 150 shapes 0.7 to 1.5 times the two-pass kernel's time and as often the one as the other: left at 64.)
// Long lists among up to 64 candidates, where most of them are listed (K = 17 to 32; two-pass, this kernel): up to one unit of the two-pass
// kernel per SM   27 x 281 x 30 x 64 13.5, 9.6   12 x 822 x 32 x 128 16.5, 12.5   37 x 272 x 49 x 64 14.7, 12.3   39 x 341 x 58 x 768 16.5, 19.4 (90 rows per SM, not
// taken);  short sequences, whose units are mostly padding   174 x 50, six heads of 768 122, 76   1144 x 22, three heads of 64 131, 83   28 x 131,
// three heads of 128 21.9, 14.6;  but 195 x 57 x 23, six heads of 192 47, 57   175 x 58, six heads of 768 63, 68   186 x 45 x 192 12.6, 13.5.
// The line of lists of five to twelve with one head of 129 to 192 channels has not been drawn again (132 images 12.3, 18.8).
// Where others win, and the lines of the rule (R rows per SM, rounds u of 256-row units per SM, w the share of their warps that
// has rows: two units of the streaming kernel share an SM and slow each other down by about w / 2):
//   * up to 128 candidates, and heads above 384 channels, only ranges that stay inside a head: a range across heads is cut into
//     segments with a product each (278 x 17 x 17 x 384, K = 9 9.2 -> 11.2; 109 x 65 x 40 x 768 10.9 -> 13.7)
//   * lists of up to four are cheap elsewhere (256 x 130 x 130 x 16, K = 3 12.9 -> 17.3; 192 x 197 x 197 x 192, K = 3 1.08 times)
//   * up to 175 candidates the streaming kernel's 64-column tiles fit better (236 x 130 x 130 x 16, K = 5 1.08 times)
//   * many wide candidates are fetched again for every segment (30 x 1000 x 250 x 384, K = 9 1.13 times; 120 x 256 x 256 x 384 0.91)
bool sim_topk_rows_wanted(const Dims& dm) {
    if (dm.S > 256) return false;
    const int R = rows_per_sm(dm);
    if (dm.nsel > 16) {
        const long long two_pass_units = (long long)dm.B * dm.H * ((dm.T + 127) / 128);
        if ((dm.T <= 40 && dm.S <= 32) || (dm.T <= 56 && dm.Cp >= 512)) return R <= 512;
        return R <= (dm.S <= 64 && two_pass_units <= device_sms() ? 80 : 48);
    }
    if (dm.S <= 128 || dm.Cp > 384) return R <= 48 && ranges_of(dm).per_head;
    const bool other_width = dm.Cp <= 128 || dm.Cp > 192;
    if (dm.nsel > 12) return R <= (other_width || dm.S < 176 ? 64 : 96);
    if (dm.Cp > 192 && dm.S > 208 && dm.T > 256) return R <= 96;
    if (dm.nsel >= 4 && dm.S >= 176 && other_width && (dm.Cp <= 128 || dm.S <= 208)) return R <= (dm.T > 256 && dm.Cp <= 128 ? 112 : dm.S > 208 || (dm.T > 256 && dm.nsel > 4) ? 80 : 64);
    if (dm.nsel > 4 && dm.S >= 176) return R <= 304;
    const int units_of = (dm.T + 255) / 256;
    const double u = (double)dm.B * dm.H * units_of / device_sms(), w = (double)((dm.T + 31) / 32) / (8 * units_of);
    if (dm.nsel <= 4) return R <= (dm.S < 144 ? 110 : dm.S < 176 ? 150 : 165) * (u <= 1 ? 1 : u <= 2 ? 1 + 0.4 * w : 2);
    return R <= (dm.S < 144 ? 128 : 190) * (u <= 1 ? 1 : u <= 2 ? 1 + 0.5 * w : 2);
}

static int launch_impl(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                       const float* kstat, const int32_t* cand, int32_t* idx, float* val, const void* v, const void* w_conv,
                       void* o, cudaStream_t st) {
    RowsParams p{};
    p.qstat = qstat; p.kstat = kstat; p.cand = cand; p.idx = idx; p.val = val;
    p.T = dm.T; p.S = dm.S; p.H = dm.H; p.K = dm.K; p.nsel = dm.nsel; p.metric = d->metric; p.sampled = d->sampled ? 1 : 0;
    p.BN = (dm.S + 15) / 16 * 16;
    p.pitch = p.BN + 4;
    p.acc_cols = 32;
    while (p.acc_cols < p.BN) p.acc_cols *= 2;
    p.sqrt_dk = (float)sqrt((double)dm.dk);
    p.rows_total = dm.B * dm.H * dm.T;
    const Ranges ranges = ranges_of(dm);
    p.rows_per_cta = ranges.rows; p.per_head = ranges.per_head;
    const int grid = ranges.grid;
    p.seg_rows = p.rows_per_cta < BM ? p.rows_per_cta : BM;
    p.inv_K = inverse_of(dm.K);
    p.v = static_cast<const uint4*>(v); p.w = static_cast<const uint4*>(w_conv); p.o = static_cast<uint4*>(o);
    p.groups = dm.dk / 8; p.softmax = d->softmax;
    const size_t fixed = 1024 + (size_t)p.seg_rows * p.pitch * 4 + (size_t)NW * WR * dm.K * 8 +
                         (o ? (size_t)dm.K * dm.dk * 2 : 0) +
                         (size_t)NW * found_pairs(dm.nsel > 16 ? -1 : 0) * 8 + (size_t)p.BN * 8 + BM * 4 +
                         (2 * MAX_STAGES + 6) * 8;
    const size_t room = 226 * 1024 - fixed;
    // (the copies fill what lies past a head with zeros; 32-channel chunks where only one of 64 would fit)
    p.KCH = dm.Cp <= 16 ? 16 : (dm.Cp <= 32 ? 32 : 64);
    if (p.KCH == 64 && room / ((size_t)(BM + p.BN) * 128) < 2) p.KCH = 32;
    p.KC = (dm.Cp + p.KCH - 1) / p.KCH;
    const size_t stage = (size_t)(BM + p.BN) * p.KCH * 2;
    p.stages = (int)(room / stage);
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    if (p.stages > 2 * p.KC) p.stages = 2 * p.KC;            // deeper than two segments' chunks serves nothing
    size_t smem = fixed + p.stages * stage;
    if (smem < 116 * 1024) smem = 116 * 1024;                // a CTA may take all of an SM's TMEM: never two on one SM

    CUtensorMap tmK, tmQ;
    const uint64_t dimsK[4] = {(uint64_t)dm.Cp, (uint64_t)dm.H, (uint64_t)dm.T, (uint64_t)dm.B};
    const uint64_t dimsQ[4] = {(uint64_t)dm.Cp, (uint64_t)dm.H, (uint64_t)dm.S, (uint64_t)dm.B};
    const uint64_t strK[3] = {(uint64_t)dm.Cp * 2, (uint64_t)dm.H * dm.Cp * 2, (uint64_t)dm.T * dm.H * dm.Cp * 2};
    const uint64_t strQ[3] = {(uint64_t)dm.Cp * 2, (uint64_t)dm.H * dm.Cp * 2, (uint64_t)dm.S * dm.H * dm.Cp * 2};
    // (a box of the CTA's rows alone: with 16 of them 86 KB land where 128 did)
    p.box_rows = (p.seg_rows + 7) / 8 * 8;
    const uint32_t boxK[4] = {(uint32_t)p.KCH, 1, (uint32_t)p.box_rows, 1};
    const uint32_t boxQ[4] = {(uint32_t)p.KCH, 1, (uint32_t)p.BN, 1};
    if (!encode_tensor_map_bf16(&tmK, k, 4, dimsK, strK, boxK, p.KCH * 2)) return CONVNN_E_CUDA;
    if (!encode_tensor_map_bf16(&tmQ, q, 4, dimsQ, strQ, boxQ, p.KCH * 2)) return CONVNN_E_CUDA;

    switch ((p.BN + 31) / 32) {
        case 1: return launch_rows_j<1>(p, smem, grid, tmK, tmQ, st);
        case 2: return launch_rows_j<2>(p, smem, grid, tmK, tmQ, st);
        case 3: return launch_rows_j<3>(p, smem, grid, tmK, tmQ, st);
        case 4: return launch_rows_j<4>(p, smem, grid, tmK, tmQ, st);
        case 5: return launch_rows_j<5>(p, smem, grid, tmK, tmQ, st);
        case 6: return launch_rows_j<6>(p, smem, grid, tmK, tmQ, st);
        case 7: return launch_rows_j<7>(p, smem, grid, tmK, tmQ, st);
        default: return launch_rows_j<8>(p, smem, grid, tmK, tmQ, st);
    }
}

int launch_sim_topk_rows(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                         const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
    return launch_impl(d, dm, q, k, qstat, kstat, cand, idx, val, nullptr, nullptr, nullptr, st);
}

// Where a CTA has at most 32 rows, two per warp: the conv's neighbour rows come from L2 a few at a time, which costs less than
// another kernel then, and more from four rows per warp on.  ViT-Tiny forward, us, lists and conv in two kernels -> in one:
// 1 image 527 -> 496, 16 images 605 -> 572 (32 rows per CTA), 37: 656 -> 655 (64), 64: 739 -> 817 (96).  Not for ranges across
// heads, whose segments are served one after the other (whole layers: 278 x 17 tokens x 64, K = 9 19.3 -> 24.9), nor for more
// than 12 KB of taps over short lists, where the conv is the longer part (23 x 100 x 768, K = 9 46.2 -> 48.7, but 3 x 197 44.9 -> 37.7).
int try_launch_sim_gather(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const void* v, const float* qstat,
                          const float* kstat, const int32_t* cand, const void* w_conv, void* o, cudaStream_t st) {
    if (!sim_topk_tc_supported(d, dm, q, k) || dm.S > 256 || dm.nsel > 16 || ranges_of(dm).rows > 32 || !ranges_of(dm).per_head ||
        dm.C != dm.dk || dm.dk % 8 != 0 || dm.K * dm.dk > (dm.S <= 128 ? 6144 : 8192) || !aligned16(v) || !aligned16(w_conv) || !aligned16(o))
        return CONVNN_E_UNSUPPORTED;
    return launch_impl(d, dm, q, k, qstat, kstat, cand, nullptr, nullptr, v, w_conv, o, st);
}

int read_sim_rows_status(int* out) {
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_sim_rows_status, sizeof(int));
    if (e != cudaSuccess) return set_error(CONVNN_E_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    *out = v;
    return CONVNN_OK;
}

}  // namespace convnn
