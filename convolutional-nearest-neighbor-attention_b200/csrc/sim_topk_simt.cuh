// Similarity + streaming top-K on the FP32 SIMT pipes.
//
// A CTA of 256 threads owns RB (128 or 64) consecutive key tokens (rows of the similarity matrix) of one
// (batch, head) and visits the candidate columns in tiles of 64.  A tile's dot products are a register-blocked
// matrix product (RB / 16 x 4 per thread, channels strictly ascending, two columns per packed multiply-add,
// operands transposed through double-buffered shared memory, the loads of the next channel step in flight); they
// become ranking keys in a shared-memory tile, which 256 / RB threads per row then scan, each with a sorted register
// list of its own; the lists of a row are merged at the end under the full (key, column) order.  The T x S matrix
// never exists in memory, and exact ties go to the lower candidate column.
//
// Bound by the shared-memory reads that feed the fp32 pipes (64 images of 197 x 192: L1 68 % busy, warps wait for shared
// memory most), and by the insertions of long lists.  One thread per row with its 64 columns in registers, before, read every operand value of a column from
// shared memory once per row: 97 us per layer at 32 x 65 tokens x 192 channels.
//
// Ranking keys (larger is better) and the values reported for the survivors:
//   cosine     key = dot * qinv[j]            val = key * kinv[i]
//   matmul     key = dot                      val = key / sqrt(d_k)
//   euclidean  key = 2*dot - |q_j|^2          val = sqrt(max(|k_i|^2 - key, 0))
// The sampled modes replace the entry (cand[j] == i) by the reference's finite sentinel
// (-0.1, or 1.1 for euclidean; layers.py:234-235, 291-292) expressed in key space.
//
// This is the float32 path of the library (accuracy ~1e-7 so that index sets match the
// reference down to 1e-6 gaps) and the fallback for bfloat16 shapes outside the tcgen05
// kernel's envelope.
#pragma once
#include <math_constants.h>

#include "common.cuh"
#include "f32x2.cuh"
#include "toplist.cuh"
#include "cluster_lists.cuh"

namespace convnn {
namespace simt_topk {

constexpr int NT = 256;
constexpr int CB = 64;      // candidate columns per tile
constexpr int BK = 16;      // channels per step
constexpr int LK = CB + 4;  // row stride of the key tile: 16-byte rows that fall into different banks

__host__ __device__ constexpr int tile_floats(int rb) { return 2 * BK * (rb + 4) + 2 * BK * (CB + 4) + rb * LK + NT; }
__host__ __device__ constexpr int merge_floats(int rb, int kcap) { return 2 * kcap * rb * (NT / rb - 1); }
__host__ __device__ constexpr int cluster_floats(int rb, int kcap) { return 4 * kcap * rb; }
__host__ __device__ constexpr int smem_bytes(int rb, int kcap, bool split) {
    const int a = tile_floats(rb), b = merge_floats(rb, kcap), c = split ? cluster_floats(rb, kcap) : 0;
    return 4 * (a > b ? (a > c ? a : c) : (b > c ? b : c));
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ float4 load_upto4(const T* p, int n, bool vec) {
    if (vec && n >= 4) return load4(p);
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (i < n) r[i] = to_f32<T>(p[i]);
    return make_float4(r[0], r[1], r[2], r[3]);
}

// (Two CTAs of 64 rows fit an SM: the other lists keep to 128 registers by themselves, 26 to 32 neighbours took 160 and ran one at a time:
// us, so -> bounded, bfloat16 20 x 439 x 439 x 97 242 -> 143, 17 x 570 x 570 x 8 201 -> 123, float32 21 x 624 x 624 x 8 209 -> 132.  0: not stated.)
template <typename T, int KCAP, int RB>
__global__ void __launch_bounds__(NT, RB == 64 && KCAP > 25 ? 2 : 0) sim_topk_simt_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const float* __restrict__ qstat,
    const float* __restrict__ kstat, const int32_t* __restrict__ cand, int32_t* __restrict__ idx,
    float* __restrict__ val, int T_, int S, int H, int Cp, int K, int nsel, int metric, int sampled,
    float sqrt_dk, int vec, int split) {
    chain_wait();               // (and no early start for the next one, see chain_begin_for())
    constexpr int TM = RB / 16, RG = TM / 4;              // 16 x 16 threads, TM x 4 dot products each
    constexpr int LA = RB + 4, LB = CB + 4;
    constexpr int NA = RB * (BK / 4) / NT, TPR = NT / RB; // loads per thread and step; scanning threads per row
    constexpr int CW = CB / TPR;                          // columns of a tile per scanning thread
    extern __shared__ __align__(16) float sm[];
    float* As = sm;                                       // [2][BK][LA]
    float* Bs = As + 2 * BK * LA;                         // [2][BK][LB]
    float* keys = Bs + 2 * BK * LB;                       // [RB][LK]
    volatile float* ranks = keys + RB * LK;               // [TPR][RB]: the RANK-th key of every list, see below
    constexpr int RANK = (KCAP + TPR - 1) / TPR;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
    const int row0 = blockIdx.x * RB;
    const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);
    const long long tstride = (long long)H * Cp;
    const T* kb = k + ((long long)b * T_ * H + h) * Cp;   // + token * tstride + c
    const T* qb = q + ((long long)b * S * H + h) * Cp;

    // staging: a warp takes 16 rows x two groups of four channels (conflict-free transposed stores)
    const T* abase[NA];
    int akq[NA], arow[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        const int c = (tid + i * NT) >> 5;
        akq[i] = (lane & 1) + 2 * (c & 1);
        arow[i] = (lane >> 1) + 16 * (c >> 1);
        abase[i] = row0 + arow[i] < T_ ? kb + (row0 + arow[i]) * tstride : nullptr;
    }
    const int bkq = (lane & 1) + 2 * (warp & 1), brow = (lane >> 1) + 16 * (warp >> 1);

    // this thread's row and column share when scanning
    const int srow = tid % RB, sq = tid / RB;
    const int row = row0 + srow;
    const bool row_ok = row < T_;
    const float* kst_row = metric != CONVNN_MATMUL ? kstat + ((long long)b * H + h) * T_ : nullptr;
    const float* qst_row = metric != CONVNN_MATMUL ? qstat + ((long long)b * H + h) * S : nullptr;
    TopList<KCAP> top;
    top.init();

    // (a cluster of `split` CTAs shares the tiles: blockIdx.z is the rank)
    const int ksteps = (Cp + BK - 1) / BK, all_tiles = (S + CB - 1) / CB, each = (all_tiles + split - 1) / split;
    const int first = (int)blockIdx.z * each, ntiles = min(all_tiles, first + each);
    float4 av[NA], bv;
    auto fetch = [&](int ct, int ks) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int c = ks * BK + akq[i] * 4;
            av[i] = abase[i] && c < Cp ? load_upto4<T>(abase[i] + c, Cp - c, vec) : z;
        }
        const int c = ks * BK + bkq * 4, col = ct * CB + brow;
        bv = col < S && c < Cp ? load_upto4<T>(qb + col * tstride + c, Cp - c, vec) : z;
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            float* d = As + (buf * BK + akq[i] * 4) * LA + arow[i];
            d[0] = av[i].x; d[LA] = av[i].y; d[2 * LA] = av[i].z; d[3 * LA] = av[i].w;
        }
        float* d = Bs + (buf * BK + bkq * 4) * LB + brow;
        d[0] = bv.x; d[LB] = bv.y; d[2 * LB] = bv.z; d[3 * LB] = bv.w;
    };

    ranks[tid] = -CUDART_INF_F;
    fetch(first, 0);
    stage(0);
    __syncthreads();
    int buf = 0;
    for (int ct = first; ct < ntiles; ++ct) {
        f32x2 acc[TM][2];
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][0] = acc[i][1] = 0ull;
        for (int ks = 0; ks < ksteps; ++ks, buf ^= 1) {
            const bool last = ks + 1 == ksteps, more = !last || ct + 1 < ntiles;
            if (more) fetch(last ? ct + 1 : ct, last ? 0 : ks + 1);
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[TM];
#pragma unroll
                for (int g = 0; g < RG; ++g) {
                    const float4 v = *reinterpret_cast<const float4*>(As + (buf * BK + kk) * LA + g * (RB / RG) + ty * 4);
                    a[4 * g] = v.x; a[4 * g + 1] = v.y; a[4 * g + 2] = v.z; a[4 * g + 3] = v.w;
                }
                const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(Bs + (buf * BK + kk) * LB + tx * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const f32x2 aa = pack2(a[i], a[i]);
                    acc[i][0] = fma2(aa, bb.x, acc[i][0]);
                    acc[i][1] = fma2(aa, bb.y, acc[i][1]);
                }
            }
            if (last) {
                // keys of this tile (the previous tile's were scanned before the last barrier)
                const int c0 = ct * CB + tx * 4;
                float st[4];
                int cd[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int col = min(c0 + j, S - 1);
                    st[j] = qst_row ? qst_row[col] : 0.f;
                    cd[j] = sampled ? cand[col] : -1;
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const int r = (i >> 2) * (RB / RG) + ty * 4 + (i & 3);
                    float d[4];
                    unpack2(acc[i][0], d[0], d[1]);
                    unpack2(acc[i][1], d[2], d[3]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (metric == CONVNN_COSINE) d[j] *= st[j];
                        else if (metric == CONVNN_EUCLIDEAN) d[j] = fmaf(2.0f, d[j], -st[j]);
                        if (sampled && cd[j] == row0 + r) {
                            const float ks_ = kst_row ? kst_row[row0 + r] : 0.f;
                            if (metric == CONVNN_COSINE) d[j] = -0.1f / ks_;
                            else if (metric == CONVNN_MATMUL) d[j] = -0.1f * sqrt_dk;
                            else d[j] = ks_ - 1.21f;
                        }
                    }
                    *reinterpret_cast<float4*>(keys + r * LK + tx * 4) = make_float4(d[0], d[1], d[2], d[3]);
                }
                __syncthreads();
                const int s0 = ct * CB + sq * CW;
                const float* kr = keys + srow * LK + sq * CW;
                if (ct == first) {                            // the list is filling up
                    if (row_ok) {
#pragma unroll 4
                        for (int j4 = 0; j4 < CW; j4 += 4) {
                            const float4 v = *reinterpret_cast<const float4*>(kr + j4);
                            const float kv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (s0 + j4 + j < S && kv[j] > top.worst()) top.insert_sorted(kv[j], s0 + j4 + j);
                        }
                    }
                } else {
                    // The columns that enter: those above this list's last key and not below the smallest of the lists' RANK-th keys,
                    // which at least KCAP keys of the row reach (the others' may be a tile old: they only grow).  They are taken one per
                    // lane and step, whichever columns the lanes are at.
                    float floor = ranks[srow];
#pragma unroll
                    for (int l = 1; l < TPR; ++l) floor = fminf(floor, ranks[l * RB + srow]);
                    uint32_t mask = 0;
#pragma unroll
                    for (int j4 = 0; j4 < CW; j4 += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(kr + j4);
                        const float kv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) mask |= kv[j] > top.worst() && kv[j] >= floor ? 1u << (j4 + j) : 0u;
                    }
                    if (S - s0 < CW) mask &= S > s0 ? (1u << (S - s0)) - 1u : 0u;
                    if (!row_ok) mask = 0;
                    const int steps = __reduce_max_sync(0xffffffffu, __popc(mask));
#pragma unroll 1
                    for (int n = 0; n < steps; ++n) {
                        const int j = mask ? __ffs(mask) - 1 : 0;
                        const float key = kr[j];
                        if (mask && key > top.worst()) top.insert_sorted(key, s0 + j);
                        mask &= mask - 1;
                    }
                }
                ranks[tid] = top.v[RANK - 1];
            }
            if (more) {
                stage(buf ^ 1);
                __syncthreads();
            }
        }
    }

    // merge the lists of a row: lists 1 .. TPR - 1 through shared memory into list 0
    __syncthreads();
    float* mk = sm;                                       // [TPR - 1][KCAP][RB]
    int* mc = reinterpret_cast<int*>(sm + (TPR - 1) * KCAP * RB);
    if (sq > 0) {
#pragma unroll
        for (int s = 0; s < KCAP; ++s) {
            mk[((sq - 1) * KCAP + s) * RB + srow] = top.v[s];
            mc[((sq - 1) * KCAP + s) * RB + srow] = top.i[s];
        }
    }
    __syncthreads();
    if (sq == 0 && row_ok) {
        for (int l = 0; l < (TPR - 1) * KCAP; ++l) {
            const float key = mk[l * RB + srow];
            if (key >= top.worst() && key > -CUDART_INF_F) top.insert_ordered(key, mc[l * RB + srow]);
        }
    }
    if (split > 1) {
        float2* lists = reinterpret_cast<float2*>(sm);
        __syncthreads();
        if (sq == 0) {
#pragma unroll
            for (int s = 0; s < KCAP; ++s) lists[s * RB + srow] = make_float2(top.v[s], __int_as_float(top.i[s]));
        }
        const ListOutput o{kst_row, cand, idx, val, T_, K, nsel, metric, sampled, sqrt_dk};
        merge_cluster_lists<KCAP>(lists, lists + KCAP * RB, RB, split, (int)blockIdx.z, tid, row0, ((long long)b * H + h) * T_ + row0, true, o);
        return;
    }
    if (sq > 0 || !row_ok) return;

    const float kst = kst_row ? kst_row[row] : 0.f;
    const long long obase = (((long long)b * H + h) * T_ + row) * K;
    int off = 0;
    if (sampled) {
        idx[obase] = row;
        val[obase] = 1.0f;
        off = 1;
    }
#pragma unroll
    for (int s = 0; s < KCAP; ++s) {
        if (s < nsel) {
            const int col = top.i[s];
            const float key = top.v[s];
            float v;
            if (metric == CONVNN_COSINE) v = key * kst;
            else if (metric == CONVNN_MATMUL) v = key / sqrt_dk;
            else v = sqrtf(fmaxf(kst - key, 0.f));
            int tok = col;
            if (sampled) {
                tok = cand[col];
                if (tok == row) v = (metric == CONVNN_EUCLIDEAN) ? 1.1f : -0.1f;
            }
            idx[obase + off + s] = tok;
            val[obase + off + s] = v;
        }
    }
}

// CTAs that share a block's columns where the blocks alone leave room: one CTA of 128 rows fits an SM, two of 64 (us, float32, one CTA per block, a cluster: 577 x
// 577 x 384 209, 75; 8 x 500 x 500 x 64 48, 33; 5000 x 5000 x 193, K = 25 1196, 880; 9363 x 9363 x 192 1467, 1228 with 64 rows).
inline int split_of(const Dims& dm, int rb) {
    const long long ctas = (long long)dm.B * dm.H * ((dm.T + rb - 1) / rb);
    int split = 1;
    while (split < MAX_SPLIT && ctas * 2 * split <= (rb == 128 ? 1ll : 2ll) * device_sms() && dm.S >= 2 * CB * 2 * split) split *= 2;
    return split;
}

template <typename T, int KCAP, int RB>
int launch(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
           const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
    const int split = split_of(dm, RB);
    const size_t smem = smem_bytes(RB, KCAP, split > 1);
    auto kern = sim_topk_simt_kernel<T, KCAP, RB>;
    CONVNN_ENSURE_SMEM(kern, smem);
    const int vec = dm.Cp % 4 == 0 && aligned16(q) && aligned16(k);
    if (split > 1) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = split;
        attr[1] = chained_attribute(st);
        cfg.gridDim = dim3((dm.T + RB - 1) / RB, dm.B * dm.H, split); cfg.blockDim = dim3(NT);
        cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 2;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<const T*>(q), static_cast<const T*>(k), qstat, kstat, cand, idx, val,
                                                 dm.T, dm.S, dm.H, dm.Cp, dm.K, dm.nsel, (int)d->metric, (int)d->sampled,
                                                 (float)sqrt((double)dm.dk), vec, split);
        if (e != cudaSuccess) return set_error(CONVNN_E_CUDA, "sim_topk_simt launch: %s", cudaGetErrorString(e));
        return CONVNN_OK;
    }
    launch_late(sizeof(T) == 4 || d->coord, kern, dim3((dm.T + RB - 1) / RB, dm.B * dm.H), NT, smem, st,
        static_cast<const T*>(q), static_cast<const T*>(k), qstat, kstat, cand, idx, val, dm.T, dm.S, dm.H, dm.Cp, dm.K,
        dm.nsel, d->metric, d->sampled, (float)sqrt((double)dm.dk), vec, 1);
    CONVNN_CHECK_LAUNCH("sim_topk_simt");
    return CONVNN_OK;
}

// Rows per CTA and CTAs.  128 rows per CTA use the pipes better (8 x 4 dot products per thread instead of 4 x 4); 64 where the
// 128-row grid leaves SMs without work or most of a tile is padding.
struct Blocks {
    int rows;
    long long ctas;
};
inline Blocks blocks_of(const Dims& dm) {
    const long long bh = (long long)dm.B * dm.H, wide = (dm.T + 127) / 128 * bh;
    const long long shares = dm.S > 256 ? split_of(dm, 128) : 1;
    if (wide * shares * (shares > 1 ? 2 : 1) >= device_sms() && ((dm.T + 127) / 128) * 128 <= ((dm.T + 63) / 64) * 64 * 5 / 4) return {128, wide};
    return {64, (dm.T + 63) / 64 * bh};
}

template <typename T>
int dispatch(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
             const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
    const bool rows128 = blocks_of(dm).rows == 128;
#define CONVNN_LAUNCH(KC)                                                                                     \
    return rows128 ? launch<T, KC, 128>(d, dm, q, k, qstat, kstat, cand, idx, val, st)                        \
                   : launch<T, KC, 64>(d, dm, q, k, qstat, kstat, cand, idx, val, st)
    // A list longer than needed costs its upkeep: 64 images of 197 tokens, 192 channels, ten to twelve neighbours 88 us with
    // twelve slots, 98 with sixteen; five to eight neighbours 77 with eight, 79 with nine.
    const int n = dm.nsel;
    if (n <= 4) CONVNN_LAUNCH(4);
    if (n <= 8) CONVNN_LAUNCH(8);
    if (n <= 9) CONVNN_LAUNCH(9);
    if (n <= 12) CONVNN_LAUNCH(12);
    if (n <= 16) CONVNN_LAUNCH(16);
    if (n <= 25) CONVNN_LAUNCH(25);
    CONVNN_LAUNCH(32);
#undef CONVNN_LAUNCH
}

}  // namespace simt_topk
}  // namespace convnn
