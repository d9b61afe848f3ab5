// fp32 similarity + top-K for at most 256 candidates: the whole candidate list at once, then a warp per key row.
//
// A CTA of 256 threads owns 32 key tokens of one (batch, head).  Their dot products with all candidates are one
// register-blocked product (8 rows x 4 columns per thread, channels strictly ascending, operands transposed through
// double-buffered shared memory); they become ranking keys in shared memory and the eight warps take four rows each
// (topk_rows.cuh).  The streaming kernel of sim_topk_simt.cuh visits 64 columns at a time in CTAs of 64 or 128 rows and keeps
// two to four lists per row: at 65 tokens it ran a second tile for one column and a second CTA for one row.
#pragma once
#include "sim_topk_simt.cuh"
#include "topk_rows.cuh"

namespace convnn {
namespace simt_topk_rows {

using namespace topk_rows;
using simt_topk::load4;
using simt_topk::load_upto4;

constexpr int NT = 256, NW = NT / 32;
constexpr int RB = 32;      // key rows per CTA
constexpr int BK = 32;      // channels per step
constexpr int LA = RB + 4;

template <typename T, int J, int NS>
__global__ void __launch_bounds__(NT) sim_topk_simt_rows_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const float* __restrict__ qstat, const float* __restrict__ kstat,
    const int32_t* __restrict__ cand, int32_t* __restrict__ idx, float* __restrict__ val, int T_, int S, int H, int Cp, int K,
    int nsel, int metric, int sampled, float sqrt_dk, int vec) {
    chain_wait();               // (and no early start for the next one, see chain_begin_for())
    constexpr int NB = 32 * J, LB = NB + 4;
    extern __shared__ __align__(16) float sm[];
    float* As = sm;                                       // [2][BK][LA]
    float* Bs = As + 2 * BK * LA;                         // [2][BK][LB]
    float* keys = Bs + 2 * BK * LB;                       // [RB][LB]
    float2* found = reinterpret_cast<float2*>(keys + RB * LB);                 // [NW][found_pairs]
    float2* lists = found + NW * found_pairs(NS);                              // [NW][RB / NW][K]
    float* kst_s = reinterpret_cast<float*>(lists + RB * K);                   // [RB]
    int* cs = reinterpret_cast<int*>(kst_s + RB);                              // [NB]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
    const int row0 = blockIdx.x * RB;
    const int cg = warp * 8 + (lane >> 2), rg = lane & 3, ncg = (S + 3) / 4;   // four columns, eight rows of this thread
    const long long tstride = (long long)H * Cp;
    const T* kb = k + ((long long)b * T_ * H + h) * Cp;
    const T* qb = q + ((long long)b * S * H + h) * Cp;
    const float* kst_row = metric != CONVNN_MATMUL ? kstat + (long long)bh * T_ : nullptr;
    const float* qst_row = metric != CONVNN_MATMUL ? qstat + (long long)bh * S : nullptr;
    if (tid < RB) kst_s[tid] = kst_row && row0 + tid < T_ ? kst_row[row0 + tid] : 0.f;
    if (sampled)
        for (int c = tid; c < S; c += NT) cs[c] = cand[c];

    // staging: a warp takes 16 rows x two groups of four channels (conflict-free transposed stores)
    const int arow = (lane >> 1) + 16 * (warp & 1), akq = (lane & 1) + 2 * (warp >> 1);
    const T* abase = row0 + arow < T_ ? kb + (row0 + arow) * tstride : nullptr;
    float4 av, bv[J];
    auto fetch = [&](int ks) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const int c = ks * BK + akq * 4;
        av = abase && c < Cp ? load_upto4<T>(abase + c, Cp - c, vec) : z;
#pragma unroll
        for (int i = 0; i < J; ++i) {
            const int set = i * NW + warp, col = (set % (2 * J)) * 16 + (lane >> 1), cc = ks * BK + ((set / (2 * J)) * 2 + (lane & 1)) * 4;
            bv[i] = col < S && cc < Cp ? load_upto4<T>(qb + col * tstride + cc, Cp - cc, vec) : z;
        }
    };
    auto stage = [&](int buf) {
        float* d = As + (buf * BK + akq * 4) * LA + arow;
        d[0] = av.x; d[LA] = av.y; d[2 * LA] = av.z; d[3 * LA] = av.w;
#pragma unroll
        for (int i = 0; i < J; ++i) {
            const int set = i * NW + warp;
            float* e = Bs + (buf * BK + ((set / (2 * J)) * 2 + (lane & 1)) * 4) * LB + (set % (2 * J)) * 16 + (lane >> 1);
            e[0] = bv[i].x; e[LB] = bv[i].y; e[2 * LB] = bv[i].z; e[3 * LB] = bv[i].w;
        }
    };

    f32x2 acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
    const int ksteps = (Cp + BK - 1) / BK;
    fetch(0);
    stage(0);
    __syncthreads();
    for (int ks = 0; ks < ksteps; ++ks) {
        const int buf = ks & 1;
        const bool more = ks + 1 < ksteps;
        if (more) fetch(ks + 1);
        if (warp * 8 < ncg) {
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                const float4 a0 = *reinterpret_cast<const float4*>(As + (buf * BK + kk) * LA + rg * 8);
                const float4 a1 = *reinterpret_cast<const float4*>(As + (buf * BK + kk) * LA + rg * 8 + 4);
                const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(Bs + (buf * BK + kk) * LB + cg * 4);
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const f32x2 aa = pack2(a[i], a[i]);
                    acc[i][0] = fma2(aa, bb.x, acc[i][0]);
                    acc[i][1] = fma2(aa, bb.y, acc[i][1]);
                }
            }
        }
        if (more) {
            stage(buf ^ 1);
            __syncthreads();
        }
    }

    if (cg < ncg) {
        float st[4];
        int cd[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = min(cg * 4 + j, S - 1);
            st[j] = qst_row ? qst_row[col] : 0.f;
            cd[j] = sampled ? cs[col] : -1;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = rg * 8 + i;
            float d[4];
            unpack2(acc[i][0], d[0], d[1]);
            unpack2(acc[i][1], d[2], d[3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (metric == CONVNN_COSINE) d[j] *= st[j];
                else if (metric == CONVNN_EUCLIDEAN) d[j] = fmaf(2.0f, d[j], -st[j]);
                if (sampled && cd[j] == row0 + r) {
                    const float kst = kst_s[r];
                    if (metric == CONVNN_COSINE) d[j] = -0.1f / kst;
                    else if (metric == CONVNN_MATMUL) d[j] = -0.1f * sqrt_dk;
                    else d[j] = kst - 1.21f;
                }
                if (cg * 4 + j >= S) d[j] = -CUDART_INF_F;
            }
            *reinterpret_cast<float4*>(keys + r * LB + cg * 4) = make_float4(d[0], d[1], d[2], d[3]);
        }
    }
    __syncthreads();
    const RowsTask task{kst_s, cs, idx, val, LB, ncg * 4, nsel, K, inverse_of(K), metric, sampled, sqrt_dk};
    select_and_write<J, NS, NW>(task, keys, lists + warp * (RB / NW) * K,
                                static_cast<uint32_t>(__cvta_generic_to_shared(found + warp * found_pairs(NS))), warp,
                                min(RB, T_ - row0), bh * T_ + row0, row0);
}

template <typename T, int J, int NS>
int launch(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat, const float* kstat,
           const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
    constexpr int LB = 32 * J + 4;
    const size_t smem = (size_t)(2 * BK * LA + 2 * BK * LB + RB * LB + RB + 32 * J) * 4 +
                        (size_t)(NW * found_pairs(NS) + RB * dm.K) * 8;
    auto kern = sim_topk_simt_rows_kernel<T, J, NS>;
    CONVNN_ENSURE_SMEM(kern, smem);
    const int vec = dm.Cp % 4 == 0 && aligned16(q) && aligned16(k);
    launch_late(sizeof(T) == 4 || d->coord, kern, dim3((dm.T + RB - 1) / RB, dm.B * dm.H), NT, smem, st,
        static_cast<const T*>(q), static_cast<const T*>(k), qstat, kstat, cand, idx, val, dm.T, dm.S, dm.H, dm.Cp, dm.K,
        dm.nsel, d->metric, d->sampled ? 1 : 0, (float)sqrt((double)dm.dk), vec);
    CONVNN_CHECK_LAUNCH("sim_topk_simt_rows");
    return CONVNN_OK;
}

// What bounds it: shared-memory reads of the product (12 values per 32 multiply-adds), with one or two CTAs per SM; the
// streaming kernel reads less per multiply-add in its 128-row CTAs and catches up once every SM has several of them.  From
// 8/3 CTAs per SM on the padded work of its busiest SM (rounds x rows x 64-column tiles) is therefore weighed against this
// kernel's, a 32-row CTA of which costs as much as 32 (a S + b).  Long lists cost the streaming kernel more: from 10 on up
// to 25/6 CTAs per SM, above 16 always.  us, streaming -> this kernel (float32, K = 9, one head, unless noted):
//   65 x 65 x 192       1 to 32 images 29 -> 13       256: 52.8 -> 41.9
//   197 x 197 x 192     1: 50.1 -> 19.2    64: 76.3 -> 58.5    256: 209 -> 199 (not taken)
//   577 x 150 x 385 bfloat16, K = 16    7: 101 -> 42    32: 187 -> 134        65 x 65 x 192, K = 25    300: 157 -> 59
//   197 x 64 x 384      16: 30.0 -> 23.5   64: 43.3 -> 51.4 (not taken)       197 x 49, 3 heads of 64  16: 15.7 -> 10.9
//   100 x 100 x 192     150: 0.87 of the time   230: 57.4 -> 64.1 (not taken)   130 x 130 x 400, K = 16  152: 232 -> 123
//   1000 x 100 x 192    18: 43.8 -> 49.6 (not taken)   16 channels, K = 16  18: 34.4 -> 17.8
//   256 x 256 x 400     75: 0.81 of the time   115: 1.25 times (not taken)      100 x 100 x 16, K = 1  230: 11.8 -> 17.3 (not taken)
static bool wanted(const Dims& dm) {
    const long long bh = (long long)dm.B * dm.H, ctas = (dm.T + RB - 1) / RB * bh, sms = device_sms();
    if (dm.S > 256) return false;
    if (dm.nsel > 16 && dm.S > 64) return true;
    const bool light = dm.nsel <= 4 && dm.Cp <= 64;                   // little to select, little to multiply: mostly fixed costs
    if (light && dm.Cp <= 32 && dm.S > 32) return ctas <= 2 * sms;    // (109 x 65 x 40 x 16, K = 1 6.9 -> 7.4 from there on)
    if (ctas <= sms * 8 / 3) return true;
    if (dm.S <= 64 || ctas > sms * 25 / 4) return false;
    const bool few = ctas <= sms * 25 / 6;
    if (dm.nsel >= 10 && few) return true;
    double a = 1.0, b = 50;
    if (dm.Cp > 256) { a = 1.3; b = 40; }
    else if (dm.nsel >= 10) { a = 1.1; b = 20; }
    else if (light) { a = 0.9; b = few ? 110 : 130; }
    const simt_topk::Blocks other = simt_topk::blocks_of(dm);
    const long long streamed = (other.ctas + sms - 1) / sms * other.rows * ((dm.S + 63) / 64 * 64);
    return (double)((ctas + sms - 1) / sms) * RB * (a * dm.S + b) < (double)streamed;
}

template <typename T, int J>
int launch_ns(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat, const float* kstat,
              const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
    if (dm.nsel == 9) return launch<T, J, 9>(d, dm, q, k, qstat, kstat, cand, idx, val, st);
    if (dm.nsel <= 12) return launch<T, J, 0>(d, dm, q, k, qstat, kstat, cand, idx, val, st);
    if (dm.nsel <= 16) return launch<T, J, -3>(d, dm, q, k, qstat, kstat, cand, idx, val, st);
    return launch<T, J, -2>(d, dm, q, k, qstat, kstat, cand, idx, val, st);
}

template <typename T>
int dispatch(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat, const float* kstat,
             const int32_t* cand, int32_t* idx, float* val, cudaStream_t st) {
#define CONVNN_ROWS(J) return launch_ns<T, J>(d, dm, q, k, qstat, kstat, cand, idx, val, st)
    switch ((dm.S + 31) / 32) {
        case 1: CONVNN_ROWS(1);
        case 2: CONVNN_ROWS(2);
        case 3: CONVNN_ROWS(3);
        case 4: CONVNN_ROWS(4);
        case 5: CONVNN_ROWS(5);
        case 6: CONVNN_ROWS(6);
        case 7: CONVNN_ROWS(7);
        default: CONVNN_ROWS(8);
    }
#undef CONVNN_ROWS
}

}  // namespace simt_topk_rows
}  // namespace convnn
