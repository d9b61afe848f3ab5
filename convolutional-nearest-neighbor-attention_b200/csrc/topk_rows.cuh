// Selection with a WARP per key row: the keys of a row lie in shared memory, lane l takes columns l, l + 32, ...
//
//   bound      the nsel-th largest of the 32 lane maxima (nsel warp-wide maxima): at least nsel keys reach it
//   survivors  the keys that reach it (9 of 197: ~10.5) are packed into shared memory
//   rank       every survivor counts the survivors above it: its slot of the list
//
// Two rows are interleaved.  A row with equal keys among its best, with more survivors than the buffer holds, or with fewer
// than nsel keys above -inf (NaN inputs) takes its list one (key, column) maximum at a time instead: lists are those of the
// streaming kernels, lower column first among equal keys.
#pragma once
#include <limits.h>
#include <math_constants.h>

#include <type_traits>

#include "common.cuh"

namespace convnn {
namespace topk_rows {

constexpr int R = 2;                    // rows a warp interleaves

// A block of key rows of one (batch, head) and where its lists go.
struct RowsTask {
    const float* kst;       // shared: statistic of every row
    const int* cs;          // shared: candidate tokens (sampled modes)
    int32_t* idx;
    float* val;
    int pitch, BN;          // words between key rows; columns that hold keys (a multiple of 4)
    int nsel, K, inv_K;     // list length, entries per row, inverse_of(K)
    int metric, sampled;
    float sqrt_dk;
};
// e / K = e * inverse_of(K) >> 16 for e < 16 K, K <= 32
__host__ __device__ constexpr int inverse_of(int K) { return (65536 + K - 1) / K; }
// survivors of a warp: R rows of 32 (64: lists of more than 16) pairs
__host__ __device__ constexpr int found_pairs(int NS) { return R * (NS == -1 || NS == -2 ? 64 : 32); }

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Largest value of the warp (NaN only if every lane holds NaN).
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
template <int N>
__device__ __forceinline__ float max_of(const float (&v)[N], int first, int step) {
    float m = v[first];
    int j = first + step;
#pragma unroll
    for (; j + step < N; j += 2 * step) m = max3(m, v[j], v[j + step]);
    if (j < N) m = fmaxf(m, v[j]);
    return m;
}

__device__ __forceinline__ void sts_entry(uint32_t at, float key, int col) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(__float_as_uint(key)), "r"(col) : "memory");
}

// Exact list of one row under the full (key, column) order, one maximum at a time; keys of -inf and NaN never enter.
template <int J>
__device__ __noinline__ void select_ordered(const float* keys, int BN, int nsel, uint32_t list) {
    const int lane = threadIdx.x & 31;
    float v[J];
#pragma unroll
    for (int j = 0; j < J; ++j) v[j] = 32 * j + lane < BN ? keys[32 * j + lane] : -CUDART_INF_F;
    float last = CUDART_INF_F;
    int last_col = -1;
    for (int s = 0; s < nsel; ++s) {
        float best = -CUDART_INF_F;
        int col = INT_MAX;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int c = 32 * j + lane;
            if ((v[j] < last || (v[j] == last && c > last_col)) && v[j] > best) { best = v[j]; col = c; }
        }
        last = warp_max(best);
        last_col = __reduce_min_sync(0xffffffffu, best == last ? col : INT_MAX);
        if (!(last > -CUDART_INF_F)) last_col = 0;
        if (lane == 0) sts_entry(list + s * 8, last, last_col);
    }
}

// Keys that reach the bound: (key, column) pairs at `at`, which moves on.
__device__ __forceinline__ void store_if_reached(float key, float bound, int col, uint32_t& at) {
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ge.f32 p, %1, %2;\n\t"
                 "@p st.shared.v2.b32 [%0], {%3, %4};\n\t"
                 "@p add.u32 %0, %0, 8;\n\t}"
                 : "+r"(at) : "f"(key), "f"(bound), "r"(__float_as_uint(key)), "r"(col) : "memory");
}
__device__ __forceinline__ float4 lds_v4(uint32_t at) {
    float4 r;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(at) : "memory");
    return r;
}

// R rows of the key buffer at once (rows at, at + NW, ...): J columns per lane, GR groups of them per lane whose maxima give
// the bound, room for 32 E survivors per row at `found`.  Returns the rows (bit r) that need select_ordered().
template <int J, int GR, int E, int NS, int R, int NW>
__device__ __forceinline__ uint32_t select_rows(const RowsTask& p, const float* keybuf, uint32_t found, uint32_t list,
                                                uint32_t list_stride, int at) {
    constexpr int CAP = 32 * E;
    const int lane = threadIdx.x & 31;
    const uint32_t below = (1u << lane) - 1u;
    const int nsel = NS ? NS : p.nsel;
    float v[R][J];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float* kr = keybuf + (at + r * NW) * p.pitch + lane;
#pragma unroll
        for (int j = 0; j < J - 1; ++j) v[r][j] = kr[32 * j];
        v[r][J - 1] = -CUDART_INF_F;
        if (32 * (J - 1) + lane < p.BN) v[r][J - 1] = kr[32 * (J - 1)];
    }
    float m[R][GR], bound[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < GR; ++q) m[r][q] = max_of<J>(v[r], q < J ? q : 0, GR);
#pragma unroll
    for (int r = 0; r < R; ++r) bound[r] = warp_max(GR == 2 ? fmaxf(m[r][0], m[r][GR - 1]) : m[r][0]);
    auto lower = [&] {
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int q = 0; q < GR; ++q) m[r][q] = m[r][q] == bound[r] ? -CUDART_INF_F : m[r][q];
            bound[r] = warp_max(GR == 2 ? fmaxf(m[r][0], m[r][GR - 1]) : m[r][0]);
        }
    };
    if (NS) {
#pragma unroll
        for (int s = 1; s < NS; ++s) lower();
    } else {
#pragma unroll 1
        for (int s = 1; s < nsel; ++s) lower();
    }
    // where each lane's survivors go: exclusive prefix of the lanes' counts, bit by bit
    int mine[R], before[R], n[R], most = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        mine[r] = 0;
#pragma unroll
        for (int j = 0; j < J; ++j)
            if (v[r][j] >= bound[r]) ++mine[r];
        before[r] = __popc(__ballot_sync(0xffffffffu, mine[r] & 1) & below);
        if (J >= 2) before[r] += 2 * __popc(__ballot_sync(0xffffffffu, mine[r] & 2) & below);
        most = max(most, mine[r]);
    }
    if (J >= 4 && __any_sync(0xffffffffu, most >= 4)) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            before[r] += 4 * __popc(__ballot_sync(0xffffffffu, mine[r] & 4) & below);
            if (J >= 8) before[r] += 8 * __popc(__ballot_sync(0xffffffffu, mine[r] & 8) & below);
        }
    }
    uint32_t redo = 0;
    int n_max = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) n[r] = __shfl_sync(0xffffffffu, before[r] + mine[r], 31);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (n[r] > CAP || !(bound[r] > -CUDART_INF_F)) {
            redo |= 1u << r;                     // (keys of +inf may still be stored: a lane's J from slot 0 on)
            n[r] = 0;
            bound[r] = CUDART_INF_F;
            before[r] = 0;
        }
        n_max = max(n_max, n[r]);
        uint32_t to = found + (r * CAP + before[r]) * 8;
#pragma unroll
        for (int j = 0; j < J; ++j) store_if_reached(v[r][j], bound[r], 32 * j + lane, to);
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (lane + 32 * e >= n[r])
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(found + (r * CAP + lane + 32 * e) * 8), "r"(0xff800000u) : "memory");
    }
    __syncwarp();
    float key[R][E];
    int col[R][E], rank[R][E];
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=f"(key[r][e]), "=r"(col[r][e])
                         : "r"(found + (r * CAP + lane + 32 * e) * 8) : "memory");
            rank[r][e] = 0;
        }
    }
    auto count_above = [&](int i) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float4 a = lds_v4(found + (r * CAP + i) * 8), b = lds_v4(found + (r * CAP + i) * 8 + 16);
#pragma unroll
            for (int e = 0; e < E; ++e) {
                if (a.x > key[r][e]) ++rank[r][e];
                if (a.z > key[r][e]) ++rank[r][e];
                if (b.x > key[r][e]) ++rank[r][e];
                if (b.z > key[r][e]) ++rank[r][e];
            }
        }
    };
    constexpr int FIRST = NS ? (NS + 3) / 4 * 4 : 0;    // (9 of 197 columns: 12 survivors suffice for nine rows in ten)
#pragma unroll
    for (int i = 0; i < FIRST; i += 4) count_above(i);
#pragma unroll 1
    for (int i = FIRST; i < n_max; i += 4) count_above(i);
    __syncwarp();
    // A lane past the survivors holds -inf and rank n.  Equal keys share a rank and leave a later one out: the list is right
    // if the ranks below nsel all occur and are nsel in number.
    const uint32_t all = nsel == 32 ? 0xffffffffu : (1u << nsel) - 1u;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        uint32_t bits = 0;
        int listed = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool in = rank[r][e] < nsel;
            listed += __popc(__ballot_sync(0xffffffffu, in));
            if (in) bits |= 1u << rank[r][e];
        }
        const bool good = __reduce_or_sync(0xffffffffu, bits) == all && listed == nsel && !(redo >> r & 1u);
        if (!good) redo |= 1u << r;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (good && rank[r][e] < nsel) sts_entry(list + r * list_stride + rank[r][e] * 8, key[r][e], col[r][e]);
    }
    return redo;
}

// The rows w, w + NW, ... below n_rows of a key buffer (tokens row0 + r of their sequence): lists through `list` (room for K
// pairs per row of the warp), then sink(row of the warp, slot, token, value) for every entry.  Returns the rows of the warp.
// NS: number of neighbours where it is fixed, 0: any up to 12, -3: 13 to 16, -1: up to 25, -2: up to 32.  From 13 on (up to 16: of more
// than 128 keys) two maxima per lane give the bound: of 197 keys 48 reach the 25th of 32 maxima, so that a row in two hundred overflowed the buffer and the
// batch waited for its ordered list, but 29 reach the 25th of 64 (us, one maximum, two: 3 x 197 x 197 x 32, K = 25 18.0, 8.2; 20 x 197 x
// 197 x 96 20.9, 10.8; 64 x 197 x 197 x 192, K = 16 20.5, 15.6).
template <int J, int NS, int NW, class Sink>
__device__ __forceinline__ int select_lists(const RowsTask& p, const float* keybuf, float2* list, uint32_t found0, int w,
                                            int n_rows, int row0, Sink sink) {
    constexpr int E = NS == -1 || NS == -2 ? 2 : 1, GR = NS < 0 && J > (NS == -3 ? 4 : 1) ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const uint32_t list0 = static_cast<uint32_t>(__cvta_generic_to_shared(list + p.sampled)), list_stride = p.K * 8;
    uint32_t redo = 0;                       // bit n: row w + n NW
    int n = 0;
    auto select = [&](auto rows) {
        constexpr int RR = decltype(rows)::value;
        redo |= select_rows<J, GR, E, (NS > 0 ? NS : 0), RR, NW>(p, keybuf, found0, list0 + n * list_stride, list_stride,
                                                                 w + n * NW) << n;
        n += RR;
    };
    while (w + (n + R - 1) * NW < n_rows) select(std::integral_constant<int, R>{});
    if (w + n * NW < n_rows) select(std::integral_constant<int, 1>{});
    for (; redo; redo &= redo - 1) {
        const int m = __ffs(redo) - 1;
        __syncwarp();
        select_ordered<J>(keybuf + (w + m * NW) * p.pitch, p.BN, p.nsel, list0 + m * list_stride);
    }
    __syncwarp();
    // keys back to similarity values, columns back to tokens, the row itself first in the sampled modes
    for (int e = lane; e < n * p.K; e += 32) {
        const int m = (int)((uint32_t)e * p.inv_K >> 16), slot = e - m * p.K;
        const int rw = w + m * NW, row = row0 + rw;
        int tok = row;
        float s = 1.0f;
        if (!p.sampled || slot) {
            const float2 f = list[e];
            const float kst = p.kst[rw];
            tok = __float_as_int(f.y);
            if (p.metric == CONVNN_COSINE) s = f.x * kst;
            else if (p.metric == CONVNN_MATMUL) s = f.x / p.sqrt_dk;
            else s = sqrtf(fmaxf(kst - f.x, 0.f));
            if (p.sampled) {
                tok = p.cs[tok];
                if (tok == row) s = (p.metric == CONVNN_EUCLIDEAN) ? 1.1f : -0.1f;
            }
        }
        sink(m, slot, tok, s);
    }
    __syncwarp();
    return n;
}

// The same with the lists written to global memory, as rows g + r of the flattened (batch, head, row) order.
template <int J, int NS, int NW>
__device__ __forceinline__ void select_and_write(const RowsTask& p, const float* keybuf, float2* list, uint32_t found0, int w,
                                                 int n_rows, int g, int row0) {
    select_lists<J, NS, NW>(p, keybuf, list, found0, w, n_rows, row0, [&](int m, int slot, int tok, float s) {
        const int to = (g + w + m * NW) * p.K + slot;    // (B H T K < 2^31)
        p.idx[to] = tok;
        p.val[to] = s;
    });
}

}  // namespace topk_rows
}  // namespace convnn
