// Ranking of a row's entries by ONE thread: (key, column) pairs in shared memory, in column order, to a sorted list.
//
// A sorted list takes five instructions per slot and insertion, all on the half-rate pipe.  Here the low bits of a key are
// replaced by the number of its entry, so that a sorting network moves one word per entry, two instructions per exchange.
// Keys that agree in the bits that are left are put in order afterwards, by what the entries hold; where such keys meet at the
// end of the list, the entries are inserted one by one.  The order is the ordered insertion's: larger key first, then lower column.
#pragma once
#include <math_constants.h>

#include "common.cuh"
#include "toplist.cuh"

namespace convnn {

// Descending sort (Batcher's merge exchange, any N); exchanges that only order unused outputs fall away.
template <int N>
__device__ __forceinline__ void sort_descending(float (&v)[N]) {
#pragma unroll
    for (int p = 1; p < N; p *= 2)
#pragma unroll
        for (int k = p; k >= 1; k /= 2)
#pragma unroll
            for (int x = 0; x < N; ++x) {
                const int j = k % p;
                if (x >= j && ((x - j) / k) % 2 == 0 && x + k < N && x / (2 * p) == (x + k) / (2 * p)) {
                    const float a = v[x], b = v[x + k];
                    v[x] = fmaxf(a, b);
                    v[x + k] = fminf(a, b);
                }
            }
}

__device__ __forceinline__ float2 lds_entry(uint32_t at) {
    float2 e;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(e.x), "=f"(e.y) : "r"(at) : "memory");
    return e;
}
__device__ __forceinline__ float lds_key(uint32_t at) {
    float k;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(k) : "r"(at) : "memory");
    return k;
}

template <int NSEL, int J>
__device__ __forceinline__ void insert_entries(TopList<NSEL>& top, uint32_t first, uint32_t stride, int cnt) {
    if constexpr (J < NSEL) {
        if (J < cnt) {
            const float2 x = lds_entry(first + J * stride);
            top.template insert_sorted_first<J>(x.x, __float_as_int(x.y));
        }
        insert_entries<NSEL, J + 1>(top, first, stride, cnt);
    }
}

// What the network takes; more entries than that are inserted.
template <int NSEL>
constexpr int network_of = NSEL <= 16 ? 24 : NSEL <= 25 ? 40 : 52;

// The best nsel <= NSEL of `cnt` <= SLOTS <= 64 entries at first, first + stride, ...; all lanes of a warp call it.  Rows whose
// keys are not all finite ask for the insertion (`insert`), which leaves out -inf.
template <int NSEL, int SLOTS>
__device__ __forceinline__ void rank_entries(TopList<NSEL>& top, uint32_t first, uint32_t stride, int cnt, int nsel, bool insert) {
    constexpr int N = network_of<NSEL>;
    constexpr int BITS = N <= 32 ? 5 : 6;
    constexpr uint32_t LOW = (1u << BITS) - 1u;
    float q[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        // (+ 0: minus zero equals zero)
        const uint32_t key = __float_as_uint(lds_key(first + min(n, SLOTS - 1) * stride) + 0.f);
        q[n] = n < cnt ? __uint_as_float((key & ~LOW) | (uint32_t)n) : -CUDART_INF_F;
    }
    sort_descending(q);
    auto close = [&](int i) { return ((__float_as_uint(q[i]) ^ __float_as_uint(q[i + 1])) & ~LOW) == 0; };
    // (past the last entry there is -inf, which is close to nothing but itself; no two of a list's places are past it)
    insert |= cnt > N;
    bool near_any = false;
#pragma unroll
    for (int i = 0; i < NSEL; ++i) {
        const bool c = close(i) && i < nsel && i + 1 < cnt;
        near_any |= c;
        insert |= c && i == nsel - 1;
    }
    near_any = near_any && !insert;
    while (__any_sync(0xffffffffu, near_any)) {
        bool moved = false;
#pragma unroll
        for (int i = 0; i + 1 < NSEL; ++i) {
            if (near_any && i + 1 < nsel && close(i)) {
                const uint32_t a = __float_as_uint(q[i]) & LOW, b = __float_as_uint(q[i + 1]) & LOW;
                const float ka = lds_key(first + a * stride), kb = lds_key(first + b * stride);
                if (kb > ka || (kb == ka && b < a)) {
                    const float t = q[i];
                    q[i] = q[i + 1];
                    q[i + 1] = t;
                    moved = true;
                }
            }
        }
        near_any = moved;
    }
#pragma unroll
    for (int s = 0; s < NSEL; ++s) {
        const float2 e = lds_entry(first + (s < cnt ? __float_as_uint(q[s]) & LOW : 0u) * stride);
        top.v[s] = e.x;
        top.i[s] = __float_as_int(e.y);
    }
    if (__any_sync(0xffffffffu, insert)) {
        if (insert) {
            top.init();
            insert_entries<NSEL, 0>(top, first, stride, cnt);
            for (int n = NSEL; n < cnt; ++n) {
                const float2 x = lds_entry(first + n * stride);
                top.insert_sorted(x.x, __float_as_int(x.y));
            }
        }
    }
}

// The lists of a warp's rows (lane = row, `n_rows` of them) to global memory, through the warp's entry slots at `stage` (stage +
// slot * stride: 32 pairs), so that a row's K words and those of the next row leave together.
template <int NSEL, class P>
__device__ __forceinline__ void write_rows(const TopList<NSEL>& top, const P& p, const int* cs, uint32_t stage, uint32_t stride,
                                           long long obase, int n_rows, int row, float kst) {
    const int lane = threadIdx.x & 31;
    auto put = [&](int slot, int tok, float v) {
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(stage + slot * stride + ((lane + slot) & 31) * 8), "r"(tok),
                     "r"(__float_as_uint(v)) : "memory");
    };
    __syncwarp();                                    // every row's entries have been read
    if (lane < n_rows) {
        if (p.sampled) put(0, row, 1.0f);
#pragma unroll
        for (int s = 0; s < NSEL; ++s) {
            if (s < p.nsel) {
                int tok = top.i[s];
                float v;
                if (p.metric == CONVNN_COSINE) v = top.v[s] * kst;
                else if (p.metric == CONVNN_MATMUL) v = top.v[s] / p.sqrt_dk;
                else v = sqrtf(fmaxf(kst - top.v[s], 0.f));
                if (p.sampled) {
                    tok = cs[tok];
                    if (tok == row) v = (p.metric == CONVNN_EUCLIDEAN) ? 1.1f : -0.1f;
                }
                put(s + p.sampled, tok, v);
            }
        }
    }
    __syncwarp();
    const uint32_t inv = (65536u + p.K - 1) / p.K;   // e / K = e * inv >> 16 for e < 32 K, K <= 32
    for (uint32_t e = lane; e < (uint32_t)(n_rows * p.K); e += 32) {
        const uint32_t m = e * inv >> 16, slot = e - m * p.K;
        const float2 x = lds_entry(stage + slot * stride + ((m + slot) & 31) * 8);
        p.idx[obase + e] = __float_as_int(x.x);
        p.val[obase + e] = x.y;
    }
    __syncwarp();                                    // (the slots are the next unit's)
}

}  // namespace convnn
