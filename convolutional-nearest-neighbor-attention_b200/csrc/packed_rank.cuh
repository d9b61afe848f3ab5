// Ranking of a row's entries by ONE thread: (key, column) pairs in shared memory, in column order, to a sorted list.
//
// A sorted list takes five instructions per slot and insertion, all on the half-rate pipe.  Here the low bits of a key are
// replaced by the number of its entry, so that a sorting network moves one word per entry, two instructions per exchange.
// Keys that agree in the bits that are left are put in order afterwards, by what the entries hold; where more than two such keys
// meet at the end of the list, the entries are inserted one by one.  The order is the ordered insertion's: larger key first, then lower column.
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

template <int NSEL, int J, class At>
__device__ __forceinline__ void insert_entries(TopList<NSEL>& top, const At& at, int cnt) {
    if constexpr (J < NSEL) {
        if (J < cnt) {
            const float2 x = lds_entry(at(J));
            top.template insert_sorted_first<J>(x.x, __float_as_int(x.y));
        }
        insert_entries<NSEL, J + 1>(top, at, cnt);
    }
}

// What the network takes; more entries than that are inserted.  (Ten to twelve: all of them, 256 x 6 heads of 197 x 197 x 64, K = 12
// 111.6 us, 113.8 with a network of 24.)
template <int NSEL>
constexpr int network_of = NSEL <= 4 ? 8 : NSEL <= 8 ? 12 : NSEL <= 9 ? 16 : NSEL <= 12 ? 0 : NSEL <= 16 ? 28 : NSEL <= 25 ? 44 : 52;

// The best nsel <= NSEL of `cnt` <= 64 entries, entry n at the address at(n); all lanes of a warp call it.  Rows whose keys are
// not all finite ask for the insertion (`insert`), which leaves out -inf.
template <int NSEL, class At>
__device__ __forceinline__ void rank_entries(TopList<NSEL>& top, const At& at, int cnt, int nsel, bool insert) {
    constexpr int N = network_of<NSEL>;
    if constexpr (N < NSEL) {
        top.init();
        insert_entries<NSEL, 0>(top, at, cnt);
        const int most = __reduce_max_sync(0xffffffffu, cnt);
#pragma unroll 1
        for (int n = NSEL; n < most; ++n) {
            if (n < cnt) {
                const float2 x = lds_entry(at(n));
                top.insert_sorted(x.x, __float_as_int(x.y));
            }
        }
    } else {
        constexpr int BITS = N <= 32 ? 5 : 6;
        constexpr uint32_t LOW = (1u << BITS) - 1u;
        float q[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            // (+ 0: minus zero equals zero)
            const uint32_t key = __float_as_uint(lds_key(at(n)) + 0.f);
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
            // (the last place and the first beyond change places like any two, unless a third is as close)
            insert |= c && (NSEL <= 12 || (i == nsel - 1 && close(i + 1) && i + 2 < cnt));
        }
        near_any = near_any && !insert;
        while (NSEL > 12 && __any_sync(0xffffffffu, near_any)) {
            bool moved = false;
#pragma unroll
            for (int i = 0; i < NSEL; ++i) {
                if (near_any && i < nsel && i + 1 < cnt && close(i)) {
                    const uint32_t a = __float_as_uint(q[i]) & LOW, b = __float_as_uint(q[i + 1]) & LOW;
                    const float ka = lds_key(at((int)a)), kb = lds_key(at((int)b));
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
            const float2 e = lds_entry(at(s < cnt ? (int)(__float_as_uint(q[s]) & LOW) : 0));
            top.v[s] = e.x;
            top.i[s] = __float_as_int(e.y);
        }
        if (__any_sync(0xffffffffu, insert)) {
            if (insert) {
                top.init();
                insert_entries<NSEL, 0>(top, at, cnt);
                for (int n = NSEL; n < cnt; ++n) {
                    const float2 x = lds_entry(at(n));
                    top.insert_sorted(x.x, __float_as_int(x.y));
                }
            }
        }
    }
}

// Four words at `at` of shared memory to words i .. i + 3 of `to`, those below n of them; `to` + i is on a 16-byte boundary.
__device__ __forceinline__ void copy_four(int* to, int i, int n, uint32_t at) {
    int4 x;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(at) : "memory");
    if (i >= 0 && i + 4 <= n) {
        *reinterpret_cast<int4*>(to + i) = x;
        return;
    }
    if (i >= 0 && i < n) to[i] = x.x;
    if (i + 1 >= 0 && i + 1 < n) to[i + 1] = x.y;
    if (i + 2 >= 0 && i + 2 < n) to[i + 2] = x.z;
    if (i + 3 >= 0 && i + 3 < n) to[i + 3] = x.w;
}

// The lists of a warp's rows (lane = row, `n_rows` of them) to global memory from word obase on, by one of
//   WORDS   a word at a time, a sector each
//   LINES   through `stage`, where the words lie as they will in global memory, 16-byte boundaries included, so that a row's K
//           words and the next row's leave together; odd K (a row per lane meets no bank twice)
//   SKEWED  through `stage`, pair (row, slot) at slot * 32 + (row + slot) % 32; any K
// `stage`: shared, 16-byte aligned, 256 K + 32 bytes, the entries of these rows.
enum Way { WORDS, LINES, SKEWED };

template <int NSEL, Way WAY, class P>
__device__ __forceinline__ void write_rows(const TopList<NSEL>& top, const P& p, const int* cs, uint32_t stage, long long obase,
                                           int n_rows, int row, float kst) {
    const int lane = threadIdx.x & 31, n = n_rows * p.K;
    auto each = [&](auto put) {
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
    };
    int* idx = p.idx + obase;
    int* val = reinterpret_cast<int*>(p.val) + obase;
    if (WAY != WORDS) __syncwarp();                  // every row's entries have been read
    if (WAY == LINES) {
        const int at_idx = static_cast<int>(reinterpret_cast<uintptr_t>(idx) >> 2) & 3;
        const int at_val = static_cast<int>(reinterpret_cast<uintptr_t>(val) >> 2) & 3;
        const uint32_t vals = stage + 128 * p.K + 16;
        const uint32_t to_idx = stage + (lane * p.K + at_idx) * 4, to_val = vals + (lane * p.K + at_val) * 4;
        if (lane < n_rows)
            each([&](int slot, int tok, float v) {
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(to_idx + slot * 4), "r"(tok) : "memory");
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(to_val + slot * 4), "r"(__float_as_uint(v)) : "memory");
            });
        __syncwarp();
        for (int i = 4 * lane; i < n + 3; i += 128) {
            copy_four(idx, i - at_idx, n, stage + 4 * i);
            copy_four(val, i - at_val, n, vals + 4 * i);
        }
    } else if (WAY == SKEWED) {
        if (lane < n_rows)
            each([&](int slot, int tok, float v) {
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(stage + slot * 256 + ((lane + slot) & 31) * 8), "r"(tok),
                             "r"(__float_as_uint(v)) : "memory");
            });
        __syncwarp();
        const uint32_t inv = (65536u + p.K - 1) / p.K;   // e / K = e * inv >> 16 for e < 32 K, K <= 32
        for (int e = lane; e < n; e += 32) {
            const uint32_t m = e * inv >> 16, slot = e - m * p.K;
            const float2 x = lds_entry(stage + slot * 256 + ((m + slot) & 31) * 8);
            idx[e] = __float_as_int(x.x);
            val[e] = __float_as_int(x.y);
        }
    } else if (lane < n_rows) {
        each([&](int slot, int tok, float v) {
            idx[lane * p.K + slot] = tok;
            val[lane * p.K + slot] = __float_as_int(v);
        });
    }
    if (WAY != WORDS) __syncwarp();                  // (the slots are the next unit's)
}

}  // namespace convnn
