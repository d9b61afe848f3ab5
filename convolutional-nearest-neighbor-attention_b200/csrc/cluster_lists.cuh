// Lists of the same rows over shares of the columns, one per CTA of a cluster, merged through distributed shared memory.
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace convnn {

constexpr int MAX_SPLIT = 8;

// What turns a row's merged keys into its output.
struct ListOutput {
    const float* kstat;      // of the (batch, head)
    const int32_t* cand;
    int32_t* idx;
    float* val;
    int T, K, nsel, metric, sampled;
    float sqrt_dk;
};

// `lists`: this CTA's, [slot][rows], best first, of columns that ascend with the rank (so that of equal keys the lower rank's goes first);
// `all`: as much room again.  Every thread of the CTA calls it, tid >= 0 those that work (at least `rows` of them); CTA r takes rows
// r * rows / split ... of `row0`, `base` is the first row's place in the output.
template <int NSEL>
__device__ __forceinline__ void merge_cluster_lists(float2* lists, float2* all, int rows, int split, int rank, int tid, int row0,
                                                    long long base, bool write, const ListOutput& o) {
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int share = rows / split;
    if (tid >= 0 && tid < rows) {
        const int from = tid / share, rr = tid - from * share;
        uint32_t theirs;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs)
                     : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(lists + rank * share + rr))), "r"(from));
        float2 e[NSEL];
#pragma unroll
        for (int s = 0; s < NSEL; ++s)
            asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(e[s].x), "=f"(e[s].y) : "r"(theirs + s * rows * 8) : "memory");
#pragma unroll
        for (int s = 0; s < NSEL; ++s) all[(from * NSEL + s) * share + rr] = e[s];
    }
    __syncthreads();
    const int row = row0 + rank * share + tid;
    if (tid >= 0 && tid < share && row < o.T && write) {
        const float kst = o.metric != CONVNN_MATMUL ? o.kstat[row] : 1.0f;
        long long at = (base + rank * share + tid) * o.K;
        if (o.sampled) {
            o.idx[at] = row;
            o.val[at++] = 1.0f;
        }
        float2 head[MAX_SPLIT];
        int next[MAX_SPLIT];
#pragma unroll
        for (int l = 0; l < MAX_SPLIT; ++l) {
            next[l] = 1;
            head[l] = l < split ? all[l * NSEL * share + tid] : make_float2(-CUDART_INF_F, 0.f);
        }
#pragma unroll 1
        for (int s = 0; s < o.nsel; ++s, ++at) {
            float2 best = head[0];
            int from = 0;
#pragma unroll
            for (int l = 1; l < MAX_SPLIT; ++l)
                if (head[l].x > best.x) { best = head[l]; from = l; }
            // (the last place of a list is taken by the last round at the earliest)
            int pos = 0;
#pragma unroll
            for (int l = 0; l < MAX_SPLIT; ++l) pos = l == from ? next[l] : pos;
            const float2 after = all[(from * NSEL + min(pos, NSEL - 1)) * share + tid];
#pragma unroll
            for (int l = 0; l < MAX_SPLIT; ++l) {
                head[l] = l == from ? after : head[l];
                next[l] += l == from ? 1 : 0;
            }
            int tok = __float_as_int(best.y);
            float v;
            if (o.metric == CONVNN_COSINE) v = best.x * kst;
            else if (o.metric == CONVNN_MATMUL) v = best.x / o.sqrt_dk;
            else v = sqrtf(fmaxf(kst - best.x, 0.f));
            if (o.sampled) {
                tok = o.cand[tok];
                if (tok == row) v = (o.metric == CONVNN_EUCLIDEAN) ? 1.1f : -0.1f;
            }
            o.idx[at] = tok;
            o.val[at] = v;
        }
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // nobody reads this CTA's lists any more
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace convnn
