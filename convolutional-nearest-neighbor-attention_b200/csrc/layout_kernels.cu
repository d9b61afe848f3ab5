// Small data-movement kernels around the tensor-core GEMMs.
//   gather_rows   xq[b, r, :] = x[b, cand[r], :]   (candidate tokens of the sampled modes,
//                 reference layers.py:285, 298) so the query projection is a plain GEMM
//   merge_heads   the reference's flat head reinterpretation for H > 1 (layers.py:247-259):
//                 y[b, t', h*dk + c'] = flat(o[b, h])[c'*T + t'], a (dk x T) -> (T x dk)
//                 transpose per (batch, head), staged through shared memory: 16-byte accesses on both sides
//                 (128 x 197 x 12 heads of 32: 30 us in 2-byte tiles, 11 us now)
#include "common.cuh"

namespace convnn {
namespace {

template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ x, long long ldx, const int32_t* __restrict__ cand,
                                   T* __restrict__ xq, int Tn, int S, int D, long long total_vec, int vec) {
    chain_begin_for<T>();
    const int per_row = D / vec;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total_vec;
         i += (long long)gridDim.x * blockDim.x) {
        const int cv = (int)(i % per_row);
        const long long br = i / per_row;
        const int r = (int)(br % S);
        const long long b = br / S;
        const T* src = x + (b * Tn + cand[r]) * ldx + (long long)cv * vec;
        T* dst = xq + br * D + (long long)cv * vec;
        if (vec * sizeof(T) == 16) {
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
        } else {
            for (int e = 0; e < vec; ++e) dst[e] = src[e];
        }
    }
}

// Sequences of which eight channels exceed shared memory: 32 x 32 tiles.
template <typename T>
__global__ void merge_heads_tile_kernel(const T* __restrict__ o, T* __restrict__ y, int Tn, int H, int dk, int D) {
    chain_begin_for<T>();
    __shared__ T tile[32][33];
    const int bh = blockIdx.z;
    const int b = bh / H, h = bh - b * H;
    const T* src = o + (long long)bh * Tn * dk;          // viewed as (dk, T): src[c * T + t]
    const int t0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int c = c0 + i, t = t0 + threadIdx.x;
        if (c < dk && t < Tn) tile[i][threadIdx.x] = src[(long long)c * Tn + t];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int t = t0 + i, c = c0 + threadIdx.x;
        if (t < Tn && c < dk) y[((long long)b * Tn + t) * D + h * dk + c] = tile[threadIdx.x][i];
    }
}

// One CTA per CB of a (batch, head)'s dk channels: CB * T consecutive elements of `o`, brought into shared memory with
// 16-byte loads, leave as VEC-channel vectors of the T token rows.  Eight token rows x four channel vectors per warp: the
// 2-byte reads of a vector fall into different banks for odd T, the stores are whole sectors.
template <typename T, int VEC>
__global__ void __launch_bounds__(256) merge_heads_kernel(const T* __restrict__ o, T* __restrict__ y, int Tn, int H, int dk,
                                                          int D, int CB) {
    chain_begin_for<T>();
    extern __shared__ __align__(16) unsigned char mh_smem[];
    T* s = reinterpret_cast<T*>(mh_smem);                 // [CB][Tn]
    constexpr int PER = 16 / sizeof(T);
    const int bh = blockIdx.x, b = bh / H, h = bh - b * H;
    const int c0 = blockIdx.y * CB, nc = min(CB, dk - c0);
    const T* src = o + ((long long)bh * dk + c0) * Tn;    // viewed as (dk, T)
    const int n = nc * Tn;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        for (int i = threadIdx.x; i < n / PER; i += 256) reinterpret_cast<uint4*>(s)[i] = reinterpret_cast<const uint4*>(src)[i];
        for (int i = n / PER * PER + threadIdx.x; i < n; i += 256) s[i] = src[i];
    } else {
        for (int i = threadIdx.x; i < n; i += 256) s[i] = src[i];
    }
    __syncthreads();
    T* dst = y + (long long)b * Tn * D + h * dk + c0;
    const int nv = nc / VEC, g4 = (nv + 3) / 4 * 4;       // channel vectors, four side by side
    for (int i = threadIdx.x; i < (Tn + 7) / 8 * 8 * g4; i += 256) {
        const int l = i & 31, blk = i >> 5;
        const int cv = (blk % (g4 / 4)) * 4 + (l & 3), t = blk / (g4 / 4) * 8 + (l >> 2);
        if (cv >= nv || t >= Tn) continue;
        __align__(16) T v[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) v[e] = s[(cv * VEC + e) * Tn + t];
        T* d = dst + (long long)t * D + cv * VEC;
        if (VEC * sizeof(T) == 16) *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(v);
        else
#pragma unroll
            for (int e = 0; e < VEC; ++e) d[e] = v[e];
    }
}

template <typename T>
int merge_heads(const void* o, void* y, int B, int Tn, int H, int dk, cudaStream_t st) {
    constexpr int V = 16 / sizeof(T);
    const bool vec = dk % V == 0 && aligned16(y);         // (D = H * dk)
    int CB = (int)(40 * 1024 / ((size_t)Tn * sizeof(T)));
    CB = CB / 32 * 32 ? CB / 32 * 32 : (CB / V * V ? CB / V * V : V);
    if (CB > dk) CB = dk;
    const size_t smem = (size_t)CB * Tn * sizeof(T);
    if (smem > 200 * 1024) {
        launch_chained(merge_heads_tile_kernel<T>, dim3((Tn + 31) / 32, (dk + 31) / 32, B * H), dim3(32, 8), 0, st, 
            static_cast<const T*>(o), static_cast<T*>(y), Tn, H, dk, H * dk);
        CONVNN_CHECK_LAUNCH("merge_heads");
        return CONVNN_OK;
    }
    const dim3 grid(B * H, (dk + CB - 1) / CB);
    if (vec) {
        auto kern = merge_heads_kernel<T, V>;
        CONVNN_ENSURE_SMEM(kern, smem);
        launch_chained(kern, grid, 256, smem, st, static_cast<const T*>(o), static_cast<T*>(y), Tn, H, dk, H * dk, CB);
    } else {
        auto kern = merge_heads_kernel<T, 1>;
        CONVNN_ENSURE_SMEM(kern, smem);
        launch_chained(kern, grid, 256, smem, st, static_cast<const T*>(o), static_cast<T*>(y), Tn, H, dk, H * dk, CB);
    }
    CONVNN_CHECK_LAUNCH("merge_heads");
    return CONVNN_OK;
}

}  // namespace

int launch_gather_rows(int dtype, const void* x, long long ldx, const int32_t* cand, void* xq, int B, int Tn, int S,
                       int D, cudaStream_t st) {
    const size_t elt = dtype == CONVNN_F32 ? 4 : 2;
    int vec = (int)(16 / elt);
    if (D % vec != 0 || ldx % vec != 0 || !aligned16(x) || !aligned16(xq)) vec = 1;
    const long long total = (long long)B * S * (D / vec);
    int blocks = (int)((total + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    if (dtype == CONVNN_F32)
        launch_chained(gather_rows_kernel<float>, blocks, 256, 0, st, static_cast<const float*>(x), ldx, cand,
                                                         static_cast<float*>(xq), Tn, S, D, total, vec);
    else
        launch_chained(gather_rows_kernel<__nv_bfloat16>, blocks, 256, 0, st, static_cast<const __nv_bfloat16*>(x), ldx, cand,
                                                                 static_cast<__nv_bfloat16*>(xq), Tn, S, D, total, vec);
    CONVNN_CHECK_LAUNCH("gather_rows");
    return CONVNN_OK;
}

int launch_merge_heads(int dtype, const void* o, void* y, int B, int Tn, int H, int dk, cudaStream_t st) {
    return dtype == CONVNN_F32 ? merge_heads<float>(o, y, B, Tn, H, dk, st) : merge_heads<__nv_bfloat16>(o, y, B, Tn, H, dk, st);
}

}  // namespace convnn
