// Neighbour weighting + gather + K-tap stride-K Conv1d (reference layers.py:389-406, 313).
//
// Weights over the K selected values (softmax, raw value, or reciprocal distance) are computed
// once per token into shared memory, then
//   depthwise            o[t, c] = sum_j w[j, c] * p[t, j] * v[idx[t, j], c]
//   standard             o[t, o] = sum_{j, c} w[o, j, c] * p[t, j] * v[idx[t, j], c]
//   depthwise-separable  depthwise, then a (d_k x C) matrix
// Kernels, in the order the dispatcher tries them:
//   * depthwise with 16-byte rows: gather_conv_dw_stream.cu (short bfloat16 sequences, V through shared memory) and
//     gather_conv_dw.cu; other channel counts: a scalar kernel here;
//   * bfloat16 standard, heads of 16, 32 or 64 channels, where it is faster: conv_std_tc.cu, whose neighbour block stays on the SM;
//   * bfloat16 standard / separable on the tensor cores: a gather kernel writes the GEMM's A
//     operand (the weighted neighbour block, or the depthwise result) and gemm_tc multiplies it
//     with the (d_k, K*C) tap matrix / the (d_k, C) pointwise matrix;
//   * float32, and the coordinate channel: the SIMT GEMM, standard with the neighbour block as its implicit A operand,
//     separable over the depthwise result;
//   * channel counts that are no multiple of four: shared-memory staged block times the weights.
// The three K-times expanded copies of V that the reference builds never exist (the tensor-core
// standard conv of the other shapes materialises the weighted block once, in bfloat16).
#include "common.cuh"
#include "token_weights.cuh"

namespace convnn {
namespace {

constexpr int THREADS = 256;

// ---- depthwise, channel counts whose rows are no multiple of 16 bytes ------------------------------------------
template <typename T, int TT>
__global__ void __launch_bounds__(THREADS) gather_conv_dw_scalar_kernel(
    const T* __restrict__ v, const int32_t* __restrict__ idx, const float* __restrict__ val,
    const T* __restrict__ wconv, T* __restrict__ o, int T_, int H, int dk, int Cp, int K, int maximum,
    int softmax) {
    chain_begin_for<T>();
    __shared__ float ps[TT][kMaxK];
    __shared__ int ns[TT][kMaxK];
    const int bh = blockIdx.y;
    const int b = bh / H, h = bh - b * H;
    const int t0 = blockIdx.x * TT;
    const int nt = min(TT, T_ - t0);
    const long long nbase = ((long long)bh * T_ + t0) * K;
    for (int e = threadIdx.x; e < nt * K; e += THREADS) ns[e / K][e % K] = idx[nbase + e];
    if (threadIdx.x < nt) token_weights(val + nbase + (long long)threadIdx.x * K, ps[threadIdx.x], K, maximum, softmax);
    __syncthreads();
    const T* vb = v + ((long long)b * T_ * H + h) * Cp;
    const long long tstride = (long long)H * Cp;
    for (int item = threadIdx.x; item < nt * dk; item += THREADS) {
        const int tt = item / dk, c = item - tt * dk;
        float acc = 0.f;
        for (int j = 0; j < K; ++j)
            acc = fmaf(to_f32<T>(wconv[j * dk + c]), ps[tt][j] * to_f32<T>(vb[ns[tt][j] * tstride + c]), acc);
        o[((long long)bh * T_ + t0 + tt) * dk + c] = from_f32<T>(acc);
    }
}

// ---- standard / depthwise-separable --------------------------------------------------
// Dynamic shared memory: P[TT][JC * C] floats (weighted neighbour block for JC taps, or
// the depthwise result with JC = 1 for the separable type).
template <typename T, int ITEMS>
__global__ void __launch_bounds__(THREADS) gather_conv_mat_kernel(
    const T* __restrict__ v, const int32_t* __restrict__ idx, const float* __restrict__ val,
    const T* __restrict__ wconv, const T* __restrict__ wpw, T* __restrict__ o, int T_, int H, int dk,
    int C, int Cp, int K, int maximum, int softmax, int separable, int TT, int JC) {
    chain_begin_for<T>();
    extern __shared__ __align__(16) float P[];
    __shared__ float ps[32][kMaxK];
    __shared__ int ns[32][kMaxK];
    const int bh = blockIdx.y;
    const int b = bh / H, h = bh - b * H;
    const int t0 = blockIdx.x * TT;
    const int nt = min(TT, T_ - t0);
    const long long nbase = ((long long)bh * T_ + t0) * K;
    for (int e = threadIdx.x; e < nt * K; e += THREADS) ns[e / K][e % K] = idx[nbase + e];
    if (threadIdx.x < nt) token_weights(val + nbase + (long long)threadIdx.x * K, ps[threadIdx.x], K, maximum, softmax);
    __syncthreads();

    const T* vb = v + ((long long)b * T_ * H + h) * Cp;
    const long long tstride = (long long)H * Cp;
    const int tgroups = (TT + 3) / 4;
    const int n_items = dk * tgroups;
    float acc[ITEMS][4];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[it][e] = 0.f;

    const int ntaps = separable ? 1 : K;
    const int pstride = JC * C;
    for (int j0 = 0; j0 < ntaps; j0 += JC) {
        const int jn = min(JC, ntaps - j0);
        // fill P (zero rows for tokens past the end so the matrix step needs no guard)
        for (int e = threadIdx.x; e < TT * jn * C; e += THREADS) {
            const int tt = e / (jn * C);
            const int r = e - tt * jn * C;
            const int jj = r / C, c = r - jj * C;
            float x = 0.f;
            if (tt < nt) {
                if (separable) {
                    for (int j = 0; j < K; ++j)
                        x = fmaf(to_f32<T>(wconv[j * C + c]),
                                 ps[tt][j] * to_f32<T>(vb[ns[tt][j] * tstride + c]), x);
                } else {
                    const int j = j0 + jj;
                    x = ps[tt][j] * to_f32<T>(vb[ns[tt][j] * tstride + c]);
                }
            }
            P[tt * pstride + r] = x;
        }
        __syncthreads();
        // standard: w[oc][j*C + c] (d_k, K*C);  separable stage 1: w[oc][c] (d_k, C)
        const T* wm = separable ? wpw : wconv + (long long)j0 * C;
        const long long wld = separable ? C : (long long)K * C;
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int item = threadIdx.x + it * THREADS;
            if (item < n_items) {
                const int oc = item % dk, tg = item / dk;
                const float* p0 = P + (tg * 4) * pstride;
                for (int r = 0; r < jn * C; ++r) {
                    const float w = to_f32<T>(wm[(long long)oc * wld + r]);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (tg * 4 + e < TT) acc[it][e] = fmaf(w, p0[e * pstride + r], acc[it][e]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const int item = threadIdx.x + it * THREADS;
        if (item < n_items) {
            const int oc = item % dk, tg = item / dk;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tt = tg * 4 + e;
                if (tt < nt) o[((long long)bh * T_ + t0 + tt) * dk + oc] = from_f32<T>(acc[it][e]);
            }
        }
    }
}

template <typename T>
int launch_dw_scalar(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                     const void* w_conv, void* o, cudaStream_t st) {
    constexpr int TT = 16;
    dim3 grid((dm.T + TT - 1) / TT, dm.B * dm.H);
    launch_chained(gather_conv_dw_scalar_kernel<T, TT>, grid, THREADS, 0, st, 
        static_cast<const T*>(v), idx, val, static_cast<const T*>(w_conv), static_cast<T*>(o), dm.T, dm.H,
        dm.dk, dm.Cp, dm.K, d->metric != CONVNN_EUCLIDEAN, d->softmax);
    CONVNN_CHECK_LAUNCH("gather_conv_dw_scalar");
    return CONVNN_OK;
}

// Depthwise conv into rows of d_k values: short bfloat16 sequences with the value rows streamed through shared memory,
// everything else with 16-byte rows flat over the tokens.
int try_launch_dw(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                  const void* w_conv, void* o, cudaStream_t st) {
    const int rc = try_launch_gather_conv_dw_stream(d, dm, v, idx, val, w_conv, o, st);
    return rc != CONVNN_E_UNSUPPORTED ? rc : try_launch_gather_conv_dw(d, dm, v, idx, val, w_conv, o, false, st);
}

template <typename T>
int launch_mat(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
               const void* w_conv, const void* w_pw, void* o, cudaStream_t st) {
    constexpr int ITEMS = 4;
    const int separable = d->conv_type == CONVNN_DEPTHWISE_SEPARABLE;
    // token tile: dk * ceil(TT/4) work items must fit ITEMS passes of the CTA
    int TT = (THREADS * ITEMS / dm.dk) * 4;
    if (TT > 32) TT = 32;
    if (TT < 4) return set_error(CONVNN_E_UNSUPPORTED, "d_k=%d too large for the matrix conv kernel", dm.dk);
    const int ntaps = separable ? 1 : dm.K;
    const size_t budget = 64 * 1024;
    int JC = (int)(budget / ((size_t)TT * dm.C * sizeof(float)));
    if (JC < 1) JC = 1;
    if (JC > ntaps) JC = ntaps;
    size_t smem = (size_t)TT * JC * dm.C * sizeof(float);
    if (smem > 200 * 1024) return set_error(CONVNN_E_UNSUPPORTED, "conv tile needs %zu bytes of shared memory", smem);
    auto kern = gather_conv_mat_kernel<T, ITEMS>;
    CONVNN_ENSURE_SMEM(kern, smem);
    dim3 grid((dm.T + TT - 1) / TT, dm.B * dm.H);
    launch_chained(kern, grid, THREADS, smem, st, static_cast<const T*>(v), idx, val, static_cast<const T*>(w_conv),
                                      static_cast<const T*>(w_pw), static_cast<T*>(o), dm.T, dm.H, dm.dk, dm.C,
                                      dm.Cp, dm.K, d->metric != CONVNN_EUCLIDEAN, d->softmax, separable, TT, JC);
    CONVNN_CHECK_LAUNCH("gather_conv_mat");
    return CONVNN_OK;
}

}  // namespace

// bfloat16 standard / depthwise-separable conv on the tensor cores: a gather kernel builds the
// GEMM's A operand in `scratch`, the tap / pointwise weights are its (N, K) operand.
// Returns CONVNN_E_UNSUPPORTED (last_error untouched) when the shape does not qualify.
int try_launch_gather_conv_tc(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx,
                              const float* val, const void* w_conv, const void* w_pw, void* o, void* scratch,
                              cudaStream_t st) {
    if (d->dtype != CONVNN_BF16 || d->coord || !scratch || force_simt() || dm.C % 8 != 0 || !aligned16(v) ||
        !aligned16(scratch))
        return CONVNN_E_UNSUPPORTED;
    const int M = dm.B * dm.H * dm.T;
    void* cs[1] = {o};
    int rc;
    if (d->conv_type == CONVNN_STANDARD) {
        if ((rc = try_launch_conv_std_tc(d, dm, v, idx, val, w_conv, o, false, st)) != CONVNN_E_UNSUPPORTED) return rc;
        const int Kd = dm.K * dm.C;
        if (!gemm_tc_supported(scratch, Kd, w_conv, Kd, dm.dk, 1, cs, dm.dk)) return CONVNN_E_UNSUPPORTED;
        if ((rc = launch_gather_weighted(d, dm, v, idx, val, scratch, st))) return rc;
        return launch_gemm_tc(scratch, Kd, w_conv, M, dm.dk, Kd, 1, cs, dm.dk, GemmTcOpts(), st);
    }
    if (d->conv_type == CONVNN_DEPTHWISE_SEPARABLE) {
        if (!gemm_tc_supported(scratch, dm.C, w_pw, dm.C, dm.dk, 1, cs, dm.dk)) return CONVNN_E_UNSUPPORTED;
        // stage 0: the depthwise kernels with the (K, C) taps, result (B, H, T, C) rounded to bf16
        if ((rc = try_launch_dw(d, dm, v, idx, val, w_conv, scratch, st))) return rc;
        return launch_gemm_tc(scratch, dm.C, w_pw, M, dm.dk, dm.C, 1, cs, dm.dk, GemmTcOpts(), st);
    }
    return CONVNN_E_UNSUPPORTED;
}

int launch_gather_conv_simt(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx,
                            const float* val, const void* w_conv, const void* w_pw, void* o, void* scratch,
                            cudaStream_t st) {
    const bool f32 = d->dtype == CONVNN_F32;
    if (d->conv_type != CONVNN_DEPTHWISE) {
        const int rc = try_launch_gather_conv_tc(d, dm, v, idx, val, w_conv, w_pw, o, scratch, st);
        if (rc != CONVNN_E_UNSUPPORTED) return rc;
    }
    if (d->conv_type == CONVNN_DEPTHWISE) {
        const int rc = try_launch_dw(d, dm, v, idx, val, w_conv, o, st);
        if (rc != CONVNN_E_UNSUPPORTED) return rc;
        return f32 ? launch_dw_scalar<float>(d, dm, v, idx, val, w_conv, o, st)
                   : launch_dw_scalar<__nv_bfloat16>(d, dm, v, idx, val, w_conv, o, st);
    }
    if (dm.Cp % 4 == 0 && aligned16(v)) {
        GemmParams p{};
        p.w = w_conv; p.c = o; p.ldc = dm.dk; p.M = dm.B * dm.H * dm.T; p.N = dm.dk; p.c_mode = C_ROWS;
        p.T = dm.T; p.H = dm.H; p.dk = dm.dk; p.Cp = dm.Cp; p.C = dm.C;
        if (d->conv_type == CONVNN_STANDARD) {
            // implicit GEMM over the weighted neighbour block, gathered tile by tile as the A operand
            p.a = v; p.a_mode = A_NEIGHBOURS; p.Kd = dm.K * dm.Cp; p.ldw = (long long)dm.K * dm.C;
            p.nb_idx = idx; p.nb_val = val; p.taps = dm.K; p.nb_maximum = d->metric != CONVNN_EUCLIDEAN; p.nb_softmax = d->softmax;
            return launch_gemm_simt(d->dtype, p, st);
        }
        if (scratch && aligned16(scratch) && (f32 || d->coord)) {
            // depthwise stage into scratch (float32, padded to the stored channels where there are more), then the
            // pointwise matrix
            const int rc = try_launch_gather_conv_dw(d, dm, v, idx, val, w_conv, scratch, true, st);
            if (rc != CONVNN_E_UNSUPPORTED) {
                if (rc) return rc;
                p.a = scratch; p.lda = dm.Cp; p.a_mode = A_ROWS; p.a_f32 = 1; p.chained = 1; p.Kd = dm.C; p.w = w_pw; p.ldw = dm.C;
                return launch_gemm_simt(d->dtype, p, st);
            }
        }
    }
    return f32 ? launch_mat<float>(d, dm, v, idx, val, w_conv, w_pw, o, st)
               : launch_mat<__nv_bfloat16>(d, dm, v, idx, val, w_conv, w_pw, o, st);
}

}  // namespace convnn
