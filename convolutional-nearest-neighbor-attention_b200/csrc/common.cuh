// Shared host/device helpers of the convnn_b200 library.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>

#include "../../include/convnn_b200.h"

namespace convnn {

// ---- error reporting -------------------------------------------------------------
int set_error(int status, const char* fmt, ...);
void clear_error();

void count_launch();

#define CONVNN_CHECK_LAUNCH(what)                                                    \
    do {                                                                             \
        ::convnn::count_launch();                                                    \
        cudaError_t e__ = cudaGetLastError();                                        \
        if (e__ != cudaSuccess)                                                      \
            return ::convnn::set_error(CONVNN_E_CUDA, "%s: %s", what, cudaGetErrorString(e__)); \
    } while (0)

// Kernels of a chain: each is launched while its predecessor on the stream still runs (programmatic stream
// serialization), so that its launch, barrier set-up and TMEM allocation overlap the predecessor's tail.  The rule that
// makes this safe: EVERY thread of a kernel launched with launch_chained() calls chain_wait() before its first access to
// global memory, read or write, and chain_next() comes after that.  The wait ends when the predecessor has completed and its
// writes are visible; the predecessor has waited likewise, so completion is transitive along the stream and nothing older than the
// predecessor can still run when a kernel starts.  In kernels that allocate TMEM chain_next() also comes after the allocation (a
// successor's CTA may take only what is left, and gives it back).
// Two exceptions, both only inside one call of this library:
//   * Beside: a kernel that does not need its predecessor's results lets the next one start and does its work without waiting, and
//     waits for the predecessor at its own end (chain_leave()), so that whoever waits for it has waited for both.  When the next
//     kernel starts, two may still run: this one and its predecessor, which therefore has to be one that waited at its own start.
//     So never two of them in a row: OtherHalf::stage() with `beside` follows a launch of the layer's own each time
//     (layer_forward(), select_and_conv()), and a launcher that has no such form ignores the flag and waits.  What it reads was
//     complete before that predecessor started, what it writes is apart from what that one reads or writes.
//   * Weights at rest may be read before chain_wait() where none of the kernels that may still run writes them: the call's own earlier
//     launches, the predecessor and, behind a kernel beside it, that one's.  The call's first kernel has waited for all that came
//     before it on the stream, a kernel of the caller's that wrote the weights included, and never does this itself.
// A ViT-Tiny forward is 64 kernels (52 up to 21 images) with gaps of ~1.9 us and prologues of ~2 us.  One image 827 -> 712 us, 37 images
// 923 -> 808 us, 256 images 1757 -> 1673 us, BranchConv 64 images 1788 -> 1500 us, ViT-Small 256 images 4588 -> 4441 us.
// The GEMM and MLP kernels' roles each wait for themselves, after their set-up (in the MLP block of one image 4.7 us passed
// between the wait and the first product, 0.9 of them barriers, 1.7 the first instructions and copies of the roles, 1.9 moments
// read a row at a time), and load weights at rest meanwhile: one image 483 -> 436 us, 37 images 655 -> 609 us, 256 1659 -> 1587 us.
__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void chain_next() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void chain_begin() {
    chain_wait();
    chain_next();
}
// float32 kernels (and what runs between them) never let their successor start early: it starts as their last CTAs leave.  Their
// chains end in grids of many small CTAs, which would pile up on the SMs that are free first and wait there (ViT-Tiny
// float32 1970 -> 2430 us), while a plain launch costs the gap.
template <typename T>
__device__ __forceinline__ void chain_begin_for() {
    chain_wait();
    if (sizeof(T) != 4) chain_next();
}
// A kernel launched beside its predecessor, see above.
__device__ __forceinline__ void chain_wait_unless(bool beside) {
    if (!beside) chain_wait();
}
__device__ __forceinline__ void chain_leave(bool beside) {
    if (beside && threadIdx.x == 0) chain_wait();
}
// Under capture the launch is a plain one: a graph's own launches are cheap, its kernels overlap across branches already
// (two batches in flight, 128 launches: 2844 us with chained edges, 2831 us without), and instantiating chained edges
// took the host 0.3 s.
static inline bool starts_early(cudaStream_t st) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &capture);
    return capture == cudaStreamCaptureStatusNone;
}
static inline cudaLaunchAttribute chained_attribute(cudaStream_t st) {
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = starts_early(st);
    return a;
}
template <class... P, class... A>
void launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1] = {chained_attribute(st)};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);   // an error stays the thread's last error (CONVNN_CHECK_LAUNCH)
}

// `chained`: the predecessor does not let this kernel start early (float32, and where the caller launched such a one); else, many
// small CTAs that they are, these kernels are launched plainly.
template <class... P, class... A>
void launch_late(bool chained, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    if (chained) launch_chained(kern, grid, block, smem, st, args...);
    else kern<<<grid, block, smem, st>>>(static_cast<P>(args)...);
}

// SM count of the current device, asked once per device.
int device_sms();
// Its share of them where several forwards are in flight (convnn_b200_forwards_in_flight(), the calling thread's).
int sms_of_a_forward();

// Raises a kernel's dynamic shared-memory limit.  cudaFuncSetAttribute costs a launch about as much host time as
// building a tensor map, so a call site keeps one of these per kernel and calls the runtime only when the size grows.
struct SmemLimit {
    std::atomic<int> bytes[16];
    int ensure(const void* kern, size_t smem);
};
#define CONVNN_ENSURE_SMEM(kern, smem)                                                        \
    do {                                                                                      \
        static ::convnn::SmemLimit limit__{};                                                 \
        const int rc__ = limit__.ensure(reinterpret_cast<const void*>(kern), smem);           \
        if (rc__ != CONVNN_OK) return rc__;                                                   \
    } while (0)

// Clusters of a launch configuration that fit on the device at once, remembered per shared-memory size.
struct ClusterLimit {
    std::atomic<long long> seen[4];          // (shared-memory bytes << 20) | clusters; 0 = free
    int query(const void* kern, const cudaLaunchConfig_t* cfg, int* clusters);
};

// ---- descriptor-derived quantities -------------------------------------------------
struct Dims {
    int B, T, S, D, H, K, dk, C, Cp;   // C = input channels per head, Cp = stored channels
    int nsel;                          // neighbours picked from the candidates: K or K-1
    size_t elt;                        // bytes per element of dtype
};

// Validates the descriptor the way the reference would fail (or this build refuses)
// and fills Dims.  Returns CONVNN_OK or a negative status with last_error set.
int validate(const convnn_desc* d, Dims* out);

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

constexpr int kMaxK = 32;              // register-resident sorted list per row

// ---- dtype helpers -----------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// ---- kernel launchers (one translation unit each) ------------------------------------
// A operand addressing of the SIMT GEMM.
enum AMode : int {
    A_ROWS = 0,       // A[m, kk] = a[m * lda + kk]
    A_TOKENS = 1,     // m = (b, r): token = cand ? cand[r] : r; a[(b*T + token) * lda + kk]
    A_HEAD_QUIRK = 2, // m = (b, t'), kk = h*dk + c': a[((b*H + h) * T) * dk + c' * T + t']
    A_NEIGHBOURS = 3, // m = (b, h, t), kk = j*Cp + c: weight[m, j] * a[(b, neighbour[m, j], h, c)], a (B, T, H, Cp); Cp % 4 == 0
    A_CONV1D = 4      // m = (b, h, t), kk = j*Cp + c: a[(b, t + j - pad, h, c)], zero outside the sequence; Cp % 4 == 0
};
// C placement of the SIMT GEMM.
enum CMode : int {
    C_ROWS = 0,       // c[m * ldc + n]
    C_HEADS = 1       // n = h*dk + c: c[m * H*Cp + h*Cp + c]
};

struct GemmParams {
    const void* a;
    const void* w;        // (N, Kd) row-major: C = A * W^T
    const void* bias;     // (N) in dtype or nullptr
    void* c;
    const int32_t* cand;  // A_TOKENS only
    long long lda, ldc;
    int M, N, Kd;
    int a_mode, c_mode;
    int rows_per_batch;   // A_TOKENS: rows per batch item (T or S); A_HEAD_QUIRK: T
    int T, H, dk, Cp;     // geometry for A_TOKENS / A_HEAD_QUIRK / C_HEADS
    int gelu;             // apply exact GELU after bias
    const void* residual; // (M, N) with row stride ldr, added after rounding to dtype; or nullptr
    long long ldr;
    // the N columns may be split into up to three outputs of part_cols columns each (0: one output)
    void *c1, *c2;
    int part_cols;
    long long ldw;        // row stride of w (0: Kd)
    int bias_first;       // the sum starts from the bias instead of adding it at the end
    int a_f32;            // bfloat16 weights and output, float32 A operand (A_ROWS)
    // A_NEIGHBOURS: lists (M, taps) and how their values become weights; w rows hold taps x C values
    const int32_t* nb_idx;
    const float* nb_val;
    int taps, C, nb_maximum, nb_softmax;
    int pad;              // A_CONV1D
    int chained;          // the launch before this one is the caller's and does not let this one start early
    bool a_vec, w_vec, c_vec;   // set by the launcher
};

int launch_gemm_simt(int dtype, const GemmParams& p, cudaStream_t st);

// Coordinate and padding channels and / or the similarity's statistic of stored q, k, v (nullptr: not this tensor / no
// statistic), in one launch.
int launch_head_fill_and_stats(const convnn_desc* d, const Dims& dm, void* q, float* qstat, void* k, float* kstat, void* v,
                               cudaStream_t st);
int launch_sim_topk_simt_f32(const convnn_desc* d, const Dims& dm, const void* q, const void* k,
                             const float* qstat, const float* kstat, const int32_t* cand,
                             int32_t* idx, float* val, cudaStream_t st);
int launch_sim_topk_simt_bf16(const convnn_desc* d, const Dims& dm, const void* q, const void* k,
                              const float* qstat, const float* kstat, const int32_t* cand,
                              int32_t* idx, float* val, cudaStream_t st);
bool sim_topk_tc_supported(const convnn_desc* d, const Dims& dm, const void* q, const void* k);
int launch_sim_topk_tc(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                       const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st);
bool sim_topk_tc2_wanted(const convnn_desc* d, const Dims& dm);
int launch_sim_topk_tc2(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                        const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st);
// Candidate lists that fit one accumulator (S <= 256): bfloat16 operands, same rules as launch_sim_topk_tc.
bool sim_topk_rows_wanted(const Dims& dm);
int launch_sim_topk_rows(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                         const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st);
bool sim_topk_short_wanted(const Dims& dm);
int launch_sim_topk_short(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const float* qstat,
                          const float* kstat, const int32_t* cand, int32_t* idx, float* val, cudaStream_t st);
int read_sim_short_status(int* out);
// The same kernel with the depthwise conv over the neighbours in it (o (B, H, T, d_k), no lists); CONVNN_E_UNSUPPORTED
// (last_error untouched) where it does not take the shape.
int try_launch_sim_gather(const convnn_desc* d, const Dims& dm, const void* q, const void* k, const void* v, const float* qstat,
                          const float* kstat, const int32_t* cand, const void* w_conv, void* o, cudaStream_t st);
int read_sim_rows_status(int* out);
int read_sim_topk_status(int* out);
int read_sim_topk2_status(int* out);
int try_launch_gather_conv_dw_stream(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx,
                                     const float* val, const void* w_conv, void* o, cudaStream_t st);
int try_launch_gather_conv_dw(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                              const void* w_conv, void* o, bool out_f32, cudaStream_t st);
int launch_gather_weighted(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val, void* P,
                           cudaStream_t st);
int read_dw_stream_status(int* out);
int read_gemm_tc_status(int* out);
// bfloat16 tensor-core GEMM C = A W^T (+bias, +GELU); `parts` outputs share M and split N evenly.
bool gemm_tc_supported(const void* a, long long lda, const void* w, int Kd, int N, int parts, const void* const* c,
                       long long ldc);
struct GemmTcOpts {
    const void* bias = nullptr;       // (N) bf16
    const void* residual = nullptr;   // (M, N) bf16 with row stride ldr, added after rounding
    long long ldr = 0;
    int gelu = 0;
    float* stat[3] = {nullptr, nullptr, nullptr};   // per part: fused per-(row, head) statistic
    int stat_mode = 0, dk = 0, heads = 1, rows_per_batch = 1;
    // heads wider than a tile: room for gemm_tc_stat_pieces() x M x heads floats per part with a
    // statistic (the tiles' partial sums, combined by a second small kernel)
    float* stat_scratch = nullptr;
    // Pre-norm fold: `a` holds the rows BEFORE their LayerNorm, `w` is W * diag(gamma) and ln_wextra
    // the (N, 16) extra rows of fold_layernorm(); ln_moments = [ln_planes][gemm_tc_moment_stride(M)][2]
    // partial (sum, sum of squares) of the rows of a.  No bias / skip connection (the bias is folded).
    const float* ln_moments = nullptr;
    int ln_planes = 0;
    float ln_eps = 0.f;
    const void* ln_wextra = nullptr;
    // What may still run on the stream is this library's own, launched by the same call, and does not write W, its extra
    // rows or the bias: they may be read before the predecessor has ended (see chain_wait()).
    bool w_at_rest = false;
    bool beside = false;              // see chain_leave(); where the epilogue has no such form, the kernel waits at its start
    // Row moments of the stored rows, [gemm_tc_moment_planes(N)][gemm_tc_moment_stride(M)][2]; needs a skip connection.
    float* moments_out = nullptr;
};
bool gemm_tc_prenorm_supported(int N, int Kd, int parts, bool has_stat, bool gelu);
int gemm_tc_moment_planes(int N);
long long gemm_tc_moment_stride(long long M);   // entries between the planes of a moments buffer
bool gemm_tc_can_fuse_stats(int part_cols, int dk);
// Column tiles a head is spread over when the statistic is fused: 1 = a tile holds whole heads,
// m >= 2 = each head spans m tiles (partial sums + combine), 0 = cannot be fused.
int gemm_tc_stat_pieces(int part_cols, int dk);
int launch_gemm_tc(const void* a, long long lda, const void* w, int M, int N, int Kd, int parts, void* const* c,
                   long long ldc, const GemmTcOpts& o, cudaStream_t st);
int launch_layernorm(int dtype, const void* x, long long ldx, const void* gamma, const void* beta, float eps, void* y,
                     long long ldy, long long rows, int D, const void* pe, const void* cls, int Np,
                     long long cls_rows, float* moments, cudaStream_t st);
// The encoder's MLP block (norm2 folded, GELU, both Linear layers, skip connection) as one kernel.
bool mlp_tc_supported(int D, int DM, int planes);
int mlp_tc_moment_planes();
int launch_mlp_tc(const void* x, long long ldx, const float* moments, int planes, float eps, const void* w1_folded,
                  const void* w1_extra, const void* w2, const void* b2, void* out, long long ldo, int M, int D, int DM,
                  float* moments_out, const void* w_o, const void* resid, long long ldr, bool weights_at_rest, cudaStream_t st);
int read_mlp_tc_status(int* out);
// Stages (0, 1, 2) of the other half of a branching block, for layer_forward() to launch beside its own.
struct OtherHalf {
    bool conv1d;                                   // else softmax attention
    const void *x, *w_in, *b_in, *w_conv, *b_conv, *w_out, *b_out;
    void *out, *workspace;
    int64_t ldx, ldo;
    int32_t B, T, D, H, kernel_size;
    int dtype;
    int stage(int i, bool beside, bool at_rest, void* stream) const;
};
// The entry points of these names; at_rest: as GemmTcOpts::w_at_rest, for the call's first weights.
int prenorm_mlp(const void* x, int64_t ldx, const float* moments, int32_t planes, float eps, const void* w1_folded,
                const void* w1_extra, const void* w2, const void* b2, void* out, int64_t ldo, int64_t M, int32_t D, int32_t DM,
                float* moments_out, bool at_rest, void* stream);
int prenorm_forward(const convnn_desc* d, const void* x, int64_t ldx, const float* moments, int32_t planes, float eps,
                    const void* w_qkv_folded, const void* w_qkv_extra, const void* w_conv, const void* w_pw, const void* w_o,
                    const void* residual, int64_t ldr, void* out, int64_t ldo, float* moments_out, void* workspace,
                    size_t workspace_bytes, bool at_rest, void* stream);
int layer_forward(const convnn_desc* d, const void* x, int64_t ldx, const void* w_qkv, const void* w_conv, const void* w_pw,
                  const void* w_o, const int32_t* cand, const void* residual, int64_t ldr, void* out, int64_t ldo, void*
                  workspace, size_t workspace_bytes, bool at_rest, void* stream, const OtherHalf* other = nullptr);
int linear(int dtype, const void* a, int64_t lda, const void* w, const void* bias, const void* residual, int64_t ldr, void*
           out, int64_t ldo, int64_t M, int32_t N, int32_t K, int32_t gelu, bool at_rest, void* stream, bool beside = false);
int prenorm_linear(const void* a, int64_t lda, const float* moments, int32_t planes, float eps, const void* w_folded, const
                   void* w_extra, void* out, int64_t ldo, int64_t M, int32_t N, int32_t K, int32_t gelu, bool at_rest, void*
                   stream);
int linear_moments(const void* a, int64_t lda, const void* w, const void* bias, const void* residual, int64_t ldr, void* out,
                   int64_t ldo, int64_t M, int32_t N, int32_t K, float* moments_out, bool at_rest, void* stream);
int softmax_attention(int dtype, const void* x, int64_t ldx, const void* w_qkv, const void* w_o, void* out, int64_t ldo,
                      int32_t B, int32_t T, int32_t D, int32_t H, void* workspace, size_t workspace_bytes, bool at_rest, void*
                      stream);
int conv1d_attention(int dtype, const void* x, int64_t ldx, const void* w_x, const void* b_x, const void* w_conv, const void*
                     b_conv, const void* w_o, const void* b_o, void* out, int64_t ldo, int32_t B, int32_t T, int32_t D,
                     int32_t H, int32_t kernel_size, void* workspace, size_t workspace_bytes, bool at_rest, void* stream);
int launch_row_moments(const void* x, long long ldx, long long rows, int D, float* moments, cudaStream_t st);
int launch_fold_layernorm(const void* w, const void* bias, const void* gamma, const void* beta, int N, int K,
                          void* w_folded, void* w_extra, cudaStream_t st);
int launch_patchify(int dtype, const void* img, void* out, int B, int C, int Hh, int Ww, int P, cudaStream_t st);
int launch_patchify_u8(int dtype, const uint8_t* img, const float* mean, const float* inv_std, void* out, int B, int C,
                       int Hh, int Ww, int P, cudaStream_t st);
int launch_gather_rows(int dtype, const void* x, long long ldx, const int32_t* cand, void* xq, int B, int Tn, int S,
                       int D, cudaStream_t st);
int launch_merge_heads(int dtype, const void* o, void* y, int B, int Tn, int H, int dk, cudaStream_t st);
int launch_attention(int dtype, const void* q, const void* k, const void* v, void* o, int B, int Tn, int D, int H,
                     cudaStream_t st, bool beside = false);
int read_attention_status(int* out);
int launch_conv1d_heads(int dtype, const void* y, const void* w, const void* bias, void* o, void* unfold, int B,
                        int Tn, int H, int dk, int ks, cudaStream_t st);
// Conv1d half and its flat reinterpretation in one kernel (heads of 16, 32 or 64 channels whose taps fit in shared memory, by a rule
// on the number and length of the slices).
int try_launch_conv1d_tc(const void* y, const void* w, const void* bias, void* out, int B, int Tn, int H, int dk, int ks,
                         cudaStream_t st, bool beside = false);
int read_conv1d_tc_status(int* out);
// Standard conv with its weighted neighbour block kept on the SM (bfloat16 heads of 16, 32 or 64 channels whose taps fit, by a rule on
// tiles per SM and taps); merged: o is (B, T, D) in the flat reinterpretation.
int try_launch_conv_std_tc(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx, const float* val,
                           const void* w_conv, void* o, bool merged, cudaStream_t st);
int read_conv_std_status(int* out);
bool force_simt();   // debugging switch: environment variable CONVNN_B200_FORCE_SIMT=1
int launch_gather_conv_simt(const convnn_desc* d, const Dims& dm, const void* v, const int32_t* idx,
                            const float* val, const void* w_conv, const void* w_pw, void* o, void* scratch,
                            cudaStream_t st);

}  // namespace convnn
