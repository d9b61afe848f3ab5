// The Conv1d half of MultiHeadBranchingConv on the tensor cores: convolution and the flat reinterpretation of its result in one
// kernel (reference layers.py:477-500), for heads of 16, 32 or 64 channels whose taps and one set of boxes fit beside a
// slice (nine taps: 32 channels up to 2074 tokens, 64 channels up to 21) and where conv1d_tc_wanted() finds it the faster way.
//
//   o[b, h, t, oc] = bias[oc] + sum_{j, c} w[oc, j, c] * y[b, t + j - pad, h, c]          (zero outside the sequence)
//   out[b, t', h * dk + c'] = flat(o[b, h])[c' * T + t']
//
// Implicit GEMM: the A operand of tap j is the same 128 x dk box of y, j rows further down (TMA fills what lies outside the
// sequence with zeros), so the taps are never unfolded in memory; the tap weights stay in shared memory for the CTA's life.
// A CTA owns whole (batch, head) slices, so the bfloat16 result is collected in shared memory and leaves transposed, without
// the copy and the second kernel that the reinterpretation cost.  Terms are added in the order of the unfolded GEMM (bias,
// then taps and channels ascending in steps of 16): the same bits.
//
// Bound by latency (a handful of tiles per SM; 0.12 instructions per cycle and scheduler, the warps wait for boxes and for one
// another): 64 images x 197 tokens x 3 heads of 32, 9 taps: 11 us, 24 as unfold (11), GEMM (8.6) and reinterpretation (4.6) in
// kernels of their own.
//
// Warps: 0 TMA (lane j loads tap j), 1 MMA issuer, 2-9 epilogue: two sets of four (lane quarters), one per accumulator.
#include "common.cuh"
#include "sm100.cuh"

namespace convnn {

__device__ int g_conv1d_tc_status = 0;

namespace {

using namespace sm100;

constexpr int BM = 128;
constexpr int NEPI = 256;               // epilogue threads
constexpr int NT = 64 + NEPI;
constexpr size_t SMEM_MAX = 226 * 1024;

struct Conv1dParams {
    const __nv_bfloat16* bias;
    __nv_bfloat16* out;
    int T, H, dk, ks, pad, D;
    int n_units, n_tiles;       // (batch, head) slices, 128-row tiles of one
    int nbuf;                   // tap sets in flight
    uint32_t slab;              // bytes of one collected slice
    int acc_cols;
};

__device__ __forceinline__ void fail(volatile int* abort_flag, int code) {
    *abort_flag = 1;
    atomicCAS(&g_conv1d_tc_status, 0, code);
}
__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(NEPI) : "memory"); }

template <bool BESIDE>                    // see chain_leave()
__global__ void __launch_bounds__(NT, 1)
conv1d_tc_kernel(const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmW, const Conv1dParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t pitch = p.dk * 2, a_bytes = BM * pitch, set_bytes = p.ks * a_bytes, w_tap = p.dk * pitch;
    uint8_t* sW = smem + p.nbuf * set_bytes;                        // [ks][dk x dk]
    uint8_t* ones = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sW + p.ks * w_tap) + 255) & ~(uintptr_t)255);
    uint8_t* btile = ones + 4096;                                   // bias rows, 32 bytes each
    __nv_bfloat16* slab = reinterpret_cast<__nv_bfloat16*>(btile + p.dk * 32);
    uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(slab) + p.slab);
    uint64_t* empty = full + 2;
    uint64_t* tfull = empty + 2;
    uint64_t* tempty = tfull + 2;
    uint64_t* wfull = tempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wfull + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], 1);
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 4);
        }
        mbar_init(wfull, 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmY);
        prefetch_tensormap(&tmW);
    }
    const uint32_t ncols = 2u * p.acc_cols;
    if (warp == 1) {
        tmem_alloc(tmem_slot, ncols);
        tmem_relinquish();
    }
    chain_wait_unless(BESIDE);
    // accumulator := bias by one K = 16 step: rows of `ones` hold 1.0 at the start of both 16-byte halves, a bias row its
    // value at the start of one, so the product picks it up whatever the swizzle
    for (int i = threadIdx.x; i < 1024; i += NT) reinterpret_cast<uint32_t*>(ones)[i] = (i & 3) == 0 ? 0x3f80u : 0u;
    for (int i = threadIdx.x; i < p.dk * 8; i += NT)
        reinterpret_cast<uint32_t*>(btile)[i] =
            (i & 7) == 0 && p.bias ? (uint32_t)__bfloat16_as_ushort(p.bias[i >> 3]) : 0u;
    fence_proxy_async();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_next();

    if (warp == 0) {
        if (lane < p.ks) {
            const uint32_t mask = p.ks == 32 ? 0xffffffffu : (1u << p.ks) - 1u;
            if (lane == 0) mbar_expect_tx_a(smem_u32(wfull), p.ks * w_tap);
            __syncwarp(mask);
            bool first = true, ok = true;
            uint32_t buf = 0, ph = 0;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x) {
                const int b = unit / p.H, h = unit - b * p.H;
                for (int i = 0; i < p.n_tiles; ++i) {
                    ok = mbar_wait(&empty[buf], ph ^ 1u, abort_flag);
                    ok = __all_sync(mask, ok);
                    if (!ok) { if (lane == 0) fail(abort_flag, 101); break; }
                    if (lane == 0) mbar_expect_tx_a(smem_u32(&full[buf]), set_bytes);
                    __syncwarp(mask);
                    tma_load_4d_a(smem_u32(smem) + buf * set_bytes + lane * a_bytes, &tmY, smem_u32(&full[buf]), 0, h,
                                  i * BM + lane - p.pad, b);
                    if (first) tma_load_2d_a(smem_u32(sW) + lane * w_tap, &tmW, smem_u32(wfull), lane * p.dk, 0);
                    first = false;
                    if (++buf == (uint32_t)p.nbuf) { buf = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc = make_idesc_bf16_f32(BM, p.dk);
            const uint64_t dhi = kmajor_desc_hi(pitch), dhi32 = kmajor_desc_hi(32);
            auto desc = [&](uint64_t hi, const void* at) { return hi | (uint64_t)((smem_u32(at) & 0x3FFFFu) >> 4); };
            const uint64_t ones_desc = desc(dhi32, ones), bias_desc = desc(dhi32, btile);
            const int nk16 = p.dk / 16;
            bool ok = mbar_wait_warp(smem_u32(wfull), 0, abort_flag);
            if (!ok) fail(abort_flag, 102);
            uint32_t buf = 0, ph = 0, n = 0;
            for (int unit = blockIdx.x; unit < p.n_units && ok; unit += gridDim.x) {
                for (int i = 0; i < p.n_tiles; ++i, ++n) {
                    const uint32_t a = n & 1u;
                    if (!mbar_wait_warp(smem_u32(&tempty[a]), ((n >> 1) & 1u) ^ 1u, abort_flag) ||
                        !mbar_wait_warp(smem_u32(&full[buf]), ph, abort_flag)) {
                        fail(abort_flag, 103);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t d = tmem_base + a * p.acc_cols;
                    if (elect_one()) {
                        if (p.bias) mma_bf16_ss(d, ones_desc, bias_desc, idesc, 0);
                        for (int j = 0; j < p.ks; ++j)
                            mma_chunk(d, desc(dhi, smem + buf * set_bytes + j * a_bytes), desc(dhi, sW + j * w_tap), idesc, nk16,
                                      j != 0 || p.bias);
                        mma_commit(&empty[buf]);
                        mma_commit(&tfull[a]);
                    }
                    if (++buf == (uint32_t)p.nbuf) { buf = 0; ph ^= 1u; }
                }
            }
        }
    } else {
        // Every epilogue warp makes the same passes and meets both barriers of a unit, also after a wait has expired.
        const int set = (warp - 2) >> 2, lq = warp & 3, tid = threadIdx.x - 64;
        uint32_t n = 0;
        for (int unit = blockIdx.x; unit < p.n_units; unit += gridDim.x) {
            const int b = unit / p.H, h = unit - b * p.H;
            for (int i = 0; i < p.n_tiles; ++i, ++n) {
                if ((int)(n & 1u) != set) continue;
                bool ok = mbar_wait(&tfull[set], (n >> 1) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { if (lane == 0) fail(abort_flag, 104); continue; }
                tc_fence_after_sync();
                const int t = i * BM + lq * 32 + lane;
                for (int c = 0; c < p.dk; c += 16) {
                    uint32_t a[16], w[8];
                    tmem_ld_x16(tmem_base + ((uint32_t)(lq * 32) << 16) + set * p.acc_cols + c, a);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(a[2 * e]), __uint_as_float(a[2 * e + 1]));
                        w[e] = *reinterpret_cast<const uint32_t*>(&v);
                    }
                    if (t < p.T) {
                        uint4* dst = reinterpret_cast<uint4*>(slab + t * p.dk + c);
                        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[set]);
            }
            epilogue_barrier();                      // the slice is complete
            // eight output channels per thread; neighbouring threads share an output row
            const int groups = p.dk / 8;
            __nv_bfloat16* out = p.out + (long long)b * p.T * p.D + h * p.dk;
            for (int e = tid; e < p.T * groups; e += NEPI) {
                const int t = e / groups, g = e - t * groups;
                const __nv_bfloat16* src = slab + g * 8 * p.T + t;
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    w[q] = (uint32_t)__bfloat16_as_ushort(src[2 * q * p.T]) | ((uint32_t)__bfloat16_as_ushort(src[(2 * q + 1) * p.T]) << 16);
                *reinterpret_cast<uint4*>(out + (long long)t * p.D + g * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            epilogue_barrier();                      // and may be overwritten
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
    chain_leave(BESIDE);
}

}  // namespace

// Where this kernel is faster than unfold + GEMM + merge_heads, which spread a long slice over the chip while one CTA walks its
// tiles here (0.4 to 5 us each, by taps and channels), and which waste no tile on sequences of a few tokens.  us for the whole
// branch (two more GEMMs on both sides), others -> this kernel:
//   slices of up to 256 tokens           8 x 197 x 32, 9 taps 18.9 -> 15.7     300 x 256 x 64, 5 taps 59.7 -> 35.7
//   longer, few slices                   1 x 600 x 32, 9 taps 19.3 -> 20.4, 1 x 1000 20.9 -> 30.8, 1 x 4096 x 16 29.4 -> 47.1 (not taken)
//                                        1 x 300 x 32, 9 taps 17.9 -> 16.9     8 x 1000 x 16, 5 taps 21.2 -> 19.1
//   from a fifth / 0.3 of the SMs        32 x 1000 x 64, 3 taps 30.8 -> 35.0, 25 x 600 x 16, 25 taps 28.3 -> 31.9 (not taken)
//                                        32 x 1000 x 32, 9 taps 34.2 -> 33.2     48 x 2000 x 32, 9 taps 70.5 -> 57.9
//   fewer than 32 tokens, many slices    1536 x 9 x 32, 9 taps 23.3 -> 29.1, 300 x 17 x 32, 15 taps 21.1 -> 21.7 (not taken)
static bool conv1d_tc_wanted(int B, int Tn, int H, int dk, int ks) {
    const int sms = device_sms();
    const long long units = (long long)B * H, tiles = (Tn + BM - 1) / BM, n = (units + sms - 1) / sms * tiles;
    if (Tn < 32) return n == 1 || (n <= 5 && n * ks * dk <= 1100);
    if (tiles <= 2 || units * 10 >= sms * 3) return true;
    return tiles * (ks + 4) * dk <= (units * 5 < sms ? 1250 : dk == 64 ? 2400 : 3500);
}

// y (B, T, H, dk) bfloat16, w (dk, ks, dk), bias (dk) or nullptr -> out (B, T, H dk).  CONVNN_E_UNSUPPORTED (last_error
// untouched) where the heads are of another width, the other kernels are faster (above), pointers are unaligned, or a slice
// does not fit beside the taps and one set of boxes (nine taps: 64 channels up to 21 tokens).
int try_launch_conv1d_tc(const void* y, const void* w, const void* bias, void* out, int B, int Tn, int H, int dk, int ks,
                         cudaStream_t st, bool beside) {
    if ((dk != 16 && dk != 32 && dk != 64) || ks > 32 || !conv1d_tc_wanted(B, Tn, H, dk, ks) || !aligned16(y) || !aligned16(w) || !aligned16(out)) return CONVNN_E_UNSUPPORTED;
    Conv1dParams p{};
    p.bias = static_cast<const __nv_bfloat16*>(bias); p.out = static_cast<__nv_bfloat16*>(out);
    p.T = Tn; p.H = H; p.dk = dk; p.ks = ks; p.pad = (ks - 1) / 2; p.D = H * dk;
    p.n_units = B * H; p.n_tiles = (Tn + BM - 1) / BM;
    p.acc_cols = dk < 32 ? 32 : dk;
    const size_t slab = ((size_t)Tn * dk * 2 + 15) / 16 * 16;
    const size_t fixed = 1024 + 256 + (size_t)ks * dk * dk * 2 + 4096 + dk * 32 + slab + 16 * 8;
    const size_t set = (size_t)ks * BM * dk * 2;
    if (fixed + set > SMEM_MAX) return CONVNN_E_UNSUPPORTED;
    p.nbuf = fixed + 2 * set <= SMEM_MAX ? 2 : 1;
    p.slab = (uint32_t)slab;
    CUtensorMap tmY, tmW;
    {
        const uint64_t dims[4] = {(uint64_t)dk, (uint64_t)H, (uint64_t)Tn, (uint64_t)B};
        const uint64_t str[3] = {(uint64_t)dk * 2, (uint64_t)H * dk * 2, (uint64_t)Tn * H * dk * 2};
        const uint32_t box[4] = {(uint32_t)dk, 1, (uint32_t)BM, 1};
        if (!encode_tensor_map_bf16(&tmY, y, 4, dims, str, box, dk * 2)) return CONVNN_E_CUDA;
    }
    {
        const uint64_t dims[2] = {(uint64_t)ks * dk, (uint64_t)dk}, str[1] = {(uint64_t)ks * dk * 2};
        const uint32_t box[2] = {(uint32_t)dk, (uint32_t)dk};
        if (!encode_tensor_map_bf16(&tmW, w, 2, dims, str, box, dk * 2)) return CONVNN_E_CUDA;
    }
    size_t smem = fixed + p.nbuf * set;
    const int grid = p.n_units < device_sms() ? p.n_units : device_sms();
    if (beside) {
        CONVNN_ENSURE_SMEM(conv1d_tc_kernel<true>, smem);
        launch_chained(conv1d_tc_kernel<true>, grid, NT, smem, st, tmY, tmW, p);
    } else {
        CONVNN_ENSURE_SMEM(conv1d_tc_kernel<false>, smem);
        launch_chained(conv1d_tc_kernel<false>, grid, NT, smem, st, tmY, tmW, p);
    }
    CONVNN_CHECK_LAUNCH("conv1d_tc");
    return CONVNN_OK;
}

int read_conv1d_tc_status(int* out) {
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_conv1d_tc_status, sizeof(int));
    if (e != cudaSuccess) return set_error(CONVNN_E_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    *out = v;
    return CONVNN_OK;
}

}  // namespace convnn
