// Per-(row, head) post-pass over a projected q / k / v tensor (B, rows, H, Cp):
// writes the optional coordinate channel (reference layers.py:439-450) and the padding
// channels, and reduces the statistic the similarity needs from the STORED values
// (so that a bfloat16 tensor's norm is the norm of the rounded vector):
//   cosine    -> 1 / max(||t||, 1e-12)   (F.normalize's eps, layers.py:337-338)
//   euclidean -> ||t||^2                  (layers.py:328-329)
#include "common.cuh"

namespace convnn {
namespace {

// torch.linspace(-1, 1, steps)[i] in float32: stepped from the start below the middle
// and back from the end above it.
__device__ __forceinline__ float linspace_pm1(int i, int steps) {
    if (steps <= 1) return -1.0f;
    float step = 2.0f / (float)(steps - 1);
    return (i < steps / 2) ? (-1.0f + step * (float)i) : (1.0f - step * (float)(steps - 1 - i));
}

// Up to three tensors of one layer in a launch, one per grid row: bound by the latency of a row's loads and shuffles, so six CTAs per SM
// (40 registers), and nothing in local memory: the tensor is picked by comparisons, since an index that is no constant would put the
// struct on the stack.  Projections with statistics, us, a launch per tensor -> one: 1 x 197 x 2 heads of 16 7.3 -> 5.5, 32 x 65 x 192
// float32 26.1 -> 23.9, 128 x 197 x 3 heads of 64 float32 174.6 -> 168.2 (with the stack: 4 CTAs, 176.2; 100 x 197 x 2 heads of 16 31.1 for 26.1).
struct HeadTensors {
    void* t[3];
    float* stat[3];
    int rows[3];
};

template <typename T>
__global__ void __launch_bounds__(256, 6) head_stats_kernel(const HeadTensors in, int B, int H, int dk, int C, int Cp, int coord, int metric) {
    chain_wait();
    if (sizeof(T) != 4 && !coord) chain_next();      // (with the coordinate channel the fp32 pipes' selection follows, see chain_begin_for())
    const int which = blockIdx.y;
    T* t = static_cast<T*>(which == 0 ? in.t[0] : which == 1 ? in.t[1] : in.t[2]);
    float* stat = which == 0 ? in.stat[0] : which == 1 ? in.stat[1] : in.stat[2];
    const int rows = which == 0 ? in.rows[0] : which == 1 ? in.rows[1] : in.rows[2];
    const int warps_per_block = blockDim.x >> 5;
    const long long total = (long long)B * rows * H;
    const int lane = threadIdx.x & 31;
    for (long long w = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5); w < total;
         w += (long long)gridDim.x * warps_per_block) {
        int h = (int)(w % H);
        long long br = w / H;
        int r = (int)(br % rows);
        int b = (int)(br / rows);
        T* p = t + (br * H + h) * Cp;
        if (coord) {
            for (int c = dk + lane; c < Cp; c += 32)
                p[c] = from_f32<T>(c == dk ? linspace_pm1(r, rows) : 0.0f);
            __syncwarp();
        }
        if (stat) {
            float ss = 0.f;
            constexpr int VEC = 16 / sizeof(T);
            if (C % VEC == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
                for (int c = lane * VEC; c < C; c += 32 * VEC) {     // 16-byte loads
                    const uint4 raw = *reinterpret_cast<const uint4*>(p + c);
                    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
                    for (int j = 0; j < VEC; ++j) {
                        const float v = to_f32<T>(e[j]);
                        ss = fmaf(v, v, ss);
                    }
                }
            } else {
                for (int c = lane; c < C; c += 32) {
                    float v = to_f32<T>(p[c]);
                    ss = fmaf(v, v, ss);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) {
                float s = (metric == CONVNN_COSINE) ? 1.0f / fmaxf(sqrtf(ss), 1e-12f) : ss;
                stat[((long long)b * H + h) * rows + r] = s;
            }
        }
    }
}

}  // namespace

int launch_head_fill_and_stats(const convnn_desc* d, const Dims& dm, void* q, float* qstat, void* k, float* kstat, void* v,
                               cudaStream_t st) {
    HeadTensors in{};
    int n = 0, most = 0;
    auto add = [&](void* t, int rows, float* stat) {
        if (!t || (!d->coord && !stat)) return;
        in.t[n] = t; in.stat[n] = stat; in.rows[n++] = rows;
        if (rows > most) most = rows;
    };
    add(q, dm.S, qstat);
    add(k, dm.T, kstat);
    add(v, dm.T, nullptr);
    if (n == 0) return CONVNN_OK;
    const long long total = (long long)dm.B * most * dm.H;
    int blocks = (int)((total + 7) / 8 < 148 * 16 ? (total + 7) / 8 : 148 * 16);
    if (blocks < 1) blocks = 1;
    if (d->dtype == CONVNN_F32)
        launch_chained(head_stats_kernel<float>, dim3(blocks, n), 256, 0, st, in, dm.B, dm.H, dm.dk, dm.C, dm.Cp, d->coord, d->metric);
    else
        launch_chained(head_stats_kernel<__nv_bfloat16>, dim3(blocks, n), 256, 0, st, in, dm.B, dm.H, dm.dk, dm.C, dm.Cp, d->coord,
                       d->metric);
    CONVNN_CHECK_LAUNCH("head_stats");
    return CONVNN_OK;
}

}  // namespace convnn
