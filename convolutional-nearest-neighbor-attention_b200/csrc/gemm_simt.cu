// FP32-accumulate SIMT GEMM  C = A * W^T (+ bias, + GELU)  with the operand addressing modes the ConvNN path needs:
// token gather for the sampled-query projection, head-split stores for q / k / v (up to three outputs from one packed
// weight), the reference's flat head reinterpretation, and two implicit operands that are never written to memory:
// the weighted neighbour block of the standard conv and the shifted rows of the Conv1d branch.  This is the float32
// path (tensor cores would need a split of every operand to keep the 1e-6 similarity accuracy the top-K parity asks
// for) and the fallback for bfloat16 shapes the tcgen05 kernels do not cover.
//
// Bound by the fp32 pipes and the shared-memory reads that feed them.  Each thread accumulates TM x TN outputs, k strictly
// ascending with one fused multiply-add per term, so a result does not depend on the tile it was computed in.  Two columns
// share one packed multiply-add instruction; operand tiles are transposed into shared memory ([k][row]) so that a warp (4 x 8 threads)
// reads one 64-byte and one 128-byte span per k step without conflicts; the next tile's global loads are in flight
// while the current one is multiplied.
#include "common.cuh"
#include "f32x2.cuh"
#include "token_weights.cuh"

namespace convnn {

namespace {

__device__ __forceinline__ float gelu_exact(float x) {
    return 0.5f * x * (1.0f + erff(x * 0.70710678118654752440f));
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}
// four consecutive values from p (or `n` of them, the rest zero)
template <typename T>
__device__ __forceinline__ float4 load_upto4(const T* p, int n, bool vec) {
    if (vec && n >= 4) return load4(p);
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (i < n) r[i] = to_f32<T>(p[i]);
    return make_float4(r[0], r[1], r[2], r[3]);
}

// One operand row of this thread: where its values for the k range [kk, kk + 4) are.
template <typename TA>
struct ARow {
    const TA* base;       // nullptr: a row past M
    int m_local;          // row inside the tile (A_NEIGHBOURS)
    int t;                // token (A_CONV1D)
};

// Bias, GELU, skip connection and store of a thread's outputs: TM rows row_of(i) by CG groups of VN neighbouring columns, the
// first of group g being n0 + g * step; value(i, g, r) reads a group's sums.
template <typename T, int TM, int CG, int VN, class Row, class Value>
__device__ __forceinline__ void store_outputs(const GemmParams& p, int n0, int step, Row row_of, Value value) {
    const T* bias = static_cast<const T*>(p.bias);
#pragma unroll
    for (int g = 0; g < CG; ++g) {
        const int n = n0 + g * step;
        if (n >= p.N) continue;
        const int nv = min(VN, p.N - n);
        const int part = n / p.part_cols, pn = n - part * p.part_cols;
        T* c = static_cast<T*>(part == 0 ? p.c : (part == 1 ? p.c1 : p.c2));
        int col = pn;
        if (p.c_mode == C_HEADS) {
            const int h = pn / p.dk;
            col = h * p.Cp + (pn - h * p.dk);
        }
        const bool vec = VN == 4 && p.c_vec && nv == 4;         // the four columns are neighbours in one output row
        float bb[VN] = {};
        if (bias && !p.bias_first)
#pragma unroll
            for (int j = 0; j < VN; ++j)
                if (j < nv) bb[j] = to_f32<T>(bias[n + j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = row_of(i);
            if (m >= p.M) continue;
            float r[VN];
            value(i, g, r);
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                if (bias && !p.bias_first) r[j] += bb[j];
                if (p.gelu) r[j] = gelu_exact(r[j]);
            }
            const long long row = p.c_mode == C_HEADS ? (long long)m * p.H * p.Cp : (long long)m * p.ldc;
            if constexpr (VN == 4) {
                if (vec) {
                    if (p.residual) {
                        const float4 q = load4(static_cast<const T*>(p.residual) + (long long)m * p.ldr + n);
                        const float rq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) r[j] = to_f32<T>(from_f32<T>(r[j])) + rq[j];
                    }
                    store4(c + row + col, r);
                    continue;
                }
            }
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                if (j >= nv) continue;
                float v = r[j];
                const int nn = n + j, pp = nn / p.part_cols;
                int cj = nn - pp * p.part_cols;
                T* cc = static_cast<T*>(pp == 0 ? p.c : (pp == 1 ? p.c1 : p.c2));
                if (p.c_mode == C_HEADS) {
                    const int h = cj / p.dk;
                    cj = h * p.Cp + (cj - h * p.dk);
                }
                if (p.residual)
                    v = to_f32<T>(from_f32<T>(v)) + to_f32<T>(static_cast<const T*>(p.residual)[(long long)m * p.ldr + nn]);
                cc[row + cj] = from_f32<T>(v);
            }
        }
    }
}

// Four values of an operand row as they came from memory, made float32 when they are stored to shared memory, a step later.
template <typename T> struct Four;
template <> struct Four<float> {
    float4 v;
    __device__ __forceinline__ void none() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load(const float* p, int n, bool vec) { v = load_upto4(p, n, vec); }
    __device__ __forceinline__ float4 get() const { return v; }
};
template <> struct Four<__nv_bfloat16> {
    uint32_t r[4];             // two pairs, or four values one by one (`vec` tells)
    bool pairs;
    __device__ __forceinline__ void none() {
        pairs = true;
        r[0] = r[1] = 0u;
    }
    __device__ __forceinline__ void load(const __nv_bfloat16* p, int n, bool vec) {
        pairs = vec && n >= 4;
        if (pairs) {
            const uint2 w = *reinterpret_cast<const uint2*>(p);
            r[0] = w.x;
            r[1] = w.y;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = i < n ? reinterpret_cast<const unsigned short*>(p)[i] : 0u;
        }
    }
    __device__ __forceinline__ float4 get() const {
        if (pairs)
            return make_float4(__uint_as_float(r[0] << 16), __uint_as_float(r[0] & 0xffff0000u), __uint_as_float(r[1] << 16),
                               __uint_as_float(r[1] & 0xffff0000u));
        return make_float4(__uint_as_float(r[0] << 16), __uint_as_float(r[1] << 16), __uint_as_float(r[2] << 16),
                           __uint_as_float(r[3] << 16));
    }
};

// Tile BM x BN, NT = (BM / TM) * (BN / TN) threads in warps of 4 (rows) x 8 (columns).
// TA: type of the A operand (float32 against bfloat16 weights for the separable conv's unrounded intermediate).
template <typename TA, typename T, int MODE, int BM, int BN, int BK, int TM, int TN, int MINB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB) gemm_simt_kernel(const GemmParams p) {
    chain_wait();                           // (and no early start for the next one, see chain_begin_for())
    constexpr int NT = (BM / TM) * (BN / TN);
    constexpr int VM = TM < 4 ? TM : 4, VN = TN < 4 ? TN : 4;   // rows / columns read with one instruction
    constexpr int RG = TM / VM, CG = TN / VN;               // groups of them per thread
    constexpr int WN = BN / TN / 8;                         // warps side by side along the columns
    constexpr int LA = BM + 4, LB = BN + 4;
    constexpr int NA = BM * (BK / 4) / NT, NB = BN * (BK / 4) / NT;     // four-value loads per thread and step
    extern __shared__ __align__(16) float gs[];
    float* As = gs;                                         // [2][BK][LA]
    float* Bs = As + 2 * BK * LA;                           // [2][BK][LB]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int ty = (warp / WN) * 4 + (lane >> 3), tx = (warp % WN) * 8 + (lane & 7);

    float* ps = Bs + 2 * BK * LB;                           // A_NEIGHBOURS: weights, row offsets [BM][taps]
    int* ns = reinterpret_cast<int*>(ps + BM * p.taps);
    if constexpr (MODE == A_NEIGHBOURS) {
        const int nm = min(BM, p.M - m0);
        for (int e = tid; e < nm * p.taps; e += NT) ns[e] = p.nb_idx[(long long)m0 * p.taps + e] * (p.H * p.Cp);
        for (int r = tid; r < nm; r += NT)
            token_weights(p.nb_val + (long long)(m0 + r) * p.taps, ps + r * p.taps, p.taps, p.nb_maximum, p.nb_softmax);
        __syncthreads();
    }

    // Staging assignment: a warp takes 16 rows x two groups of four k (one full 32-byte sector per row in float32);
    // the transposed stores of such a set fall into 32 different banks.
    ARow<TA> ar[NA];
    int akq[NA], arow[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        const int c = (tid + i * NT) >> 5;
        akq[i] = (lane & 1) + 2 * (c % (BK / 8));
        arow[i] = (lane >> 1) + 16 * (c / (BK / 8));
        const int m = m0 + arow[i];
        ar[i].base = nullptr;
        if (m < p.M) {
            const TA* a = static_cast<const TA*>(p.a);
            if (MODE == A_ROWS) {
                ar[i].base = a + (long long)m * p.lda;
            } else if (MODE == A_TOKENS) {
                const int b = m / p.rows_per_batch, r = m - b * p.rows_per_batch;
                ar[i].base = a + ((long long)b * p.T + (p.cand ? p.cand[r] : r)) * p.lda;
            } else if (MODE == A_HEAD_QUIRK) {
                // y[b, t', h*dk + c'] = flat(o[b, h])[c' * T + t']   (reference layers.py:247-259)
                const int b = m / p.T;
                ar[i].base = a + (long long)b * p.H * p.T * p.dk + (m - b * p.T);
            } else {
                // m = (b, h, t): rows (b, token, h, :) of a (B, T, H, Cp) tensor
                const int bh = m / p.T, b = bh / p.H, h = bh - b * p.H;
                ar[i].t = m - bh * p.T;
                ar[i].base = a + ((long long)b * p.T * p.H + h) * p.Cp;
            }
            ar[i].m_local = arow[i];
        }
    }
    const T* wbase[NB];
    int bkq[NB], brow[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int c = (tid + i * NT) >> 5;
        bkq[i] = (lane & 1) + 2 * (c % (BK / 8));
        brow[i] = (lane >> 1) + 16 * (c / (BK / 8));
        const int n = n0 + brow[i];
        wbase[i] = n < p.N ? static_cast<const T*>(p.w) + (long long)n * p.ldw : nullptr;
    }
    const bool avec = p.a_vec, wvec = p.w_vec;

    // Operands stay as they came until they are stored to shared memory, a step later: converted or weighted here, a load is waited
    // for before the products it should hide behind (bfloat16, 7 x 577 x 384 with the coordinate channel, k and v 80.5 -> 69.4 us;
    // standard conv, 9 taps, float32 8 x 197 x 192 104 -> 91, 32 x 197 x 384 678 -> 592, 1 x 197 x 3 heads of 64 28.2 -> 23.0; bfloat16 with the
    // coordinate channel 8 x 197 x 192 150 -> 110, 32 x 197 x 384 893 -> 783).
    std::conditional_t<MODE == A_HEAD_QUIRK, Four<float>, Four<TA>> av[NA];
    Four<T> bv[NB];
    float aw[MODE == A_NEIGHBOURS ? NA : 1];                // the neighbours' weights
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int kk = k0 + akq[i] * 4;
            av[i].none();
            if constexpr (MODE == A_NEIGHBOURS) aw[i] = 0.f;
            if (ar[i].base && kk < p.Kd) {
                if constexpr (MODE == A_ROWS || MODE == A_TOKENS) {
                    av[i].load(ar[i].base + kk, p.Kd - kk, avec);
                } else if constexpr (MODE == A_HEAD_QUIRK) {
                    float e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (kk + j < p.Kd) {
                            const int h = (kk + j) / p.dk, c = kk + j - h * p.dk;
                            e[j] = to_f32<TA>(ar[i].base[((long long)h * p.dk + c) * p.T]);
                        }
                    av[i].v = make_float4(e[0], e[1], e[2], e[3]);
                } else if constexpr (MODE == A_NEIGHBOURS) {
                    // k = (tap, stored channel): Cp is a multiple of four, so the four values share a tap
                    const int j = kk / p.Cp, c = kk - j * p.Cp;
                    const int e = ar[i].m_local * p.taps + j;
                    aw[i] = ps[e];
                    av[i].load(ar[i].base + ns[e] + c, 4, avec);
                } else {                                          // A_CONV1D: k = (tap, channel)
                    const int j = kk / p.Cp, c = kk - j * p.Cp, tt = ar[i].t + j - p.pad;
                    if (tt >= 0 && tt < p.T) av[i].load(ar[i].base + (long long)tt * p.H * p.Cp + c, 4, avec);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int kk = k0 + bkq[i] * 4;
            bv[i].none();
            if (wbase[i] && kk < p.Kd) {
                if (MODE == A_NEIGHBOURS && p.C != p.Cp) {        // taps of C values against C + padding stored channels
                    const int j = kk / p.Cp, c = kk - j * p.Cp;
                    bv[i].load(wbase[i] + (long long)j * p.C + c, p.C - c, false);
                } else {
                    bv[i].load(wbase[i] + kk, p.Kd - kk, wvec);
                }
            }
        }
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            float* d = As + (buf * BK + akq[i] * 4) * LA + arow[i];
            float4 v = av[i].get();
            if constexpr (MODE == A_NEIGHBOURS) { v.x *= aw[i]; v.y *= aw[i]; v.z *= aw[i]; v.w *= aw[i]; }
            d[0] = v.x; d[LA] = v.y; d[2 * LA] = v.z; d[3 * LA] = v.w;
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            float* d = Bs + (buf * BK + bkq[i] * 4) * LB + brow[i];
            const float4 v = bv[i].get();
            d[0] = v.x; d[LB] = v.y; d[2 * LB] = v.z; d[3 * LB] = v.w;
        }
    };

    f32x2 acc[TM][TN / 2];
    const T* bias = static_cast<const T*>(p.bias);
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
        f32x2 init = 0ull;
        if (p.bias_first && bias) {
            const int n = n0 + (2 * j / VN) * (BN / CG) + tx * VN + 2 * j % VN;
            init = pack2(n < p.N ? to_f32<T>(bias[n]) : 0.f, n + 1 < p.N ? to_f32<T>(bias[n + 1]) : 0.f);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = init;
    }

    fetch(0);
    stage(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < p.Kd; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < p.Kd;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM];
            f32x2 b[TN / 2];
#pragma unroll
            for (int g = 0; g < RG; ++g) {
                const float* src = As + (buf * BK + k) * LA + g * (BM / RG) + ty * VM;
                if (VM == 4) {
                    const float4 v = *reinterpret_cast<const float4*>(src);
                    a[4 * g] = v.x; a[4 * g + 1] = v.y; a[(4 * g + 2) % TM] = v.z; a[(4 * g + 3) % TM] = v.w;
                } else {
                    const float2 v = *reinterpret_cast<const float2*>(src);
                    a[2 * g] = v.x; a[2 * g + 1] = v.y;
                }
            }
#pragma unroll
            for (int g = 0; g < CG; ++g) {
                const float* src = Bs + (buf * BK + k) * LB + g * (BN / CG) + tx * VN;
                if (VN == 4) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src);
                    b[2 * g] = v.x; b[(2 * g + 1) % (TN / 2)] = v.y;
                } else {
                    b[g] = *reinterpret_cast<const f32x2*>(src);
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const f32x2 aa = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(aa, b[j], acc[i][j]);
            }
        }
        if (more) {
            stage(buf ^ 1);
            __syncthreads();
        }
    }

    store_outputs<T, TM, CG, VN>(
        p, n0 + tx * VN, BN / CG, [&](int i) { return m0 + (i / VM) * (BM / RG) + ty * VM + i % VM; },
        [&](int i, int g, float (&r)[VN]) {
#pragma unroll
            for (int j = 0; j < VN / 2; ++j) unpack2(acc[i][g * (VN / 2) + j], r[2 * j], r[2 * j + 1]);
        });
}

// float32 rows that can be copied 16 bytes at a time: steps of 32 k values land by asynchronous copies, three ahead, in the
// order they have in memory (a row is 128 bytes, its 16-byte pieces exchanged, so that the lanes of a warp read their rows
// without conflicts and nothing is transposed); a thread reads four k values of its rows at once, the next four while
// these are multiplied.  Plain multiply-adds: they run at the rate of the packed ones (70 against 67 TFLOP/s with four
// warps per scheduler) and need no pairs.  Same sums as above, k strictly ascending.  A tile is two warps, so that its
// steps wait for no others and small outputs spread evenly over the SMs; the shared-memory port, TM + TN cycles per
// warp and k value, and the latency of a lone warp per scheduler bound it.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Where a 16-byte piece of a tile row (32 k values; rows of A, then of W) lies, in floats: rows that the lanes of a warp
// read side by side differ in the exchange.
template <int BM, int TM>
__device__ __forceinline__ int place_piece(int row, int piece) {
    const int x = row < BM ? row / TM : (row - BM) / 4;
    return row * 32 + ((piece ^ (x & 7)) << 2);
}
// The products of one step of 32 k values, ascending; the next four values of every row are read while four are multiplied.
// (Eight columns per thread leave no registers for that: 128 x 64 tiles of this kind 110 us where 64 x 64 take 86.)
template <int BM, int TM, int TN>
__device__ __forceinline__ void multiply_step(const float* tile, int ty, int tx, float (&acc)[TM][TN]) {
    static_assert(TN == 4, "four columns per thread");
    const float* pa = tile + ty * TM * 32;
    const float* pb = tile + (BM + tx * 4) * 32;
    float4 a[2][TM], b[2][TN];
    auto read = [&](int q, int u) {
#pragma unroll
        for (int i = 0; i < TM; ++i) a[u][i] = *reinterpret_cast<const float4*>(pa + i * 32 + ((q ^ (ty & 7)) << 2));
#pragma unroll
        for (int j = 0; j < TN; ++j) b[u][j] = *reinterpret_cast<const float4*>(pb + j * 32 + ((q ^ (tx & 7)) << 2));
    };
    read(0, 0);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int u = q & 1;
        if (q + 1 < 8) read(q + 1, u ^ 1);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf((&a[u][i].x)[e], (&b[u][j].x)[e], acc[i][j]);
    }
}

template <int MODE, int BM, int BN, int TM, int TN, int MINB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB) gemm_simt_copy_kernel(const GemmParams p) {
    static_assert(MODE == A_ROWS || MODE == A_TOKENS, "plain rows");
    chain_wait();                           // (and no early start for the next one, see chain_begin_for())
    constexpr int NT = (BM / TM) * (BN / TN), BK = 32, ST = 4, PIECES = BK / 4;
    constexpr int WN = BN / TN / 8;
    constexpr int NL = (BM + BN) * PIECES / NT;                 // copies per thread and step
    static_assert((BM + BN) * PIECES % NT == 0 && NT % 32 == 0 && (BN / TN) % 8 == 0 && TN == 4, "tile");
    extern __shared__ __align__(128) float gs[];               // [ST][BM + BN][BK]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int ty = (warp / WN) * 4 + (lane >> 3), tx = (warp % WN) * 8 + (lane & 7);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(gs);
    const int piece = tid % PIECES;                             // (NT is a multiple of the pieces of a row)
    const float* src[NL];
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        const int row = (tid + i * NT) / PIECES;
        src[i] = nullptr;
        if (row < BM) {
            const int m = m0 + row;
            if (m < p.M) {
                long long r = m;
                if (MODE == A_TOKENS) {
                    const int b = m / p.rows_per_batch, t = m - b * p.rows_per_batch;
                    r = (long long)b * p.T + (p.cand ? p.cand[t] : t);
                }
                src[i] = static_cast<const float*>(p.a) + r * p.lda + piece * 4;
            }
        } else if (n0 + row - BM < p.N) {
            src[i] = static_cast<const float*>(p.w) + (long long)(n0 + row - BM) * p.ldw + piece * 4;
        }
    }
    auto request = [&](int slot, int k0) {
        const int left = (p.Kd - k0 - piece * 4) * 4;           // bytes of this piece inside the row; the rest is zeros
        const int bytes = left >= 16 ? 16 : (left > 0 ? left : 0);
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            const int row = (tid + i * NT) / PIECES;
            const bool on = src[i] && bytes > 0;
            copy16(base + 4u * (uint32_t)(slot * (BM + BN) * BK + place_piece<BM, TM>(row, piece)), on ? src[i] + k0 : p.a, on ? bytes : 0);
        }
    };

    float acc[TM][TN];
    const float* bias = static_cast<const float*>(p.bias);
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const int n = n0 + tx * 4 + j;
        const float init = p.bias_first && bias && n < p.N ? bias[n] : 0.f;
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = init;
    }

    const int steps = (p.Kd + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < steps) request(s, s * BK);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int slot = 0, next = ST - 1;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();                                        // everyone's copies of this step; the slot of the last one is free
        if (step + ST - 1 < steps) request(next, (step + ST - 1) * BK);
        asm volatile("cp.async.commit_group;" ::: "memory");
        multiply_step<BM, TM, TN>(gs + slot * (BM + BN) * BK, ty, tx, acc);
        slot = slot + 1 == ST ? 0 : slot + 1;
        next = next + 1 == ST ? 0 : next + 1;
    }

    store_outputs<float, TM, 1, 4>(
        p, n0 + tx * 4, 0, [&](int i) { return m0 + ty * TM + i; },
        [&](int i, int, float (&r)[4]) {
#pragma unroll
            for (int j = 0; j < 4; ++j) r[j] = acc[i][j];
        });
}

// The same tiles for rows that have to be converted, or that cannot be copied 16 bytes at a time: they come through
// registers, a step ahead.
template <typename TA, typename T, int MODE, int BM, int BN, int TM, int TN, int MINB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB) gemm_simt_stage_kernel(const GemmParams p) {
    static_assert(MODE == A_ROWS || MODE == A_TOKENS, "plain rows");
    chain_wait();                           // (and no early start for the next one, see chain_begin_for())
    constexpr int NT = (BM / TM) * (BN / TN), BK = 32, PIECES = BK / 4, STEP = NT / PIECES;   // rows per pass
    constexpr int WN = BN / TN / 8, NA = BM / STEP, NB = BN / STEP;
    static_assert(BM % STEP == 0 && BN % STEP == 0 && NT % 32 == 0 && (BN / TN) % 8 == 0, "tile");
    extern __shared__ __align__(128) float gs[];                // [2][BM + BN][BK]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int ty = (warp / WN) * 4 + (lane >> 3), tx = (warp % WN) * 8 + (lane & 7);
    const int piece = tid % PIECES, row0 = tid / PIECES;

    const TA* ab[NA];
    const T* wb[NB];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        const int m = m0 + row0 + i * STEP;
        ab[i] = nullptr;
        if (m < p.M) {
            const TA* a = static_cast<const TA*>(p.a);
            if (MODE == A_ROWS) {
                ab[i] = a + (long long)m * p.lda;
            } else {
                const int b = m / p.rows_per_batch, r = m - b * p.rows_per_batch;
                ab[i] = a + ((long long)b * p.T + (p.cand ? p.cand[r] : r)) * p.lda;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int n = n0 + row0 + i * STEP;
        wb[i] = n < p.N ? static_cast<const T*>(p.w) + (long long)n * p.ldw : nullptr;
    }
    const bool avec = p.a_vec, wvec = p.w_vec;

    Four<TA> fa[NA];
    Four<T> fb[NB];
    auto fetch = [&](int step) {
        const int kk = step * BK + piece * 4, left = p.Kd - kk;
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            fa[i].none();
            if (ab[i] && left > 0) fa[i].load(ab[i] + kk, left, avec);
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            fb[i].none();
            if (wb[i] && left > 0) fb[i].load(wb[i] + kk, left, wvec);
        }
    };
    auto stage = [&](int slot) {
        float* t = gs + slot * (BM + BN) * BK;
#pragma unroll
        for (int i = 0; i < NA; ++i)
            *reinterpret_cast<float4*>(t + place_piece<BM, TM>(row0 + i * STEP, piece)) = fa[i].get();
#pragma unroll
        for (int i = 0; i < NB; ++i)
            *reinterpret_cast<float4*>(t + place_piece<BM, TM>(BM + row0 + i * STEP, piece)) = fb[i].get();
    };

    float acc[TM][TN];
    const T* bias = static_cast<const T*>(p.bias);
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const int n = n0 + tx * 4 + j;
        const float init = p.bias_first && bias && n < p.N ? to_f32<T>(bias[n]) : 0.f;
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = init;
    }
    const int steps = (p.Kd + BK - 1) / BK;
    fetch(0);
    stage(0);
    __syncthreads();
    for (int step = 0; step < steps; ++step) {
        const bool more = step + 1 < steps;
        if (more) fetch(step + 1);
        multiply_step<BM, TM, TN>(gs + (step & 1) * (BM + BN) * BK, ty, tx, acc);
        if (more) {
            stage((step + 1) & 1);
            __syncthreads();
        }
    }
    store_outputs<T, TM, 1, 4>(
        p, n0 + tx * 4, 0, [&](int i) { return m0 + ty * TM + i; },
        [&](int i, int, float (&r)[4]) {
#pragma unroll
            for (int j = 0; j < 4; ++j) r[j] = acc[i][j];
        });
}

template <typename TA, typename T, int MODE, int BM, int BN, int BK, int TM, int TN, int MINB>
int launch_tile(const GemmParams& p, cudaStream_t st) {
    const dim3 grid((p.M + BM - 1) / BM, (p.N + BN - 1) / BN);
    const size_t smem = (size_t)2 * BK * (BM + 4 + BN + 4) * 4 + (MODE == A_NEIGHBOURS ? (size_t)BM * p.taps * 8 : 0);
    auto kern = gemm_simt_kernel<TA, T, MODE, BM, BN, BK, TM, TN, MINB>;
    CONVNN_ENSURE_SMEM(kern, smem);
    launch_late(sizeof(T) == 4 || p.chained, kern, grid, (BM / TM) * (BN / TN), smem, st, p);
    return CONVNN_OK;
}

template <typename TA, typename T, int MODE, int BM, int BN, int TM, int TN, int MINB>
int launch_stage_tile(const GemmParams& p, cudaStream_t st) {
    const dim3 grid((p.M + BM - 1) / BM, (p.N + BN - 1) / BN);
    const size_t smem = (size_t)2 * (BM + BN) * 32 * 4;
    auto kern = gemm_simt_stage_kernel<TA, T, MODE, BM, BN, TM, TN, MINB>;
    CONVNN_ENSURE_SMEM(kern, smem);
    launch_late(sizeof(T) == 4 || p.chained, kern, grid, (BM / TM) * (BN / TN), smem, st, p);
    return CONVNN_OK;
}

template <int MODE, int BM, int BN, int TM, int TN, int MINB>
int launch_copy_tile(const GemmParams& p, cudaStream_t st) {
    const dim3 grid((p.M + BM - 1) / BM, (p.N + BN - 1) / BN);
    const size_t smem = (size_t)4 * (BM + BN) * 32 * 4;
    auto kern = gemm_simt_copy_kernel<MODE, BM, BN, TM, TN, MINB>;
    CONVNN_ENSURE_SMEM(kern, smem);
    launch_chained(kern, grid, (BM / TM) * (BN / TN), smem, st, p);
    return CONVNN_OK;
}

// Plain rows: the tile with the shortest time on the busiest SM, which runs `fit` tiles at a time.  `step` is what a value of
// k takes there with 1, 2, ... tiles side by side, ns, in whole steps of `bk` of them.  The numbers are fits to measured times.
struct Tile {
    int bm, bn, bk, fit;
    double launch, round, step[7];        // us per launch and per round of tiles
};
template <int COUNT>
int cheapest_tile(const Tile (&tiles)[COUNT], const GemmParams& p, int first = 0) {
    const long long sms = device_sms();
    int best = -1;
    double least = 0;
    for (int i = first; i < COUNT; ++i) {
        const Tile& t = tiles[i];
        if (t.bn < 64 && (p.N + t.bn - 1) / t.bn > 65535) continue;      // (grid rows)
        const long long n = (long long)((p.M + t.bm - 1) / t.bm) * ((p.N + t.bn - 1) / t.bn), per_sm = (n + sms - 1) / sms;
        const long long full = per_sm / t.fit, rest = per_sm % t.fit;
        const double k = 1e-3 * t.bk * ((p.Kd + t.bk - 1) / t.bk);
        double cost = t.launch + (full + (rest ? 1 : 0)) * t.round + k * full * t.step[t.fit - 1];
        if (rest) cost += k * t.step[rest - 1];
        if (best < 0 || cost < least) { least = cost; best = i; }
    }
    return best;
}

// float32 rows that can be copied.  A tile of two warps leaves two of the four schedulers idle, so tiles come in pairs.
// Over 396 shapes (65 to 25216 rows, 10 to 2304 columns, 64 to 1536 values of k; rms 3 to 7 %) the choice is within 0.6 % of the
// best of twelve tiles on average, 12 % at worst.  With the first two tiles alone (and smaller transposed ones, since
// gone) 2080 rows took 33.0 us at 192 x 768, now 25.8; 20.6 at 576 x 192, now 17.8; 1576 x 384 x 192 15.5, now 11.5; 1050
// x 384 x 384 18.7, now 15.6.
// Few values of k give the copies nothing to run ahead of, and their start costs 0.3 to 0.6 us: the smallest transposed tile then, up to
// 32 values while an SM runs few of them (24853 x 28 x 16 5.5 us with a copy tile, 4.3; 99 x 39 x 4 5.4, 4.8), up to 96 while it runs one
// (500 x 64 x 96 4.8, 4.6; with two to four 2000 x 192 x 96 6.1, 6.4), and up to 64 where columns are stored one by one (28216 x 10 x
// 44 10.3, 8.3; 3196 x 659 x 40 19.6, 17.2; with whole vectors 4100 x 384 x 64 9.9, 12.1).
template <int MODE>
int launch_plain_f32(const GemmParams& p, cudaStream_t st) {
    const int few = p.Kd <= 32 ? 14 : p.Kd <= 64 && !p.c_vec ? 21 : p.Kd <= 96 ? 1 : 0;       // tiles per SM
    if ((long long)((p.M + 31) / 32) * ((p.N + 31) / 32) <= (long long)few * device_sms() && (p.N + 31) / 32 <= 65535)
        return launch_tile<float, float, MODE, 32, 32, 32, 4, 4, 4>(p, st);
    static const Tile tiles[6] = {
        {128, 64, 1, 3, 5.4, 0.5, {65.4, 107.1, 153.3}},
        {64, 64, 1, 3, 3.2, 0.7, {38.2, 62.3, 88.9}},
        {32, 32, 1, 6, 1.7, 1.5, {19.6, 20.9, 33.3, 35.3, 51.4, 48.7}},
        {40, 32, 1, 6, 2.2, 1.6, {23.5, 25.2, 38.8, 39.7, 61.1, 58.2}},
        {48, 32, 1, 5, 2.2, 2.3, {26.3, 28.8, 42.9, 46.8, 60.0}},
        {56, 32, 1, 5, 1.9, 3.1, {30.2, 32.5, 50.4, 53.8, 72.0}},
    };
    switch (cheapest_tile(tiles, p)) {
        case 0: return launch_tile<float, float, MODE, 128, 64, 16, 8, 8, 3>(p, st);
        case 1: return launch_tile<float, float, MODE, 64, 64, 32, 8, 4, 3>(p, st);
        case 2: return launch_copy_tile<MODE, 32, 32, 4, 4, 6>(p, st);
        case 3: return launch_copy_tile<MODE, 40, 32, 5, 4, 6>(p, st);
        case 4: return launch_copy_tile<MODE, 48, 32, 6, 4, 5>(p, st);
        default: return launch_copy_tile<MODE, 56, 32, 7, 4, 5>(p, st);
    }
}

// Other plain rows: float32 ones of any alignment, bfloat16, float32 against bfloat16 weights.  Which tiles, and which times, goes by
// what the operands cost: rows that come one value at a time cost every tile more, the small ones most.  Narrow outputs of few
// values of k (the separable conv with the coordinate channel on heads of 8 to 32) end before that counts.  Fits to 209, 90, 98
// and 90 shapes (30 to 1000000 rows, 8 to 2304 columns, 9 to 2048 values of k; rms 3 to 21 %), the choice within 1.2, 1.0, 0.8
// and 0.9 % of the best of seven tiles on average; 0.95, 0.72, 0.55 and 0.71 of the time of the four transposed tiles alone, at worst
// 1.09 (kernels of 4 us).
// float32, us, staged tiles only -> now: 2813 x 768 x 769 138 -> 102, 56288 x 256 x 257 244 -> 189, 39846 x 8 x 9 9.9 -> 6.7; mixed 650981 x
// 64 x 65 277 -> 233, 109615 x 16 x 17 18.7 -> 12.3.
// bfloat16, transposed tiles only -> now: 4 x 197 x 768 x 768 130 -> 55; 2080 x 384 x 388 57.9 -> 27.8.
// The 128 x 64 tile, once it waits for no conversion, is the best of five on most large outputs of bfloat16 rows read four at a time and of mixed ones (27 shapes; the fits
// hold within 10 %), us: 4925 x 2304 x 768 468 -> 399, 25216 x 192 x 192 64 -> 54, mixed 4925 x 768 x 769 215 -> 176.
// Six 32 x 32 tiles fit an SM with the 136 to 138 registers that rows kept as they came take, eight with 128: bounded where there are more than
// six, 36230 x 96 x 9 14.1 -> 12.4 us, 21446 x 192 x 9 16.1 -> 14.5, 15506 x 64 x 196 22.3 -> 19.8; few lose a little (785 x 192 x 12 3.9 -> 4.1).
template <typename TA, typename T, int MODE>
int launch_plain_staged(const GemmParams& p, cudaStream_t st) {
    if constexpr (sizeof(T) == 4) {
        static const Tile tiles[4] = {
            {128, 64, 16, 3, 0.6, 4.8, {75.5, 117.3, 176.8}},
            {64, 64, 32, 3, 2.9, 1.6, {43.8, 73.6, 105.2}},
            {32, 32, 32, 7, 2.9, 0.0, {31.1, 35.7, 49.8, 65.0, 81.8, 88.6, 95.5}},
            {32, 64, 32, 4, 2.0, 1.4, {30.0, 51.2, 66.6, 86.9}},
        };
        switch (cheapest_tile(tiles, p)) {
            case 0: return launch_tile<TA, T, MODE, 128, 64, 16, 8, 8, 3>(p, st);
            case 1: return launch_tile<TA, T, MODE, 64, 64, 32, 8, 4, 3>(p, st);
            case 2: return launch_tile<TA, T, MODE, 32, 32, 32, 4, 4, 4>(p, st);
            default: return launch_stage_tile<TA, T, MODE, 32, 64, 4, 4, 4>(p, st);
        }
    } else {
        static const Tile by_four[5] = {
            {128, 64, 16, 3, 7.5, 2.0, {65.0, 113.0, 156.0}},
            {32, 32, 32, 7, 1.5, 1.2, {45.0, 51.0, 66.0, 68.0, 72.0, 78.0, 73.0}},
            {64, 64, 32, 3, 2.4, 2.9, {41.0, 62.8, 91.7}},
            {32, 64, 32, 4, 1.5, 1.8, {27.3, 43.1, 59.2, 76.9}},
            {40, 32, 32, 6, 1.8, 2.5, {32.2, 34.5, 46.8, 51.2, 60.2, 70.8}},
        };
        static const Tile by_value[5] = {
            by_four[0],          // (not among the choices: no layer has such rows on both sides.  4039 x 768 x 385 87 us, the third 98)
            {32, 32, 32, 7, 1.1, 0.0, {108.4, 122.0, 111.1, 150.7, 131.6, 174.3, 135.2}},
            {64, 64, 32, 3, 2.6, 3.6, {45.3, 68.7, 102.8}},
            {32, 64, 32, 4, 2.1, 1.7, {31.9, 48.3, 65.4, 92.7}},
            {40, 32, 32, 6, 2.3, 2.9, {36.8, 39.8, 54.5, 58.5, 83.1, 87.1}},
        };
        static const Tile mixed[5] = {                               // float32 rows against bfloat16 weights
            {128, 64, 16, 3, 7.5, 2.0, {64.0, 113.0, 148.0}},
            {32, 32, 32, 7, 0.9, 0.0, {90.3, 100.6, 98.8, 99.2, 114.6, 113.0, 102.3}},
            {64, 64, 32, 3, 2.1, 2.6, {42.7, 67.6, 95.9}},
            {32, 64, 32, 4, 1.9, 1.0, {31.5, 47.1, 66.7, 82.2}},
            {40, 32, 32, 6, 1.8, 2.2, {32.9, 37.0, 45.6, 55.8, 70.9, 74.7}},
        };
        switch (sizeof(TA) == 4 ? cheapest_tile(mixed, p) : p.a_vec && p.w_vec ? cheapest_tile(by_four, p) : cheapest_tile(by_value, p, 1)) {
            case 0: return launch_tile<TA, T, MODE, 128, 64, 16, 8, 8, 3>(p, st);
            case 1:
                if ((long long)((p.M + 31) / 32) * ((p.N + 31) / 32) > 6ll * device_sms())
                    return launch_tile<TA, T, MODE, 32, 32, 32, 4, 4, 8>(p, st);
                return launch_tile<TA, T, MODE, 32, 32, 32, 4, 4, 4>(p, st);
            case 2: return launch_stage_tile<TA, T, MODE, 64, 64, 8, 4, 3>(p, st);
            case 3: return launch_stage_tile<TA, T, MODE, 32, 64, 4, 4, 4>(p, st);
            default: return launch_stage_tile<TA, T, MODE, 40, 32, 5, 4, 6>(p, st);
        }
    }
}

template <typename TA, typename T, int MODE>
int launch_other_mode(const GemmParams& p, cudaStream_t st) {
    // Implicit operands and the flat head reinterpretation: the tile with the least work on the busiest SM, rounds of tiles x
    // outputs per tile over the rate of the tile's threads.  That rate is set by shared memory: a k step reads TM + TN values per
    // thread for TM * TN multiply-adds (45, 40, 29 and 26 TFLOP/s with plain rows at 16384 x 768 x 768).
    const long long sms = device_sms();
    long long tiles_of[4];
    auto cost = [&](int i, int bm, int bn, double rate) {
        tiles_of[i] = (long long)((p.M + bm - 1) / bm) * ((p.N + bn - 1) / bn);
        return (double)((tiles_of[i] + sms - 1) / sms) * bm * bn / rate;
    };
    const double c[4] = {cost(0, 128, 64, 45), cost(1, 64, 64, 40), cost(2, 32, 64, 29), cost(3, 32, 32, 26)};
    int best = 0;
    for (int i = 1; i < 4; ++i)
        if (c[i] < c[best]) best = i;
    // An implicit operand is fetched with divisions and dependent reads per value.  While an SM has few tiles that, not the
    // products, is what a step waits for, and a tile with twice the threads wins; with more of them the tiles hide each other's
    // waits, and its extra shared-memory reads per product lose.  It keeps two tiles on an SM (four of the smallest) where
    // the other form keeps three (seven), so it is taken where that takes no more passes.  Weighted neighbours, us, other form -> twice the
    // threads, float32, 9 taps unless noted; rounds of tiles per SM first:
    //   128 x 64   1: 32 x 197 x 3 heads of 64 66.2 -> 50.0   2: 64 x 197 x 3 x 64 91 -> 82   3: 256 x 65 x 192 337 -> 354 (not taken)   4: 128 x 197 x 3 x 64 165 -> 160
    //   64 x 64    1: 8 x 197 x 192 105 -> 89   3: 20 x 577 x 100 101 -> 119 (not taken)   4: 64 x 197 x 192 267 -> 289   5: 32 x 197 x 384 592 -> 687 (not taken)
    //   32 x 64    1: 8 x 197 x 3 x 64 26.5 -> 25.3   4: 32 x 197 x 192 208 -> 198
    //   32 x 32    1: 1 x 65 x 192 79 -> 53   6: 64 x 197 x 2 heads of 20 19.8 -> 25.1 (not taken)
    // The lines were drawn when operands were weighted and converted as they were fetched, 1.04 to 1.6 times these: since then the other form
    // is ahead at four rounds of 64 x 64, and of bfloat16 tap rows of C values against more stored channels (the coordinate channel, value
    // by value), which gained longest from twice the threads: 64 x 64, 4: 64 x 197 x 192 323 -> 332; 3: 24 x 197 x 384, 9 taps 423 -> 503, 24 x 577 x 96, 8
    // taps 99 -> 118 (not taken); 32 x 32, 7: 159 x 65 x 96, 25 taps 295 -> 308, 6 and one column of tiles: 48 x 577 x 20, 16 taps 44 -> 50 (not taken).
    // Shifted rows cost one division less and gain less (times of before): 16 x 197 x 192 209 -> 177 (1), 64 x 197 x 192 312 -> 342 (4, not taken),
    // 32 x 197 x 72 bfloat16 32 x 32 tiles 0.83 of the time (4).
    if constexpr (MODE == A_NEIGHBOURS || MODE == A_CONV1D) {
        const long long per_sm = (tiles_of[best] + sms - 1) / sms, here = best == 3 ? 4 : 2, other = best == 3 ? 7 : 3;
        bool twice = (per_sm + here - 1) / here <= (per_sm + other - 1) / other;
        if (MODE == A_CONV1D) {
            twice = best == 3 ? per_sm <= (sizeof(T) == 2 ? 4 : 3) : per_sm == 1;
        } else {
            const bool by_value = p.C != p.Cp && sizeof(T) == 2;
            if (per_sm > other && (best == 0 || by_value)) twice = true;
            if (by_value && (best < 3 ? p.taps % 2 != 0 : p.N > 32)) twice = true;
        }
        if (twice) {
            if (best == 0) return launch_tile<TA, T, MODE, 128, 64, 16, 8, 4, 2>(p, st);
            if (best == 1) return launch_tile<TA, T, MODE, 64, 64, 32, 4, 4, 2>(p, st);
            if (best == 2) return launch_tile<TA, T, MODE, 32, 64, 64, 4, 2, 2>(p, st);
            return launch_tile<TA, T, MODE, 32, 32, 32, 4, 2, 4>(p, st);
        }
    }
    if (best == 0) return launch_tile<TA, T, MODE, 128, 64, 16, 8, 8, 3>(p, st);
    if (best == 1) return launch_tile<TA, T, MODE, 64, 64, 32, 8, 4, 3>(p, st);
    if (best == 2) return launch_tile<TA, T, MODE, 32, 64, 64, 4, 4, 2>(p, st);
    return launch_tile<TA, T, MODE, 32, 32, 32, 4, 4, 4>(p, st);
}

template <typename TA, typename T, int MODE>
int launch_mode(const GemmParams& p, cudaStream_t st) {
    if constexpr (MODE == A_ROWS || MODE == A_TOKENS) {
        if constexpr (sizeof(TA) == 4 && sizeof(T) == 4) {
            if (p.a_vec && p.w_vec) return launch_plain_f32<MODE>(p, st);
        }
        return launch_plain_staged<TA, T, MODE>(p, st);
    } else {
        return launch_other_mode<TA, T, MODE>(p, st);
    }
}

template <typename T>
int launch_typed(const GemmParams& p, cudaStream_t st) {
    switch (p.a_mode) {
        case A_ROWS: return launch_mode<T, T, A_ROWS>(p, st);
        case A_TOKENS: return launch_mode<T, T, A_TOKENS>(p, st);
        case A_HEAD_QUIRK: return launch_mode<T, T, A_HEAD_QUIRK>(p, st);
        case A_NEIGHBOURS: return launch_mode<T, T, A_NEIGHBOURS>(p, st);
        default: return launch_mode<T, T, A_CONV1D>(p, st);
    }
}

}  // namespace

int launch_gemm_simt(int dtype, const GemmParams& params, cudaStream_t st) {
    GemmParams p = params;
    if (p.M <= 0 || p.N <= 0) return CONVNN_OK;
    const size_t v4 = dtype == CONVNN_F32 ? 16 : 8;
    auto at4 = [&](const void* q) { return reinterpret_cast<uintptr_t>(q) % v4 == 0; };
    if (p.part_cols <= 0) p.part_cols = p.N;
    if (p.ldw <= 0) p.ldw = p.Kd;
    // four-value accesses: operand rows, weight rows, output rows
    p.a_vec = (p.a_f32 ? aligned16(p.a) : at4(p.a)) && (p.a_mode == A_NEIGHBOURS || p.a_mode == A_CONV1D ? p.Cp % 4 == 0 : p.lda % 4 == 0);
    p.w_vec = at4(p.w) && p.ldw % 4 == 0;
    p.c_vec = at4(p.c) && (!p.c1 || at4(p.c1)) && (!p.c2 || at4(p.c2)) && p.part_cols % 4 == 0 &&
              (p.c_mode == C_ROWS ? p.ldc % 4 == 0 : (p.dk % 4 == 0 && p.Cp % 4 == 0)) &&
              (!p.residual || (at4(p.residual) && p.ldr % 4 == 0));
    if ((p.a_mode == A_NEIGHBOURS || p.a_mode == A_CONV1D) && p.Cp % 4 != 0)
        return set_error(CONVNN_E_UNSUPPORTED, "gemm_simt: %d channels per head are not a multiple of four", p.Cp);
    if (p.a_f32 && dtype == CONVNN_BF16 && p.a_mode != A_ROWS)
        return set_error(CONVNN_E_UNSUPPORTED, "gemm_simt: a float32 operand against bfloat16 weights comes as plain rows");
    const int rc = dtype == CONVNN_F32 ? launch_typed<float>(p, st)
                   : p.a_f32           ? launch_mode<float, __nv_bfloat16, A_ROWS>(p, st)
                                       : launch_typed<__nv_bfloat16>(p, st);
    if (rc) return rc;
    CONVNN_CHECK_LAUNCH("gemm_simt");
    return CONVNN_OK;
}

}  // namespace convnn
