// FP32 GEMMs on the CUDA cores.
//
// They serve what has to stay FP32: the per-op path, the per-block entry
// points and the weight gradients.
//
// Activations times weights on 16-byte aligned rows (gemm_nn_vec_kernel):
// tiles streamed to shared memory by a three-stage cp.async ring, packed fused
// multiply-adds (half the issue slots).  Bound by the FP32 pipes (50 of 74
// TFLOP/s at 8 x 8 outputs per thread): a 145,000 x 128 x 384 product 354 ->
// 277 us against tiles fetched through registers, the FP32 path on 37
// molecules 3.45 -> 2.70 ms a call.  An output's products are summed in the
// order of k in every kernel here, so the choice never changes a bit.
// Other layouts keep the kernel with scalar fallbacks (gemm_nn_kernel).
//
// The A^T B sums have few output tiles (12 of 64 x 64 for a 384 x 128
// gradient) over many rows, so the rows are split until every SM has four
// blocks; without the split the message block of width 128 on 145,000 edges
// spent 75 of its 102 ms there and 28 ms in column sums, which now ride along
// with the tiles of output column 0.
#include <algorithm>
#include "f32x2.cuh"
#include "gemm.cuh"
#include "profile.h"
#include "tc_ptx.cuh"

namespace mlff {

namespace {

constexpr int BK = 16;

// One BK-row step of the product: acc += As[k][rows of ty] Bs[k][cols of tx].
// A thread's TM rows are TM / CM chunks of CM consecutive ones, the chunks
// BM / (TM / CM) apart (columns alike), so that every fragment is one 8- or
// 16-byte shared load and a warp's loads fall into different banks.
template <int BM, int BN, int TM, int TN>
struct Tile {
    static constexpr int CM = TM < 4 ? TM : 4, CN = TN < 4 ? TN : 4;
    static constexpr int RM = TM / CM, RN = TN / CN;
    static constexpr int NTX = BN / TN, NTY = BM / TM, NT = NTX * NTY;
    static constexpr int LDA = BM + 4, LDB = BN + 4;
    static __device__ __forceinline__ int row(int ty, int i) { return (i / CM) * (BM / RM) + ty * CM + i % CM; }
    static __device__ __forceinline__ int col(int tx, int j) { return (j / CN) * (BN / RN) + tx * CN + j % CN; }
    template <int C, int R, int SPAN>
    static __device__ __forceinline__ void frag(const float* s, int t, float* v) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const float* p = s + q * SPAN + t * C;
            if constexpr (C == 4) *reinterpret_cast<float4*>(v + 4 * q) = *reinterpret_cast<const float4*>(p);
            else if constexpr (C == 2) *reinterpret_cast<float2*>(v + 2 * q) = *reinterpret_cast<const float2*>(p);
            else v[q] = *p;
        }
    }
    static __device__ __forceinline__ void step(const float* As, const float* Bs, int ty, int tx,
                                                float (&acc)[TM][TN], float* asum) {
#pragma unroll 4
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
            frag<CM, RM, BM / RM>(As + k * LDA, ty, a);
            frag<CN, RN, BN / RN>(Bs + k * LDB, tx, b);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            if (asum) {
#pragma unroll
                for (int i = 0; i < TM; ++i) asum[i] += a[i];
            }
        }
    }
};

__host__ __device__ inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Any layout: tiles fetched through registers, the next step's loads in flight
// during this step's arithmetic.
template <int MODE, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(Tile<BM, BN, TM, TN>::NT, 4)
    gemm_nn_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                      const float* __restrict__ bias, float* __restrict__ C,
                                                      float* __restrict__ C2, const float* __restrict__ Z,
                                                      int64_t M_static, const int32_t* __restrict__ m_dev, int N,
                                                      int K, int lda, const Status* st) {
    using T = Tile<BM, BN, TM, TN>;
    constexpr int NT = T::NT;
    __shared__ __align__(16) float As[2][BK * T::LDA];
    __shared__ __align__(16) float Bs[2][BK * T::LDB];
    if (st->code != 0) return;
    const int64_t M = m_dev ? (int64_t)(*m_dev) : M_static;
    const int t = threadIdx.x, tx = t % T::NTX, ty = t / T::NTX;
    const int n_tiles = (N + BN - 1) / BN;
    const int64_t m_tiles = (M + BM - 1) / BM;
    // 16-byte loads and stores need rows that are multiples of 4 floats on a
    // 16-byte aligned base
    const bool va = (K & 3) == 0 && (lda & 3) == 0 && aligned16(A), vb = (N & 3) == 0 && aligned16(B);
    const bool vc = T::CN == 4 && (N & 3) == 0 && aligned16(C) && (MODE != 1 || aligned16(C2)) &&
                    (MODE != 2 || aligned16(Z));
    constexpr int LA = BM * BK / NT, LB = BN * BK / NT;   // floats per thread and step
    static_assert(LA % 4 == 0 || LA == 2, "A loads");
    for (int64_t tile = blockIdx.x; tile < m_tiles * n_tiles; tile += gridDim.x) {
        const int64_t m0 = (tile / n_tiles) * BM;
        const int n0 = (int)(tile % n_tiles) * BN;
        float acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int gn = n0 + T::col(tx, j);
                acc[i][j] = MODE >= 3 && gn < N ? bias[gn] : 0.f;
            }
        float ra[LA], rb[LB];
        auto fetch = [&](int k0) {
            if (va && LA >= 4) {
#pragma unroll
                for (int q = 0; q < LA / 4; ++q) {
                    const int i = t + NT * q, r = i / (BK / 4), k = k0 + 4 * (i % (BK / 4));
                    const float4 x = (m0 + r < M && k < K) ? *reinterpret_cast<const float4*>(A + (m0 + r) * lda + k)
                                                           : make_float4(0.f, 0.f, 0.f, 0.f);
                    ra[4 * q] = x.x; ra[4 * q + 1] = x.y; ra[4 * q + 2] = x.z; ra[4 * q + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < LA; ++q) {
                    const int i = t + NT * q, r = i / BK, k = k0 + i % BK;
                    ra[q] = (m0 + r < M && k < K) ? A[(m0 + r) * lda + k] : 0.f;
                }
            }
            if (vb && LB >= 4) {
#pragma unroll
                for (int q = 0; q < LB / 4; ++q) {
                    const int i = t + NT * q, k = k0 + i / (BN / 4), n = n0 + 4 * (i % (BN / 4));
                    const float4 x = (k < K && n < N) ? *reinterpret_cast<const float4*>(B + (int64_t)k * N + n)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                    rb[4 * q] = x.x; rb[4 * q + 1] = x.y; rb[4 * q + 2] = x.z; rb[4 * q + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < LB; ++q) {
                    const int i = t + NT * q, k = k0 + i / BN, n = n0 + i % BN;
                    rb[q] = (k < K && n < N) ? B[(int64_t)k * N + n] : 0.f;
                }
            }
        };
        auto put = [&](int b) {
            if (va && LA >= 4) {
#pragma unroll
                for (int q = 0; q < LA / 4; ++q) {
                    const int i = t + NT * q, r = i / (BK / 4), k = 4 * (i % (BK / 4));
#pragma unroll
                    for (int j = 0; j < 4; ++j) As[b][(k + j) * T::LDA + r] = ra[4 * q + j];
                }
            } else {
#pragma unroll
                for (int q = 0; q < LA; ++q) {
                    const int i = t + NT * q;
                    As[b][(i % BK) * T::LDA + i / BK] = ra[q];
                }
            }
            if (vb && LB >= 4) {
#pragma unroll
                for (int q = 0; q < LB / 4; ++q) {
                    const int i = t + NT * q;
                    *reinterpret_cast<float4*>(&Bs[b][(i / (BN / 4)) * T::LDB + 4 * (i % (BN / 4))]) =
                        make_float4(rb[4 * q], rb[4 * q + 1], rb[4 * q + 2], rb[4 * q + 3]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < LB; ++q) {
                    const int i = t + NT * q;
                    Bs[b][(i / BN) * T::LDB + i % BN] = rb[q];
                }
            }
        };
        fetch(0);
        put(0);
        __syncthreads();
        int b = 0;
        for (int k0 = 0; k0 < K; k0 += BK, b ^= 1) {
            const bool more = k0 + BK < K;
            if (more) fetch(k0 + BK);   // in flight during this step's arithmetic
            T::step(As[b], Bs[b], ty, tx, acc, nullptr);
            if (more) put(b ^ 1);
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int64_t gm = m0 + T::row(ty, i);
            if (gm >= M) continue;
#pragma unroll
            for (int j0 = 0; j0 < TN; j0 += T::CN) {
                const int gn = n0 + T::col(tx, j0);
                const int64_t idx = gm * N + gn;
                if (vc && gn < N) {
                    float v[4];
#pragma unroll
                    for (int j = 0; j < T::CN; ++j) v[j] = acc[i][j0 + j];
                    if (MODE < 2 && bias) {
#pragma unroll
                        for (int j = 0; j < T::CN; ++j) v[j] += bias[gn + j];
                    }
                    if (MODE == 2) {
                        const float4 z = *reinterpret_cast<const float4*>(Z + idx);
                        v[0] *= dsilu_f(z.x); v[1] *= dsilu_f(z.y); v[2] *= dsilu_f(z.z); v[3] *= dsilu_f(z.w);
                    }
                    if (MODE == 4) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[j] = silu_f(v[j]);
                    }
                    *reinterpret_cast<float4*>(C + idx) = make_float4(v[0], v[1], v[2], v[3]);
                    if (MODE == 1)
                        *reinterpret_cast<float4*>(C2 + idx) =
                            make_float4(silu_f(v[0]), silu_f(v[1]), silu_f(v[2]), silu_f(v[3]));
                } else {
#pragma unroll
                    for (int j = 0; j < T::CN; ++j) {
                        if (gn + j >= N) continue;
                        float v = acc[i][j0 + j];
                        if (MODE < 2 && bias) v += bias[gn + j];
                        if (MODE == 2) v *= dsilu_f(Z[idx + j]);
                        C[idx + j] = MODE == 4 ? silu_f(v) : v;
                        if (MODE == 1) C2[idx + j] = silu_f(v);
                    }
                }
            }
        }
    }
}

// The same product on 16-byte aligned rows: lda, K and N multiples of 4,
// every pointer 16-byte aligned.  One tile per block: persistent blocks that
// prefetch across tiles end unevenly (145,000 x 384 x 128: 355 against 303
// us).  A stays row-major in shared memory (a thread reads 4 k's of a row at
// once), its rows padded by 4 floats against bank conflicts; thread (ty, tx)
// holds rows ty + i NTY and columns tx 4 + j.
template <int MODE, int BM, int BN, int TM, int TN, int KS>
struct VecTile {
    static constexpr int NTX = BN / TN, NTY = BM / TM, NT = NTX * NTY, LDA = KS + 4;
    static constexpr int SA = BM * LDA, SB = KS * BN, STAGES = 3;
    static constexpr int SMEM = STAGES * (SA + SB) * 4;
    static_assert(SMEM <= 48 * 1024, "shared memory without opt-in");
    static_assert((BM * KS / 4) % NT == 0 && (BN * KS / 4) % NT == 0 && TN % 4 == 0, "16-byte loads");
};

template <int MODE, int BM, int BN, int TM, int TN, int KS, int PER_SM>
__global__ void __launch_bounds__(VecTile<MODE, BM, BN, TM, TN, KS>::NT, PER_SM)
    gemm_nn_vec_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ bias,
                       float* __restrict__ C, float* __restrict__ C2, const float* __restrict__ Z, int64_t M_static,
                       const int32_t* __restrict__ m_dev, int N, int K, int lda, const Status* st) {
    using T = VecTile<MODE, BM, BN, TM, TN, KS>;
    constexpr int NT = T::NT, STAGES = T::STAGES;
    extern __shared__ __align__(16) float ring[];
    if (st->code != 0) return;
    const int64_t M = m_dev ? (int64_t)(*m_dev) : M_static;
    const int t = threadIdx.x, tx = t % T::NTX, ty = t / T::NTX;
    const int n_tiles = (N + BN - 1) / BN, steps = (K + KS - 1) / KS;
    const int64_t m0 = (blockIdx.x / n_tiles) * (int64_t)BM;
    const int n0 = (int)(blockIdx.x % n_tiles) * BN;
    if (m0 >= M) return;
    auto load = [&](int s) {   // K-step s into its slot of the ring
        if (s < steps) {
            float* as = ring + s % STAGES * (T::SA + T::SB);
            float* bs = as + T::SA;
            const int k0 = s * KS;
#pragma unroll
            for (int q = 0; q < BM * KS / 4 / NT; ++q) {
                const int i = t + NT * q, r = i / (KS / 4), k = 4 * (i % (KS / 4));
                const bool ok = m0 + r < M && k0 + k < K;
                tc::cp_async16_or_zero(as + r * T::LDA + k, ok ? A + (m0 + r) * lda + k0 + k : A, ok);
            }
#pragma unroll
            for (int q = 0; q < BN * KS / 4 / NT; ++q) {
                const int i = t + NT * q, k = i / (BN / 4), n = 4 * (i % (BN / 4));
                const bool ok = k0 + k < K && n0 + n < N;
                tc::cp_async16_or_zero(bs + k * BN + n, ok ? B + (int64_t)(k0 + k) * N + n0 + n : B, ok);
            }
        }
        tc::cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load(s);
    f32x2 acc[TM][TN / 2];
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
        const int gn = n0 + (j / 2) * (BN / (TN / 4)) + tx * 4 + 2 * (j % 2);
        const f32x2 a0 = MODE >= 3 && gn < N ? pack2(bias[gn], bias[gn + 1]) : pack2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = a0;
    }
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();   // the step has landed, and its slot before last is read
        load(s + STAGES - 1);
        const float* as = ring + s % STAGES * (T::SA + T::SB);
        const float* bs = as + T::SA;
#pragma unroll
        for (int k4 = 0; k4 < KS; k4 += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i)
                a[i] = *reinterpret_cast<const float4*>(as + (i * T::NTY + ty) * T::LDA + k4);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float4 b[TN / 4];
#pragma unroll
                for (int j = 0; j < TN / 4; ++j)
                    b[j] = *reinterpret_cast<const float4*>(bs + (k4 + k) * BN + j * (BN / (TN / 4)) + tx * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float x = k == 0 ? a[i].x : k == 1 ? a[i].y : k == 2 ? a[i].z : a[i].w;
                    const f32x2 xx = pack2(x, x);
#pragma unroll
                    for (int j = 0; j < TN / 4; ++j) {
                        acc[i][2 * j] = fma2(xx, pack2(b[j].x, b[j].y), acc[i][2 * j]);
                        acc[i][2 * j + 1] = fma2(xx, pack2(b[j].z, b[j].w), acc[i][2 * j + 1]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < TN / 4; ++j) {
        const int gn = n0 + j * (BN / (TN / 4)) + tx * 4;
        if (gn >= N) continue;
        float bj[4] = {0.f, 0.f, 0.f, 0.f};
        if (MODE < 2 && bias) {
#pragma unroll
            for (int q = 0; q < 4; ++q) bj[q] = __ldg(bias + gn + q);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int64_t gm = m0 + i * T::NTY + ty;
            if (gm >= M) break;
            const int64_t idx = gm * N + gn;
            float v[4] = {lo2(acc[i][2 * j]), hi2(acc[i][2 * j]), lo2(acc[i][2 * j + 1]), hi2(acc[i][2 * j + 1])};
            if (MODE < 2 && bias) {
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] += bj[q];
            }
            if (MODE == 2) {
                const float4 z = __ldg(reinterpret_cast<const float4*>(Z + idx));
                v[0] *= dsilu_f(z.x); v[1] *= dsilu_f(z.y); v[2] *= dsilu_f(z.z); v[3] *= dsilu_f(z.w);
            }
            if (MODE == 4) {
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = silu_f(v[q]);
            }
            *reinterpret_cast<float4*>(C + idx) = make_float4(v[0], v[1], v[2], v[3]);
            if (MODE == 1)
                *reinterpret_cast<float4*>(C2 + idx) =
                    make_float4(silu_f(v[0]), silu_f(v[1]), silu_f(v[2]), silu_f(v[3]));
        }
    }
    tc::cp_async_wait_all();
}

// partial[split][m][n] over the split's rows, partial column sums behind the
// splits' matrices
constexpr int TNB = 64;           // output tile 64 x 64, 4 x 4 per thread
constexpr int TN_MAX_SPLIT = 256;
constexpr int TN_TARGET_BLOCKS = 152 * 4;
constexpr int TN_MIN_ROWS = 64;   // rows per split

inline int tn_tiles(int64_t n) { return (int)std::max<int64_t>(1, (n + TNB - 1) / TNB); }
inline int tn_splits(int64_t M, int64_t N) {
    const int tiles = tn_tiles(M) * tn_tiles(N);
    return std::max(2, std::min(TN_MAX_SPLIT, (TN_TARGET_BLOCKS + tiles - 1) / tiles));
}

// splits [0, nsplit / segments) cover the first set of rows, the rest the second
__global__ void __launch_bounds__(256, 4) gemm_tn_kernel(GemmRows x, int lda, int ldb, int M, int N, int64_t rows,
                                                         int nsplit, int want_sum, float* __restrict__ part,
                                                         const Status* st) {
    using T = Tile<TNB, TNB, 4, 4>;
    __shared__ __align__(16) float As[2][BK * T::LDA];
    __shared__ __align__(16) float Bs[2][BK * T::LDB];
    if (st->code != 0) return;
    const int tiles_n = max(1, (N + TNB - 1) / TNB);
    const int m0 = (blockIdx.x / tiles_n) * TNB, n0 = (blockIdx.x % tiles_n) * TNB;
    const int seg_splits = x.A1 ? nsplit / 2 : nsplit, seg = blockIdx.y / seg_splits;
    const float* A = seg ? x.A1 : x.A;
    const float* B = seg ? x.B1 : x.B;
    int64_t per = (rows + seg_splits - 1) / seg_splits;
    if (per < TN_MIN_ROWS) per = TN_MIN_ROWS;
    const int64_t r0 = (int64_t)(blockIdx.y - seg * seg_splits) * per, r1 = min(rows, r0 + per);
    const int t = threadIdx.x, tx = t % T::NTX, ty = t / T::NTX;
    const bool va = (lda & 3) == 0 && (M & 3) == 0 && aligned16(A);
    const bool vb = (ldb & 3) == 0 && (N & 3) == 0 && aligned16(B);
    const bool sums = want_sum && n0 == 0 && seg == 0;
    float acc[4][4] = {}, asum[4] = {};
    float ra[4], rb[4];
    auto fetch1 = [&](const float* S, int ld, int c0, int ncol, bool vec, int64_t r, float (&v)[4]) {
        if (vec) {
            const int c = c0 + 4 * (t % (TNB / 4));
            const int64_t row = r + t / (TNB / 4);
            const float4 x = (row < r1 && c < ncol) ? *reinterpret_cast<const float4*>(S + row * ld + c)
                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = t + 256 * q, c = c0 + i % TNB;
                const int64_t row = r + i / TNB;
                v[q] = (row < r1 && c < ncol) ? S[row * ld + c] : 0.f;
            }
        }
    };
    auto put1 = [&](float* D, int ldd, bool vec, const float (&v)[4]) {
        if (vec)
            *reinterpret_cast<float4*>(D + (t / (TNB / 4)) * ldd + 4 * (t % (TNB / 4))) =
                make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = t + 256 * q;
                D[(i / TNB) * ldd + i % TNB] = v[q];
            }
        }
    };
    if (r0 < r1) {
        fetch1(A, lda, m0, M, va, r0, ra);
        fetch1(B, ldb, n0, N, vb, r0, rb);
        put1(As[0], T::LDA, va, ra);
        put1(Bs[0], T::LDB, vb, rb);
        __syncthreads();
        int b = 0;
        for (int64_t r = r0; r < r1; r += BK, b ^= 1) {
            const bool more = r + BK < r1;
            if (more) {
                fetch1(A, lda, m0, M, va, r + BK, ra);
                fetch1(B, ldb, n0, N, vb, r + BK, rb);
            }
            T::step(As[b], Bs[b], ty, tx, acc, sums ? asum : nullptr);
            if (more) {
                put1(As[b ^ 1], T::LDA, va, ra);
                put1(Bs[b ^ 1], T::LDB, vb, rb);
            }
            __syncthreads();
        }
    }
    float* out = part + (int64_t)blockIdx.y * M * N;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + 4 * ty + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + 4 * tx + j;
            if (n < N) out[(int64_t)m * N + n] = acc[i][j];
        }
        if (want_sum && n0 == 0 && tx == 0) part[(int64_t)nsplit * M * N + (int64_t)blockIdx.y * M + m] = asum[i];
    }
}

// The same sums on 16-byte aligned rows (lda, ldb, M and N multiples of 4):
// rows through the cp.async ring, 8 x 4 outputs per thread in packed pairs of
// m.  The same rows per split in the same order, so the same bits.
// 145,000 rows, 128 x 384: 298 -> 241 us.
constexpr int TV_NT = 128, TV_STAGES = 3;
__global__ void __launch_bounds__(TV_NT, 4) gemm_tn_vec_kernel(GemmRows x, int lda, int ldb, int M, int N,
                                                               int64_t rows, int nsplit, int want_sum,
                                                               float* __restrict__ part, const Status* st) {
    __shared__ __align__(16) float ring[TV_STAGES][2][BK * TNB];
    if (st->code != 0) return;
    const int tiles_n = max(1, (N + TNB - 1) / TNB);
    const int m0 = (blockIdx.x / tiles_n) * TNB, n0 = (blockIdx.x % tiles_n) * TNB;
    const int seg_splits = x.A1 ? nsplit / 2 : nsplit, seg = blockIdx.y / seg_splits;
    const float* A = seg ? x.A1 : x.A;
    const float* B = seg ? x.B1 : x.B;
    int64_t per = (rows + seg_splits - 1) / seg_splits;
    if (per < TN_MIN_ROWS) per = TN_MIN_ROWS;
    const int64_t r0 = (int64_t)(blockIdx.y - seg * seg_splits) * per, r1 = min(rows, r0 + per);
    const int steps = r0 < r1 ? (int)((r1 - r0 + BK - 1) / BK) : 0;
    const int t = threadIdx.x, tx = t % 16, ty = t / 16;   // outputs m0 + 4 ty + {0..3, 32..35}, n0 + 4 tx + {0..3}
    const bool sums = want_sum && n0 == 0 && seg == 0;
    auto load = [&](int s) {
        if (s < steps) {
#pragma unroll
            for (int q = 0; q < BK * TNB / 4 / TV_NT; ++q) {
                const int i = t + TV_NT * q, r = i / (TNB / 4), c = 4 * (i % (TNB / 4));
                const int64_t row = r0 + (int64_t)s * BK + r;
                const bool oa = row < r1 && m0 + c < M, ob = row < r1 && n0 + c < N;
                tc::cp_async16_or_zero(&ring[s % TV_STAGES][0][r * TNB + c], oa ? A + row * lda + m0 + c : A, oa);
                tc::cp_async16_or_zero(&ring[s % TV_STAGES][1][r * TNB + c], ob ? B + row * ldb + n0 + c : B, ob);
            }
        }
        tc::cp_async_commit();
    };
    f32x2 acc[4][4], asum[4];   // [pair of m][n]
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        asum[i] = pack2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = pack2(0.f, 0.f);
    }
    const f32x2 one = pack2(1.f, 1.f);
#pragma unroll
    for (int s = 0; s < TV_STAGES - 1; ++s) load(s);
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(TV_STAGES - 2) : "memory");
        __syncthreads();
        load(s + TV_STAGES - 1);
        const float* as = ring[s % TV_STAGES][0] + 4 * ty;
        const float* bs = ring[s % TV_STAGES][1] + 4 * tx;
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const float4 a0 = *reinterpret_cast<const float4*>(as + k * TNB);
            const float4 a1 = *reinterpret_cast<const float4*>(as + k * TNB + 32);
            const float4 b4 = *reinterpret_cast<const float4*>(bs + k * TNB);
            const f32x2 a[4] = {pack2(a0.x, a0.y), pack2(a0.z, a0.w), pack2(a1.x, a1.y), pack2(a1.z, a1.w)};
            const f32x2 b[4] = {pack2(b4.x, b4.x), pack2(b4.y, b4.y), pack2(b4.z, b4.z), pack2(b4.w, b4.w)};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i], b[j], acc[i][j]);
            if (sums) {
#pragma unroll
                for (int i = 0; i < 4; ++i) asum[i] = fma2(a[i], one, asum[i]);
            }
        }
    }
    tc::cp_async_wait_all();
    float* out = part + (int64_t)blockIdx.y * M * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + 4 * ty + (i / 4) * 32 + i % 4, n = n0 + 4 * tx;
        if (m >= M) continue;
        auto half = [&](f32x2 v) { return i % 2 ? hi2(v) : lo2(v); };
        if (n < N)
            *reinterpret_cast<float4*>(out + (int64_t)m * N + n) =
                make_float4(half(acc[i / 2][0]), half(acc[i / 2][1]), half(acc[i / 2][2]), half(acc[i / 2][3]));
        if (want_sum && n0 == 0 && tx == 0)
            part[(int64_t)nsplit * M * N + (int64_t)blockIdx.y * M + m] = half(asum[i / 2]);
    }
}

// sums over the splits, in split order: four interleaved chains per output
__global__ void __launch_bounds__(128) gemm_tn_sum_kernel(const float* __restrict__ part, int64_t MN, int M,
                                                          int nsplit, int acc, float* __restrict__ C,
                                                          float* __restrict__ colsum, const Status* st) {
    if (st->code != 0) return;
    const int64_t total = (C ? MN : 0) + (colsum ? M : 0);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const bool col = !C || i >= MN;
        const int64_t j = col ? i - (C ? MN : 0) : i;
        const float* p = col ? part + (int64_t)nsplit * MN + j : part + j;
        const int64_t stride = col ? M : MN;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        int sp = 0;
        for (; sp + 16 <= nsplit; sp += 16) {   // 16 loads in flight
            float x[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) x[q] = p[(int64_t)(sp + q) * stride];
#pragma unroll
            for (int q = 0; q < 16; ++q) s[q & 3] += x[q];
        }
        for (; sp + 4 <= nsplit; sp += 4)
#pragma unroll
            for (int q = 0; q < 4; ++q) s[q] += p[(int64_t)(sp + q) * stride];
        for (; sp < nsplit; ++sp) s[0] += p[(int64_t)sp * stride];
        const float v = (s[0] + s[1]) + (s[2] + s[3]);
        float* o = (col ? colsum : C) + j;
        *o = acc ? *o + v : v;
    }
}

struct NnArgs {
    const float *A, *B, *bias;
    float *C, *C2;
    const float* Z;
    int64_t M;
    const int32_t* m_dev;
    int N, K, lda;
    const Status* st;
};

template <int MODE, int BM, int BN, int TM, int TN>
int launch_nn(const NnArgs& a, cudaStream_t s, int per_sm) {
    const int64_t tiles = ((a.M + BM - 1) / BM) * ((a.N + BN - 1) / BN);
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)num_sms() * per_sm));
    gemm_nn_kernel<MODE, BM, BN, TM, TN><<<blocks, Tile<BM, BN, TM, TN>::NT, 0, s>>>(
        a.A, a.B, a.bias, a.C, a.C2, a.Z, a.M, a.m_dev, a.N, a.K, a.lda, a.st);
    MLFF_LAUNCH_CHECK("gemm_nn");
    return MLFF_OK;
}
template <int MODE, int BM, int BN, int TM, int TN, int KS, int PER_SM>
int launch_nn_vec(const NnArgs& a, cudaStream_t s) {
    using T = VecTile<MODE, BM, BN, TM, TN, KS>;
    const int64_t tiles = ((a.M + BM - 1) / BM) * ((a.N + BN - 1) / BN);
    if (tiles == 0) return MLFF_OK;
    gemm_nn_vec_kernel<MODE, BM, BN, TM, TN, KS, PER_SM><<<(unsigned)tiles, T::NT, T::SMEM, s>>>(
        a.A, a.B, a.bias, a.C, a.C2, a.Z, a.M, a.m_dev, a.N, a.K, a.lda, a.st);
    MLFF_LAUNCH_CHECK("gemm_nn_vec");
    return MLFF_OK;
}

template <int MODE>
int nn_mode(const NnArgs& a, cudaStream_t s) {
    auto tiles = [&](int bm, int bn) { return ((a.M + bm - 1) / bm) * ((a.N + bn - 1) / bn); };
    const int64_t want = 2LL * num_sms();
    const bool vec = (a.K & 3) == 0 && (a.lda & 3) == 0 && (a.N & 3) == 0 && aligned16(a.A) && aligned16(a.B) &&
                     aligned16(a.C) && (MODE != 1 || aligned16(a.C2)) && (MODE != 2 || aligned16(a.Z));
    if (vec) {
        // 64 x 128 tiles keep the FP32 pipes busiest once every SM has two (16,000 x 128 x 384: 43
        // against 49 us); below, 32 x 32 ones fill the SMs (2,400 x 384 x 128: 12 against 29 us)
        if (a.N > 64 && tiles(64, 128) >= want) return launch_nn_vec<MODE, 64, 128, 8, 8, 16, 4>(a, s);
        return launch_nn_vec<MODE, 32, 32, 4, 4, 32, 8>(a, s);
    }
    if (2 * tiles(64, 64) >= want) return launch_nn<MODE, 64, 64, 4, 4>(a, s, 6);
    return launch_nn<MODE, 32, 32, 2, 2>(a, s, 8);
}

}  // namespace

int gemm_nn(int mode, const float* A, const float* B, const float* bias, float* C, float* C2, const float* Z,
            int64_t M, const int32_t* m_dev, int N, int K, const Status* st, cudaStream_t s, int lda) {
    ProfScope prof(PK_PLAIN_GEMM, s);
    const NnArgs a{A, B, bias, C, C2, Z, M, m_dev, N, K, lda ? lda : K, st};
    return mode == 0   ? nn_mode<0>(a, s)
           : mode == 1 ? nn_mode<1>(a, s)
           : mode == 2 ? nn_mode<2>(a, s)
           : mode == 3 ? nn_mode<3>(a, s)
                       : nn_mode<4>(a, s);
}

size_t gemm_tn_floats(int64_t M, int64_t N) { return (size_t)tn_splits(M, N) * (size_t)(M * N + M); }

int gemm_tn(const GemmRows& x, int lda, int ldb, int M, int N, int64_t rows, float* C, float* colsum,
            bool accumulate, float* part, const Status* st, cudaStream_t s) {
    ProfScope prof(PK_PLAIN_GEMM, s);
    // a split holds at least TN_MIN_ROWS rows; two sets of rows take half of the splits each
    int ns = (int)std::max<int64_t>(1, std::min<int64_t>(tn_splits(M, N), (rows + TN_MIN_ROWS - 1) / TN_MIN_ROWS));
    if (x.A1) ns = 2 * std::max(1, ns / 2);
    dim3 grid(tn_tiles(M) * tn_tiles(N), ns);
    const bool vec = ((lda | ldb | M | N) & 3) == 0 && aligned16(x.A) && aligned16(x.B) && aligned16(x.A1) &&
                     aligned16(x.B1) && aligned16(part);
    if (vec) gemm_tn_vec_kernel<<<grid, TV_NT, 0, s>>>(x, lda, ldb, M, N, rows, ns, colsum != nullptr, part, st);
    else gemm_tn_kernel<<<grid, 256, 0, s>>>(x, lda, ldb, M, N, rows, ns, colsum != nullptr, part, st);
    MLFF_LAUNCH_CHECK("gemm_tn");
    const int64_t out = (int64_t)M * N + M;
    gemm_tn_sum_kernel<<<(int)std::min<int64_t>((out + 127) / 128, 152 * 16), 128, 0, s>>>(
        part, (int64_t)M * N, M, ns, accumulate ? 1 : 0, C, colsum, st);
    MLFF_LAUNCH_CHECK("gemm_tn_sum");
    return MLFF_OK;
}

}  // namespace mlff
