// The update block in FP32 on the CUDA cores, fused, for the table path:
// forward and adjoint of PaiNNUpdate (student_model.py:434-470).
//
// One CTA of 256 threads per tile of TA atoms.  The tile's MLP inputs sit in
// shared memory transposed ([k][atom]); the weights (k-major rows, 320 KB in
// all) stream through a ring of bulk copies, 16 k-rows per stage.  A thread
// owns TA / 8 atoms x 4 channels of every 128-wide output chunk, so the
// gates, the 3 x 3 mixing and the norm's derivative stay in its registers.
// The MLP's wide reductions (256 -> 128, 384 -> 128) run as two halves of k
// in the two halves of the CTA, 8 channels per thread, added through shared
// memory: 16 shared-memory floats per 64 fused multiply-adds.
//
// Why not the tensor cores here (tc_update.cu): split-FP16 MMAs accumulate
// with truncation, 24 to 48 of them per output, and that bias (2e-6 of the
// energy) was what was left of the error once the edge filters were
// evaluated in FP32; and at 3,000 atoms the tensor-core tiles are bound by
// their chain of weight stream, two GEMMs and epilogues.
#include <algorithm>
#include <mutex>
#include "common.cuh"
#include "workspace.h"
#include "profile.h"
#include "tab_edge.cuh"
#include "tc_ptx.cuh"

namespace mlff {

namespace {

constexpr int UPT = 256;            // threads
constexpr int KC = 16;              // k-rows of a stage
constexpr int STAGES = 3;
constexpr uint32_t STAGE_BYTES = KC * H3 * 4;   // 24 KB: the widest chunk

// Streams chunks of weights: chunk i of a tile is one or two blocks of KC
// rows (two: the two k-halves of a wide reduction).
struct WStream {
    unsigned char* ring;
    uint64_t* full;
    int* abort_flag;
    Status* st;
    uint32_t issued = 0, used = 0;
    __device__ __forceinline__ unsigned char* stage(uint32_t i) const { return ring + (i % STAGES) * STAGE_BYTES; }
    // (one thread) copies of n_blocks blocks of `bytes` at src + b * stride
    __device__ __forceinline__ void issue(const float* src, int n_blocks, int64_t stride, uint32_t bytes) {
        uint64_t* bar = full + issued % STAGES;
        tc::mbar_expect_tx(bar, n_blocks * bytes);
        for (int b = 0; b < n_blocks; ++b) tc::bulk_g2s(stage(issued) + b * bytes, src + b * stride, bytes, bar);
        ++issued;
    }
    // every thread: chunk `used` has landed
    __device__ __forceinline__ const float* wait() {
        if (!*(volatile int*)abort_flag && !tc::mbar_wait(full + used % STAGES, (used / STAGES) & 1, tc::WAIT_BUDGET)) {
            set_status(st, MLFF_ERR_TIMEOUT, 60);
            *(volatile int*)abort_flag = 1;
        }
        return reinterpret_cast<const float*>(stage(used));
    }
};

// acc[i][2 j], [2 j + 1] += a[i] w[j pairs] over KC k-rows: R atoms from As
// (row stride LD), NQ float4 of weights from Ws (row stride WLD floats, the
// quads QS floats apart)
template <int R, int NQ, int LD, int WLD, int QS>
__device__ __forceinline__ void mm_chunk(const float* As, const float* Ws, f32x2 (&acc)[R][2 * NQ]) {
#pragma unroll 4
    for (int k = 0; k < KC; ++k) {
        float a[R];
        if constexpr (R >= 4) {
#pragma unroll
            for (int q = 0; q < R / 4; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(As + k * LD + 4 * q);
                a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
            }
        } else {
            const float2 v = *reinterpret_cast<const float2*>(As + k * LD);
            a[0] = v.x; a[1] = v.y;
        }
        f32x2 w[2 * NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Ws + k * WLD + q * QS);
            w[2 * q] = v.x;
            w[2 * q + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const f32x2 aa = pack2(a[i], a[i]);
#pragma unroll
            for (int j = 0; j < 2 * NQ; ++j) acc[i][j] = fma2(aa, w[j], acc[i][j]);
        }
    }
}

template <int TA, int KIN>
struct UpdShape {
    static constexpr int R = TA / 8;               // atoms per thread
    static constexpr int LD = TA + 4;              // row stride of the transposed tiles
    static constexpr uint32_t A_BYTES = KIN * LD * 4;
    static constexpr uint32_t OFF_RING = 0;
    static constexpr uint32_t OFF_A = STAGES * STAGE_BYTES;
    static constexpr uint32_t OFF_H = OFF_A + A_BYTES;                   // second reduction's input [H][LD]
    static constexpr uint32_t OFF_BAR = OFF_H + H * LD * 4;
    static constexpr uint32_t SMEM = OFF_BAR + 8 * STAGES + 64;
    static_assert(OFF_A % 16 == 0 && OFF_H % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
    static_assert(SMEM <= 232448, "shared memory");
    // the second k-half's partial sums, [R * 8][UPT / 2] floats, pass through the second tile
    static_assert(UPT / 2 * R * 8 * 4 <= (int)(H * LD * 4), "partial sums fit the second tile");
};

// Chunk sequence of one tile: first KIN / 2 / KC chunks of two half blocks
// (rows k and KIN / 2 + k of W1 [KIN][H]), then H / KC chunks of W2 [H][N2].
template <int KIN, int N2>
struct ChunkPlan {
    static constexpr int C1 = KIN / 2 / KC, C2 = H / KC, PER = C1 + C2;
    static __device__ __forceinline__ void issue(WStream& ws, uint32_t total, const float* W1, const float* W2) {
        if (ws.issued >= total) return;
        const int c = ws.issued % PER;
        if (c < C1) ws.issue(W1 + (int64_t)c * KC * H, 2, (int64_t)(KIN / 2) * H, KC * H * 4);
        else ws.issue(W2 + (int64_t)(c - C1) * KC * N2, 1, 0, KC * N2 * 4);
    }
};

// The two GEMMs of a tile: hT = op(sum over KIN of A W1) left in Hs by the
// caller's `mid(acc)` (threads of the first half), then out = Hs W2.
template <int TA, int KIN, int N2, class Mid>
__device__ __forceinline__ void two_gemms(WStream& ws, uint32_t total, const float* W1, const float* W2,
                                          const float* As, float* Hs, int t, Mid&& mid,
                                          f32x2 (&out)[TA / 8][N2 / 64]) {
    using S = UpdShape<TA, KIN>;
    using C = ChunkPlan<KIN, N2>;
    constexpr int R = S::R;
    {
        const int half = t >> 7, tt = t & 127, tx = tt & 15, ty = tt >> 4;
        f32x2 acc[R][4];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = pack2(0.f, 0.f);
        for (int c = 0; c < C::C1; ++c) {
            const float* W = ws.wait() + half * KC * H + 4 * tx;
            mm_chunk<R, 2, S::LD, H, 64>(As + (half * (KIN / 2) + c * KC) * S::LD + ty * R, W, acc);
            ++ws.used;
            __syncthreads();
            if (t == 0) C::issue(ws, total, W1, W2);
        }
        // the second half's sums through shared memory (slot-major: conflict-free)
        if (half == 1) {
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    Hs[((i * 4 + j) * 2) * 128 + tt] = lo2(acc[i][j]);
                    Hs[((i * 4 + j) * 2 + 1) * 128 + tt] = hi2(acc[i][j]);
                }
        }
        __syncthreads();
        float sum[R][8];
        if (half == 0) {
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sum[i][2 * j] = lo2(acc[i][j]) + Hs[((i * 4 + j) * 2) * 128 + tt];
                    sum[i][2 * j + 1] = hi2(acc[i][j]) + Hs[((i * 4 + j) * 2 + 1) * 128 + tt];
                }
        }
        __syncthreads();
        if (half == 0) {
            // channels 4 tx + j (j < 4) and 64 + 4 tx + j - 4, atoms ty R + i: value -> Hs[channel][atom]
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int ch = (j < 4 ? 0 : 64) + 4 * tx + (j & 3);
                float v[R];
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = mid(ch, ty * R + i, sum[i][j]);
                float* o = Hs + ch * S::LD + ty * R;
                if constexpr (R >= 4) {
#pragma unroll
                    for (int q = 0; q < R / 4; ++q)
                        *reinterpret_cast<float4*>(o + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                } else {
                    *reinterpret_cast<float2*>(o) = make_float2(v[0], v[1]);
                }
            }
        }
        __syncthreads();
    }
    constexpr int NQ = N2 / H;
    const int tx = t & 31, ty = t >> 5;
    for (int c = 0; c < C::C2; ++c) {
        const float* W = ws.wait() + 4 * tx;
        mm_chunk<R, NQ, S::LD, N2, H>(Hs + c * KC * S::LD + ty * R, W, out);
        ++ws.used;
        __syncthreads();
        if (t == 0) C::issue(ws, total, W1, W2);
    }
}

// the four floats of quad q of row i of a thread's outputs
template <int N>
__device__ __forceinline__ float4 quad(const f32x2 (&row)[N], int q) {
    return make_float4(lo2(row[2 * q]), hi2(row[2 * q]), lo2(row[2 * q + 1]), hi2(row[2 * q + 1]));
}

__device__ __forceinline__ void init_stream(WStream& ws, unsigned char* bars, unsigned char* ring, Status* st, int t) {
    ws.ring = ring;
    ws.full = reinterpret_cast<uint64_t*>(bars);
    ws.abort_flag = reinterpret_cast<int*>(bars + 8 * STAGES);
    ws.st = st;
    if (t == 0) {
        for (int i = 0; i < STAGES; ++i) tc::mbar_init(ws.full + i, 1);
        tc::fence_mbar_init();
        *ws.abort_flag = 0;
    }
    __syncthreads();
}
// every copy issued has landed before the CTA exits
__device__ __forceinline__ void drain_stream(WStream& ws, int t) {
    if (t == 0)
        for (; ws.used < ws.issued; ++ws.used)
            if (!tc::mbar_wait(ws.full + ws.used % STAGES, (ws.used / STAGES) & 1, tc::WAIT_BUDGET)) {
                set_status(ws.st, MLFF_ERR_TIMEOUT, 61);
                break;
            }
    __syncthreads();
}

template <int TA>
__global__ void __launch_bounds__(UPT) upd32_fwd_kernel(const float* __restrict__ P, LayerOffsets lo,
                                                        const float* __restrict__ Xt, int n_atoms,
                                                        float* __restrict__ Xout, int out_layout,
                                                        float* __restrict__ uz, float* __restrict__ ua, Status* st) {
    using S = UpdShape<TA, 2 * H>;
    using C = ChunkPlan<2 * H, H3>;
    constexpr int R = S::R;
    extern __shared__ __align__(128) unsigned char smem[];
    float* As = reinterpret_cast<float*>(smem + S::OFF_A);
    float* Hs = reinterpret_cast<float*>(smem + S::OFF_H);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int ntiles = (n_atoms + TA - 1) / TA;
    const uint32_t total = (uint32_t)((ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * C::PER;
    const float *W1 = P + lo.u1t, *W2 = P + lo.u2t;
    WStream ws;
    init_stream(ws, smem + S::OFF_BAR, smem + S::OFF_RING, st, t);
    if (t == 0)
        for (int i = 0; i < STAGES; ++i) C::issue(ws, total, W1, W2);
    float mix[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) mix[i] = P[lo.mix + i];
    pdl_wait();   // the weights above overlap the previous kernel
    pdl_trigger();
    if (st->code == 0) {
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int a0 = tile * TA;
            // inputs [s, |v|], transposed: lane = atom, warps over groups of 4 channels
            for (int i = w; i < (TA >= 32 ? TA : 16); i += 8) {
                // (TA >= 32: c4 = i % 32, atom block i / 32; TA = 16: two channel groups per warp)
                int c4, al;
                if constexpr (TA >= 32) {
                    c4 = i & 31;
                    al = (i >> 5) * 32 + lane;
                } else {
                    c4 = 2 * i + (lane >> 4);
                    al = lane & 15;
                }
                const int a = min(a0 + al, n_atoms - 1);
                const float4* x = reinterpret_cast<const float4*>(Xt + (int64_t)a * 4 * H);
                const float4 s = x[c4], vx = x[32 + c4], vy = x[64 + c4], vz = x[96 + c4];
                float* o = As + 4 * c4 * S::LD + al;
                o[0] = s.x; o[S::LD] = s.y; o[2 * S::LD] = s.z; o[3 * S::LD] = s.w;
                o += H * S::LD;
                o[0] = pair_distance(vx.x, vy.x, vz.x);   // |v| (:437)
                o[S::LD] = pair_distance(vx.y, vy.y, vz.y);
                o[2 * S::LD] = pair_distance(vx.z, vy.z, vz.z);
                o[3 * S::LD] = pair_distance(vx.w, vy.w, vz.w);
            }
            __syncthreads();
            f32x2 out[R][6];
            {
                const int tx = t & 31;
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(P + lo.c2 + g * H + 4 * tx);
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        out[i][2 * g] = b.x;
                        out[i][2 * g + 1] = b.y;
                    }
                }
            }
            two_gemms<TA, 2 * H, H3>(ws, total, W1, W2, As, Hs, t, [&](int ch, int al, float v) {
                const float z = v + __ldg(P + lo.c1 + ch);
                if (a0 + al < n_atoms) uz[(int64_t)(a0 + al) * H + ch] = z;
                return silu_f(z);
            }, out);
            // s' = s + ds, v' = v g1 + (M v) g2 (:452-468): channels 4 lane .. + 3
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int a = a0 + w * R + i;
                if (a >= n_atoms) break;
                const float4* x = reinterpret_cast<const float4*>(Xt + (int64_t)a * 4 * H) + lane;
                const float4 s = x[0], vx = x[32], vy = x[64], vz = x[96];
                const float4 ds = quad(out[i], 0), g1 = quad(out[i], 1), g2 = quad(out[i], 2);
                float4* u = reinterpret_cast<float4*>(ua + (int64_t)a * H3) + lane;
                u[0] = ds;
                u[32] = g1;
                u[64] = g2;
                auto vnew = [&](float px, float py, float pz, float pc, float a1, float a2, int r) {
                    return pc * a1 + (mix[3 * r] * px + mix[3 * r + 1] * py + mix[3 * r + 2] * pz) * a2;
                };
                float4 q[4];
                q[0] = make_float4(s.x + ds.x, vnew(vx.x, vy.x, vz.x, vx.x, g1.x, g2.x, 0),
                                   vnew(vx.x, vy.x, vz.x, vy.x, g1.x, g2.x, 1), vnew(vx.x, vy.x, vz.x, vz.x, g1.x, g2.x, 2));
                q[1] = make_float4(s.y + ds.y, vnew(vx.y, vy.y, vz.y, vx.y, g1.y, g2.y, 0),
                                   vnew(vx.y, vy.y, vz.y, vy.y, g1.y, g2.y, 1), vnew(vx.y, vy.y, vz.y, vz.y, g1.y, g2.y, 2));
                q[2] = make_float4(s.z + ds.z, vnew(vx.z, vy.z, vz.z, vx.z, g1.z, g2.z, 0),
                                   vnew(vx.z, vy.z, vz.z, vy.z, g1.z, g2.z, 1), vnew(vx.z, vy.z, vz.z, vz.z, g1.z, g2.z, 2));
                q[3] = make_float4(s.w + ds.w, vnew(vx.w, vy.w, vz.w, vx.w, g1.w, g2.w, 0),
                                   vnew(vx.w, vy.w, vz.w, vy.w, g1.w, g2.w, 1), vnew(vx.w, vy.w, vz.w, vz.w, g1.w, g2.w, 2));
                float4* o = reinterpret_cast<float4*>(Xout + (int64_t)a * 4 * H);
                if (out_layout == GATHER_QUADS) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) o[4 * lane + j] = q[j];
                } else {
                    o[lane] = make_float4(q[0].x, q[1].x, q[2].x, q[3].x);
                    o[32 + lane] = make_float4(q[0].y, q[1].y, q[2].y, q[3].y);
                    o[64 + lane] = make_float4(q[0].z, q[1].z, q[2].z, q[3].z);
                    o[96 + lane] = make_float4(q[0].w, q[1].w, q[2].w, q[3].w);
                }
            }
            if (*(volatile int*)ws.abort_flag) break;
            // (the next tile's inputs go to As, last read before the second GEMM's barriers)
        }
    }
    drain_stream(ws, t);
}

// Adjoint: abar = dE/d(ds, g1, g2) [atom][3H] -> zbar = (abar U2) silu'(uz)
// -> (cs, cn) = zbar U1 -> dE/dXt = (sb + cs, xb g1 + M^T xb g2 + cn v / |v|),
// in the quad layout the reverse edge kernel gathers from.
template <int TA>
__global__ void __launch_bounds__(UPT) upd32_bwd_kernel(const float* __restrict__ P, LayerOffsets lo,
                                                        const float* __restrict__ Xt, const float* __restrict__ uz,
                                                        const float* __restrict__ ua, const float* __restrict__ xbo,
                                                        int n_atoms, float* __restrict__ xtbar, Status* st) {
    using S = UpdShape<TA, H3>;
    using C = ChunkPlan<H3, 2 * H>;
    constexpr int R = S::R;
    extern __shared__ __align__(128) unsigned char smem[];
    float* As = reinterpret_cast<float*>(smem + S::OFF_A);
    float* Hs = reinterpret_cast<float*>(smem + S::OFF_H);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int ntiles = (n_atoms + TA - 1) / TA;
    const uint32_t total = (uint32_t)((ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * C::PER;
    const float *W1 = P + lo.u2, *W2 = P + lo.u1;
    WStream ws;
    init_stream(ws, smem + S::OFF_BAR, smem + S::OFF_RING, st, t);
    if (t == 0)
        for (int i = 0; i < STAGES; ++i) C::issue(ws, total, W1, W2);
    float mix[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) mix[i] = P[lo.mix + i];
    pdl_wait();
    pdl_trigger();
    if (st->code == 0) {
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int a0 = tile * TA;
            auto gates = [&](float b_x, float b_y, float b_z, float v_x, float v_y, float v_z, float& o1, float& o2) {
                o1 = b_x * v_x + b_y * v_y + b_z * v_z;
                o2 = b_x * (mix[0] * v_x + mix[1] * v_y + mix[2] * v_z) +
                     b_y * (mix[3] * v_x + mix[4] * v_y + mix[5] * v_z) +
                     b_z * (mix[6] * v_x + mix[7] * v_y + mix[8] * v_z);
            };
            for (int i = w; i < (TA >= 32 ? TA : 16); i += 8) {
                int c4, al;
                if constexpr (TA >= 32) {
                    c4 = i & 31;
                    al = (i >> 5) * 32 + lane;
                } else {
                    c4 = 2 * i + (lane >> 4);
                    al = lane & 15;
                }
                const int a = min(a0 + al, n_atoms - 1);
                const float4* x = reinterpret_cast<const float4*>(Xt + (int64_t)a * 4 * H);
                const float4* b = reinterpret_cast<const float4*>(xbo + (int64_t)a * 4 * H);
                const float4 vx = x[32 + c4], vy = x[64 + c4], vz = x[96 + c4];
                const float4 sb = b[c4], bx = b[32 + c4], by = b[64 + c4], bz = b[96 + c4];
                float4 g1, g2;
                gates(bx.x, by.x, bz.x, vx.x, vy.x, vz.x, g1.x, g2.x);
                gates(bx.y, by.y, bz.y, vx.y, vy.y, vz.y, g1.y, g2.y);
                gates(bx.z, by.z, bz.z, vx.z, vy.z, vz.z, g1.z, g2.z);
                gates(bx.w, by.w, bz.w, vx.w, vy.w, vz.w, g1.w, g2.w);
                float* o = As + 4 * c4 * S::LD + al;
                o[0] = sb.x; o[S::LD] = sb.y; o[2 * S::LD] = sb.z; o[3 * S::LD] = sb.w;
                o += H * S::LD;
                o[0] = g1.x; o[S::LD] = g1.y; o[2 * S::LD] = g1.z; o[3 * S::LD] = g1.w;
                o += H * S::LD;
                o[0] = g2.x; o[S::LD] = g2.y; o[2 * S::LD] = g2.z; o[3 * S::LD] = g2.w;
            }
            __syncthreads();
            f32x2 out[R][4];
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) out[i][j] = pack2(0.f, 0.f);
            two_gemms<TA, H3, 2 * H>(ws, total, W1, W2, As, Hs, t, [&](int ch, int al, float v) {
                return v * dsilu_f(__ldg(uz + (int64_t)min(a0 + al, n_atoms - 1) * H + ch));
            }, out);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int a = a0 + w * R + i;
                if (a >= n_atoms) break;
                const float4* x = reinterpret_cast<const float4*>(Xt + (int64_t)a * 4 * H) + lane;
                const float4* b = reinterpret_cast<const float4*>(xbo + (int64_t)a * 4 * H) + lane;
                const float4* u = reinterpret_cast<const float4*>(ua + (int64_t)a * H3) + lane;
                const float4 vx = x[32], vy = x[64], vz = x[96], sb = b[0], bx = b[32], by = b[64], bz = b[96];
                const float4 g1 = u[32], g2 = u[64], cs = quad(out[i], 0), cn = quad(out[i], 1);
                auto one = [&](float sbar, float b_x, float b_y, float b_z, float v_x, float v_y, float v_z, float a1,
                               float a2, float c_s, float c_n) {
                    const float nn = pair_distance(v_x, v_y, v_z);
                    const float sc = nn > 0.0f ? c_n / nn : 0.0f;   // d|v|/dv = v / |v|, 0 at v = 0
                    return make_float4(sbar + c_s,
                                       b_x * a1 + (mix[0] * b_x + mix[3] * b_y + mix[6] * b_z) * a2 + sc * v_x,
                                       b_y * a1 + (mix[1] * b_x + mix[4] * b_y + mix[7] * b_z) * a2 + sc * v_y,
                                       b_z * a1 + (mix[2] * b_x + mix[5] * b_y + mix[8] * b_z) * a2 + sc * v_z);
                };
                float4* o = reinterpret_cast<float4*>(xtbar + (int64_t)a * 4 * H) + 4 * lane;
                o[0] = one(sb.x, bx.x, by.x, bz.x, vx.x, vy.x, vz.x, g1.x, g2.x, cs.x, cn.x);
                o[1] = one(sb.y, bx.y, by.y, bz.y, vx.y, vy.y, vz.y, g1.y, g2.y, cs.y, cn.y);
                o[2] = one(sb.z, bx.z, by.z, bz.z, vx.z, vy.z, vz.z, g1.z, g2.z, cs.z, cn.z);
                o[3] = one(sb.w, bx.w, by.w, bz.w, vx.w, vy.w, vz.w, g1.w, g2.w, cs.w, cn.w);
            }
            if (*(volatile int*)ws.abort_flag) break;
        }
    }
    drain_stream(ws, t);
}

template <class K>
int set_attr(K* kernel, uint32_t bytes) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e == cudaSuccess ? MLFF_OK : cuda_status(e, "upd32 smem attribute");
}

template <int TA>
int launch_fwd_t(const float* P, const LayerOffsets& lo, const WsLayout& L, void* ws, int layer, cudaStream_t st) {
    using S = UpdShape<TA, 2 * H>;
    static std::once_flag once;
    static int err = MLFF_OK;
    std::call_once(once, [] { err = set_attr(upd32_fwd_kernel<TA>, S::SMEM); });
    if (err) return err;
    const int64_t NX = (int64_t)L.N * 4 * H;
    const int grid = std::min((L.N + TA - 1) / TA, num_sms() * (TA == 64 ? 1 : 2));
    MLFF_LAUNCH_PDL("upd32_fwd", upd32_fwd_kernel<TA>, grid, UPT, S::SMEM, st, P, lo,
                    ws_ptr<float>(ws, L.Xt) + layer * NX, L.N, ws_ptr<float>(ws, L.X) + (layer + 1) * NX,
                    layer + 1 < L.L ? L.gather : (int)GATHER_ROWS, ws_ptr<float>(ws, L.uz) + (int64_t)layer * L.N * H,
                    ws_ptr<float>(ws, L.ua) + (int64_t)layer * L.N * H3, ws_ptr<Status>(ws, L.status));
    return MLFF_OK;
}
template <int TA>
int launch_bwd_t(const float* P, const LayerOffsets& lo, const WsLayout& L, void* ws, int layer, const float* xbo,
                 float* xtbar, cudaStream_t st) {
    using S = UpdShape<TA, H3>;
    static std::once_flag once;
    static int err = MLFF_OK;
    std::call_once(once, [] { err = set_attr(upd32_bwd_kernel<TA>, S::SMEM); });
    if (err) return err;
    const int64_t NX = (int64_t)L.N * 4 * H;
    const int grid = std::min((L.N + TA - 1) / TA, num_sms() * (TA == 64 ? 1 : 2));
    MLFF_LAUNCH_PDL("upd32_bwd", upd32_bwd_kernel<TA>, grid, UPT, S::SMEM, st, P, lo,
                    ws_ptr<float>(ws, L.Xt) + layer * NX, ws_ptr<float>(ws, L.uz) + (int64_t)layer * L.N * H,
                    ws_ptr<float>(ws, L.ua) + (int64_t)layer * L.N * H3, xbo, L.N, xtbar, ws_ptr<Status>(ws, L.status));
    return MLFF_OK;
}

// Atoms per tile: 64 atoms use each weight read most; smaller tiles give
// small systems a CTA per SM.
int tile_atoms(int n_atoms) { return n_atoms > 64 * num_sms() ? 64 : n_atoms > 16 * 2 * num_sms() ? 32 : 16; }

}  // namespace

int launch_upd32_fwd(const float* P, const LayerOffsets& lo, const WsLayout& L, void* ws, int layer, cudaStream_t st) {
    ProfScope prof(PK_UPDATE_FWD, st);
    switch (tile_atoms(L.N)) {
        case 64: return launch_fwd_t<64>(P, lo, L, ws, layer, st);
        case 32: return launch_fwd_t<32>(P, lo, L, ws, layer, st);
        default: return launch_fwd_t<16>(P, lo, L, ws, layer, st);
    }
}
int launch_upd32_bwd(const float* P, const LayerOffsets& lo, const WsLayout& L, void* ws, int layer, const float* xbo,
                     float* xtbar, cudaStream_t st) {
    ProfScope prof(PK_UPDATE_BWD, st);
    switch (tile_atoms(L.N)) {
        case 64: return launch_bwd_t<64>(P, lo, L, ws, layer, xbo, xtbar, st);
        case 32: return launch_bwd_t<32>(P, lo, L, ws, layer, xbo, xtbar, st);
        default: return launch_bwd_t<16>(P, lo, L, ws, layer, xbo, xtbar, st);
    }
}

}  // namespace mlff
