// Per-module entry points: the reference's PaiNNMessage and PaiNNUpdate
// blocks (src/mlff_distiller/models/student_model.py:297-470) evaluated on
// their own, for any hidden width and any number of radial basis functions,
// with their reverse passes (input and parameter gradients).
//
// These serve callers that use the blocks outside StudentForceField (the
// reference's unit tests build a PaiNNInteraction of width 64 and call it
// directly).  They follow the reference's per-op graph in FP32 -- filter
// GEMMs in FP32 (gemm.cu), messages scattered with float atomics as
// index_add_ does on a GPU -- and are not the fused hot path.  Edge indices
// come from the caller: an out-of-range index is reported through the
// status word (MLFF_ERR_INVALID, the edge's position) and every later kernel
// of the call returns without work, so nothing is read or written out of
// bounds (the outputs then hold the residual copies only).
#include <algorithm>
#include "common.cuh"
#include "gemm.cuh"
#include "workspace.h"

namespace mlff {

namespace {

int plain_sgemm(int mode, const float* A, const float* B, const float* bias, float* C, float* C2, const float* Z,
                int64_t M, int N, int K, const Status* st, cudaStream_t s) {
    return gemm_nn(mode, A, B, bias, C, C2, Z, M, nullptr, N, K, st, s);
}


constexpr int MOD_BLOCKS_MAX = 152 * 8;

inline int grid_for(int64_t n, int threads = 256) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, MOD_BLOCKS_MAX));
}

// Byte layout of a module workspace: a status word, then float arrays.
struct ModLayout {
    size_t st = 0;
    size_t a[16] = {};
    size_t total = 0;
};
inline ModLayout mod_layout(const int64_t* sizes, int n) {
    ModLayout L;
    size_t p = 0;
    auto take = [&](size_t bytes) {
        size_t r = p;
        p += (bytes + 255) & ~size_t(255);
        return r;
    };
    L.st = take(sizeof(Status));
    for (int i = 0; i < n; ++i) L.a[i] = take(sizeof(float) * (size_t)sizes[i]);
    L.total = p;
    return L;
}

// message workspace: w1t [R][H], w2t [H][3H], z, h [E][H], f [E][3H];
// reverse pass: gf [E][3H], gz [E][H], scratch of the weight-gradient sums
inline ModLayout msg_layout(int64_t H, int64_t R, int64_t E, bool bwd) {
    const int64_t part = (int64_t)std::max(gemm_tn_floats(3 * H, H), gemm_tn_floats(H, R));
    const int64_t s[8] = {R * H, H * 3 * H, E * H, E * H, E * 3 * H, E * 3 * H, E * H, part};
    return mod_layout(s, bwd ? 8 : 5);
}
// update workspace: u1t [2H][H], u2t [H][3H], comb [N][2H], z, h [N][H],
// a [N][3H]; reverse pass: ga [N][3H], gz [N][H], gcomb [N][2H], scratch of
// the weight-gradient sums, gmix [MIX_BLOCKS][9]
constexpr int MIX_BLOCKS = 256;
inline ModLayout upd_layout(int64_t H, int64_t N, bool bwd) {
    const int64_t part = (int64_t)std::max(gemm_tn_floats(3 * H, H), gemm_tn_floats(H, 2 * H));
    const int64_t s[11] = {2 * H * H, H * 3 * H, N * 2 * H, N * H, N * H, N * 3 * H,
                           N * 3 * H, N * H, N * 2 * H, part, MIX_BLOCKS * 9};
    return mod_layout(s, bwd ? 11 : 6);
}

template <typename T>
inline T* at(void* ws, size_t off) {
    return reinterpret_cast<T*>(static_cast<char*>(ws) + off);
}

// out[c][r] = in[r][c]
__global__ void mod_transpose_kernel(const float* __restrict__ in, float* __restrict__ out, int64_t rows, int64_t cols,
                                     const Status* st) {
    if (st->code != 0) return;
    const int64_t n = rows * cols;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / cols, c = i % cols;
        out[c * rows + r] = in[i];
    }
}

__global__ void mod_check_edges_kernel(const int64_t* __restrict__ ei, int64_t E, int32_t N, Status* st) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = ei[e], d = ei[E + e];
        if (s < 0 || s >= N || d < 0 || d >= N) set_status(st, MLFF_ERR_INVALID, (int)std::min<int64_t>(e, INT32_MAX));
    }
}

// V consecutive floats of a row: one 16-byte access and one 16-byte atomic
// when the rows allow it (V = 4: H a multiple of 4, every base 16-byte
// aligned), single floats otherwise.
template <int V>
struct Vec;
template <>
struct Vec<1> {
    float x[1];
    static __device__ __forceinline__ Vec load(const float* p) { return {{*p}}; }
    __device__ __forceinline__ void store(float* p) const { *p = x[0]; }
    __device__ __forceinline__ void add_to(float* p) const { atomicAdd(p, x[0]); }
};
template <>
struct Vec<4> {
    float x[4];
    static __device__ __forceinline__ Vec load(const float* p) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        return {{v.x, v.y, v.z, v.w}};
    }
    __device__ __forceinline__ void store(float* p) const {
        *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
    }
    __device__ __forceinline__ void add_to(float* p) const {
        atomicAdd(reinterpret_cast<float4*>(p), make_float4(x[0], x[1], x[2], x[3]));
    }
};

// scalar_out[dst] += s[src] * phi_s;  vector_out[dst][i] += v[src][i] * phi_v1
// + u[i] * phi_v2   (index_add_, student_model.py:359-385), thread per (edge,
// V channels).  Bound by the atomics: 16-byte ones issue a quarter as many.
template <int V>
__global__ void __launch_bounds__(256) msg_scatter_kernel(const float* __restrict__ s, const float* __restrict__ v,
                                                          const int64_t* __restrict__ ei,
                                                          const float* __restrict__ evec, const float* __restrict__ f,
                                                          int64_t E, int H, float* __restrict__ s_out,
                                                          float* __restrict__ v_out, const Status* st) {
    if (st->code != 0) return;
    using W = Vec<V>;
    const int per = H / V;
    const int64_t n = E * per;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = i / per;
        const int k = (int)(i % per) * V;
        const int64_t b = ei[e], a = ei[E + e];
        const float* fe = f + e * 3 * H + k;
        const W fs = W::load(fe), f1 = W::load(fe + H), f2 = W::load(fe + 2 * H);
        W m = W::load(s + b * H + k);
#pragma unroll
        for (int j = 0; j < V; ++j) m.x[j] *= fs.x[j];
        m.add_to(s_out + a * H + k);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            W x = W::load(v + (b * 3 + q) * H + k);
            const float u = evec[e * 3 + q];
#pragma unroll
            for (int j = 0; j < V; ++j) x.x[j] = x.x[j] * f1.x[j] + u * f2.x[j];
            x.add_to(v_out + (a * 3 + q) * H + k);
        }
    }
}

// reverse of the scatter: filter adjoint gf [E][3H], the gathered adjoints
// of the sender features (grad_s, grad_v hold the residual part) and
// grad_u[e][q] = sum_k gv[dst][q][k] phi_v2[e][k].  One warp per edge, V
// channels per lane and turn, so the channel sums stay in the warp and every
// row is read once.
template <int V>
__global__ void __launch_bounds__(256) msg_scatter_bwd_kernel(
    const float* __restrict__ s, const float* __restrict__ v, const int64_t* __restrict__ ei,
    const float* __restrict__ evec, const float* __restrict__ f, const float* __restrict__ gs,
    const float* __restrict__ gv, int64_t E, int H, float* __restrict__ gf, float* __restrict__ grad_s,
    float* __restrict__ grad_v, float* __restrict__ gu, const Status* st) {
    if (st->code != 0) return;
    using W = Vec<V>;
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < E; e += nw) {
        const int64_t b = ei[e], a = ei[E + e];
        const float u[3] = {evec[e * 3], evec[e * 3 + 1], evec[e * 3 + 2]};
        float du[3] = {0.f, 0.f, 0.f};
        for (int k = lane * V; k < H; k += 32 * V) {
            const float* fe = f + e * 3 * H + k;
            const W fs = W::load(fe), f1 = W::load(fe + H), f2 = W::load(fe + 2 * H);
            const W ga = W::load(gs + a * H + k), sb = W::load(s + b * H + k);
            W t0, t1, g1{}, g2{};
#pragma unroll
            for (int j = 0; j < V; ++j) {
                t0.x[j] = ga.x[j] * sb.x[j];
                t1.x[j] = ga.x[j] * fs.x[j];
            }
            float* g = gf + e * 3 * H + k;
            t0.store(g);
            t1.add_to(grad_s + b * H + k);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const W gva = W::load(gv + (a * 3 + q) * H + k), vb = W::load(v + (b * 3 + q) * H + k);
                W d;
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    g1.x[j] = fmaf(gva.x[j], vb.x[j], g1.x[j]);
                    g2.x[j] = fmaf(gva.x[j], u[q], g2.x[j]);
                    d.x[j] = gva.x[j] * f1.x[j];
                    du[q] = fmaf(gva.x[j], f2.x[j], du[q]);
                }
                d.add_to(grad_v + (b * 3 + q) * H + k);
            }
            g1.store(g + H);
            g2.store(g + 2 * H);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < 3; ++q) du[q] += __shfl_xor_sync(0xffffffffu, du[q], o);
        if (lane < 3) gu[e * 3 + lane] = lane == 0 ? du[0] : lane == 1 ? du[1] : du[2];
    }
}

inline bool rows16(int64_t H, std::initializer_list<const void*> ps) {
    if (H % 4) return false;
    for (const void* p : ps)
        if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

// comb = [s, |v|] (norm over xyz, student_model.py:437-440)
__global__ void upd_comb_kernel(const float* __restrict__ s, const float* __restrict__ v, int64_t N, int H,
                                float* __restrict__ comb, const Status* st) {
    if (st->code != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * H; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / H;
        const int k = (int)(i % H);
        const float x = v[(n * 3) * H + k], y = v[(n * 3 + 1) * H + k], z = v[(n * 3 + 2) * H + k];
        comb[n * 2 * H + k] = s[i];
        comb[n * 2 * H + H + k] = sqrtf(x * x + y * y + z * z);
    }
}

// s_out = s + a_s;  v_out = v g1 + (M v) g2, M over xyz (:452-468)
__global__ void upd_finish_kernel(const float* __restrict__ s, const float* __restrict__ v,
                                  const float* __restrict__ a, const float* __restrict__ mix, int64_t N, int H,
                                  float* __restrict__ s_out, float* __restrict__ v_out, const Status* st) {
    if (st->code != 0) return;
    float M[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) M[j] = mix[j];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * H; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / H;
        const int k = (int)(i % H);
        const float* an = a + n * 3 * H;
        s_out[i] = s[i] + an[k];
        const float g1 = an[H + k], g2 = an[2 * H + k];
        float vv[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) vv[q] = v[(n * 3 + q) * H + k];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float mixed = M[3 * q] * vv[0] + M[3 * q + 1] * vv[1] + M[3 * q + 2] * vv[2];
            v_out[(n * 3 + q) * H + k] = vv[q] * g1 + mixed * g2;
        }
    }
}

// reverse of upd_finish: ga [N][3H]; grad_s = gs; grad_v (direct part)
__global__ void upd_finish_bwd_kernel(const float* __restrict__ v, const float* __restrict__ a,
                                      const float* __restrict__ mix, const float* __restrict__ gs,
                                      const float* __restrict__ gv, int64_t N, int H, float* __restrict__ ga,
                                      float* __restrict__ grad_s, float* __restrict__ grad_v, const Status* st) {
    if (st->code != 0) return;
    float M[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) M[j] = mix[j];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * H; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / H;
        const int k = (int)(i % H);
        const float* an = a + n * 3 * H;
        const float g1 = an[H + k], g2 = an[2 * H + k];
        float vv[3], gg[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            vv[q] = v[(n * 3 + q) * H + k];
            gg[q] = gv[(n * 3 + q) * H + k];
        }
        float dg1 = 0.f, dg2 = 0.f;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float mixed = M[3 * q] * vv[0] + M[3 * q + 1] * vv[1] + M[3 * q + 2] * vv[2];
            dg1 = fmaf(gg[q], vv[q], dg1);
            dg2 = fmaf(gg[q], mixed, dg2);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
            grad_v[(n * 3 + j) * H + k] = gg[j] * g1 + g2 * (M[j] * gg[0] + M[3 + j] * gg[1] + M[6 + j] * gg[2]);
        grad_s[i] = gs[i];
        float* g = ga + n * 3 * H;
        g[k] = gs[i];
        g[H + k] = dg1;
        g[2 * H + k] = dg2;
    }
}

// adds the combined-input adjoint: grad_s += gcomb[:, :H]; grad_v += gcomb[:,
// H:] v / |v| (0 where |v| = 0, the subgradient torch.norm uses)
__global__ void upd_comb_bwd_kernel(const float* __restrict__ v, const float* __restrict__ comb,
                                    const float* __restrict__ gcomb, int64_t N, int H, float* __restrict__ grad_s,
                                    float* __restrict__ grad_v, const Status* st) {
    if (st->code != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * H; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / H;
        const int k = (int)(i % H);
        grad_s[i] += gcomb[n * 2 * H + k];
        const float nrm = comb[n * 2 * H + H + k];
        if (nrm > 0.f) {
            const float sc = gcomb[n * 2 * H + H + k] / nrm;
#pragma unroll
            for (int q = 0; q < 3; ++q) grad_v[(n * 3 + q) * H + k] += sc * v[(n * 3 + q) * H + k];
        }
    }
}

// grad_M[q][j] = sum_{n,k} gv[n][q][k] g2[n][k] v[n][j][k]: per-block partials, fixed order
__global__ void __launch_bounds__(256) upd_mix_bwd_kernel(const float* __restrict__ v, const float* __restrict__ a,
                                                          const float* __restrict__ gv, int64_t N, int H,
                                                          float* __restrict__ part, const Status* st) {
    __shared__ float red[9][256];
    if (st->code != 0) return;
    float acc[9] = {};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N * H; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / H;
        const int k = (int)(i % H);
        const float g2 = a[n * 3 * H + 2 * H + k];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float gq = gv[(n * 3 + q) * H + k] * g2;
#pragma unroll
            for (int j = 0; j < 3; ++j) acc[3 * q + j] = fmaf(gq, v[(n * 3 + j) * H + k], acc[3 * q + j]);
        }
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) red[j][threadIdx.x] = acc[j];
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
#pragma unroll
            for (int j = 0; j < 9; ++j) red[j][threadIdx.x] += red[j][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x < 9) part[blockIdx.x * 9 + threadIdx.x] = red[threadIdx.x][0];
}

__global__ void upd_mix_sum_kernel(const float* __restrict__ part, int blocks, float* __restrict__ out,
                                   const Status* st) {
    if (st->code != 0) return;
    if (threadIdx.x < 9) {
        float s = 0.f;
        for (int b = 0; b < blocks; ++b) s += part[b * 9 + threadIdx.x];
        out[threadIdx.x] = s;
    }
}

int check_mod(int32_t H, int32_t R, int64_t rows) {
    if (H < 1 || H > 4096 || R < 0 || R > 4096 || rows < 0) {
        set_error("module shape outside limits (hidden %d, n_rbf %d, rows %lld)", H, R, (long long)rows);
        return MLFF_ERR_INVALID;
    }
    return MLFF_OK;
}

#define MOD_LAUNCH(kernel, n, st, ...)                                              \
    do {                                                                            \
        kernel<<<grid_for(n), 256, 0, st>>>(__VA_ARGS__);                           \
        MLFF_LAUNCH_CHECK(#kernel);                                                 \
    } while (0)

}  // namespace
}  // namespace mlff

using namespace mlff;

extern "C" {

size_t mlff_painn_message_workspace_size(int32_t hidden, int32_t n_rbf, int64_t n_edges, int32_t with_backward) {
    if (check_mod(hidden, n_rbf, n_edges)) return 0;
    return msg_layout(hidden, n_rbf, n_edges, with_backward != 0).total;
}

int mlff_painn_message(int32_t hidden, int32_t n_rbf, int32_t n_atoms, int64_t n_edges, const float* scalar,
                       const float* vector, const int64_t* edge_index, const float* edge_rbf,
                       const float* edge_vector, const float* w1, const float* b1, const float* w2, const float* b2,
                       float* scalar_out, float* vector_out, int32_t* status, void* workspace,
                       size_t workspace_bytes, mlff_stream_t stream) {
    int r = check_mod(hidden, n_rbf, n_edges);
    if (r) return r;
    if (n_atoms < 1 || !scalar || !vector || !w1 || !b1 || !w2 || !b2 || !scalar_out || !vector_out || !status ||
        !workspace || (n_edges > 0 && (!edge_index || !edge_rbf || !edge_vector))) {
        set_error("painn_message: missing argument");
        return MLFF_ERR_INVALID;
    }
    const int64_t H = hidden, R = n_rbf, E = n_edges, N = n_atoms;
    const ModLayout L = msg_layout(H, R, E, false);
    if (workspace_bytes < L.total) {
        set_error("workspace %zu bytes < %zu needed", workspace_bytes, L.total);
        return MLFF_ERR_WORKSPACE;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Status* sw = at<Status>(workspace, L.st);
    MLFF_CUDA(cudaMemsetAsync(sw, 0, sizeof(Status), st));
    MLFF_CUDA(cudaMemcpyAsync(scalar_out, scalar, sizeof(float) * N * H, cudaMemcpyDeviceToDevice, st));
    MLFF_CUDA(cudaMemcpyAsync(vector_out, vector, sizeof(float) * N * 3 * H, cudaMemcpyDeviceToDevice, st));
    if (E > 0) {
        float *w1t = at<float>(workspace, L.a[0]), *w2t = at<float>(workspace, L.a[1]);
        float *z = at<float>(workspace, L.a[2]), *h = at<float>(workspace, L.a[3]), *f = at<float>(workspace, L.a[4]);
        MOD_LAUNCH(mod_check_edges_kernel, E, st, edge_index, E, n_atoms, sw);
        MOD_LAUNCH(mod_transpose_kernel, H * R, st, w1, w1t, H, R, sw);
        MOD_LAUNCH(mod_transpose_kernel, 3 * H * H, st, w2, w2t, 3 * H, H, sw);
        // filter = Linear(R, H) - SiLU - Linear(H, 3H)  (:318-322, :350)
        if ((r = plain_sgemm(1, edge_rbf, w1t, b1, z, h, nullptr, E, (int)H, (int)R, sw, st))) return r;
        if ((r = plain_sgemm(0, h, w2t, b2, f, nullptr, nullptr, E, (int)(3 * H), (int)H, sw, st))) return r;
        if (rows16(H, {scalar, vector, scalar_out, vector_out}))
            MOD_LAUNCH(msg_scatter_kernel<4>, E * H / 4, st, scalar, vector, edge_index, edge_vector, f, E, (int)H,
                       scalar_out, vector_out, sw);
        else
            MOD_LAUNCH(msg_scatter_kernel<1>, E * H, st, scalar, vector, edge_index, edge_vector, f, E, (int)H,
                       scalar_out, vector_out, sw);
    }
    MLFF_CUDA(cudaMemcpyAsync(status, sw, 4 * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    return MLFF_OK;
}

int mlff_painn_message_backward(int32_t hidden, int32_t n_rbf, int32_t n_atoms, int64_t n_edges, const float* scalar,
                                const float* vector, const int64_t* edge_index, const float* edge_rbf,
                                const float* edge_vector, const float* w1, const float* b1, const float* w2,
                                const float* b2, const float* grad_scalar_out, const float* grad_vector_out,
                                float* grad_scalar, float* grad_vector, float* grad_rbf, float* grad_edge_vector,
                                float* grad_w1, float* grad_b1, float* grad_w2, float* grad_b2, int32_t* status,
                                void* workspace, size_t workspace_bytes, mlff_stream_t stream) {
    int r = check_mod(hidden, n_rbf, n_edges);
    if (r) return r;
    if (n_atoms < 1 || !scalar || !vector || !w1 || !b1 || !w2 || !b2 || !grad_scalar_out || !grad_vector_out ||
        !grad_scalar || !grad_vector || !grad_w1 || !grad_b1 || !grad_w2 || !grad_b2 || !status || !workspace ||
        (n_edges > 0 && (!edge_index || !edge_rbf || !edge_vector || !grad_rbf || !grad_edge_vector))) {
        set_error("painn_message_backward: missing argument");
        return MLFF_ERR_INVALID;
    }
    const int64_t H = hidden, R = n_rbf, E = n_edges, N = n_atoms;
    const ModLayout L = msg_layout(H, R, E, true);
    if (workspace_bytes < L.total) {
        set_error("workspace %zu bytes < %zu needed (with_backward)", workspace_bytes, L.total);
        return MLFF_ERR_WORKSPACE;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Status* sw = at<Status>(workspace, L.st);
    MLFF_CUDA(cudaMemsetAsync(sw, 0, sizeof(Status), st));
    // residual part of the feature adjoints
    MLFF_CUDA(cudaMemcpyAsync(grad_scalar, grad_scalar_out, sizeof(float) * N * H, cudaMemcpyDeviceToDevice, st));
    MLFF_CUDA(cudaMemcpyAsync(grad_vector, grad_vector_out, sizeof(float) * N * 3 * H, cudaMemcpyDeviceToDevice, st));
    if (E == 0) {
        MLFF_CUDA(cudaMemsetAsync(grad_w1, 0, sizeof(float) * H * R, st));
        MLFF_CUDA(cudaMemsetAsync(grad_b1, 0, sizeof(float) * H, st));
        MLFF_CUDA(cudaMemsetAsync(grad_w2, 0, sizeof(float) * 3 * H * H, st));
        MLFF_CUDA(cudaMemsetAsync(grad_b2, 0, sizeof(float) * 3 * H, st));
        MLFF_CUDA(cudaMemcpyAsync(status, sw, 4 * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
        return MLFF_OK;
    }
    float *w1t = at<float>(workspace, L.a[0]), *w2t = at<float>(workspace, L.a[1]);
    float *z = at<float>(workspace, L.a[2]), *h = at<float>(workspace, L.a[3]), *f = at<float>(workspace, L.a[4]);
    float *gf = at<float>(workspace, L.a[5]), *gz = at<float>(workspace, L.a[6]);
    float* part = at<float>(workspace, L.a[7]);
    MOD_LAUNCH(mod_check_edges_kernel, E, st, edge_index, E, n_atoms, sw);
    // the filter of the forward pass, recomputed (no activation is kept between the calls)
    MOD_LAUNCH(mod_transpose_kernel, H * R, st, w1, w1t, H, R, sw);
    MOD_LAUNCH(mod_transpose_kernel, 3 * H * H, st, w2, w2t, 3 * H, H, sw);
    if ((r = plain_sgemm(1, edge_rbf, w1t, b1, z, h, nullptr, E, (int)H, (int)R, sw, st))) return r;
    if ((r = plain_sgemm(0, h, w2t, b2, f, nullptr, nullptr, E, (int)(3 * H), (int)H, sw, st))) return r;
    // filter adjoint and the gathered feature adjoints; unit-vector adjoint
    if (rows16(H, {scalar, vector, grad_scalar_out, grad_vector_out, grad_scalar, grad_vector}))
        MOD_LAUNCH(msg_scatter_bwd_kernel<4>, E * 32, st, scalar, vector, edge_index, edge_vector, f, grad_scalar_out,
                   grad_vector_out, E, (int)H, gf, grad_scalar, grad_vector, grad_edge_vector, sw);
    else
        MOD_LAUNCH(msg_scatter_bwd_kernel<1>, E * 32, st, scalar, vector, edge_index, edge_vector, f, grad_scalar_out,
                   grad_vector_out, E, (int)H, gf, grad_scalar, grad_vector, grad_edge_vector, sw);
    // through the filter MLP: gz = (gf W2) silu'(z), grad_rbf = gz W1
    if ((r = plain_sgemm(2, gf, w2, nullptr, gz, nullptr, z, E, (int)H, (int)(3 * H), sw, st))) return r;
    if ((r = plain_sgemm(0, gz, w1, nullptr, grad_rbf, nullptr, nullptr, E, (int)R, (int)H, sw, st))) return r;
    // parameter gradients: W2 = gf^T h, W1 = gz^T rbf, biases = column sums
    if ((r = gemm_tn({gf, h}, (int)(3 * H), (int)H, (int)(3 * H), (int)H, E, grad_w2, grad_b2, false, part, sw, st)))
        return r;
    if ((r = gemm_tn({gz, edge_rbf}, (int)H, (int)R, (int)H, (int)R, E, grad_w1, grad_b1, false, part, sw, st)))
        return r;
    MLFF_CUDA(cudaMemcpyAsync(status, sw, 4 * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    return MLFF_OK;
}

size_t mlff_painn_update_workspace_size(int32_t hidden, int32_t n_atoms, int32_t with_backward) {
    if (check_mod(hidden, 0, n_atoms)) return 0;
    return upd_layout(hidden, n_atoms, with_backward != 0).total;
}

int mlff_painn_update(int32_t hidden, int32_t n_atoms, const float* scalar, const float* vector, const float* w1,
                      const float* b1, const float* w2, const float* b2, const float* mixing, float* scalar_out,
                      float* vector_out, void* workspace, size_t workspace_bytes, mlff_stream_t stream) {
    int r = check_mod(hidden, 0, n_atoms);
    if (r) return r;
    if (n_atoms < 1 || !scalar || !vector || !w1 || !b1 || !w2 || !b2 || !mixing || !scalar_out || !vector_out ||
        !workspace) {
        set_error("painn_update: missing argument");
        return MLFF_ERR_INVALID;
    }
    const int64_t H = hidden, N = n_atoms;
    const ModLayout L = upd_layout(H, N, false);
    if (workspace_bytes < L.total) {
        set_error("workspace %zu bytes < %zu needed", workspace_bytes, L.total);
        return MLFF_ERR_WORKSPACE;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Status* sw = at<Status>(workspace, L.st);
    MLFF_CUDA(cudaMemsetAsync(sw, 0, sizeof(Status), st));
    float *u1t = at<float>(workspace, L.a[0]), *u2t = at<float>(workspace, L.a[1]);
    float *comb = at<float>(workspace, L.a[2]), *z = at<float>(workspace, L.a[3]);
    float *h = at<float>(workspace, L.a[4]), *a = at<float>(workspace, L.a[5]);
    MOD_LAUNCH(mod_transpose_kernel, 2 * H * H, st, w1, u1t, H, 2 * H, sw);
    MOD_LAUNCH(mod_transpose_kernel, 3 * H * H, st, w2, u2t, 3 * H, H, sw);
    MOD_LAUNCH(upd_comb_kernel, N * H, st, scalar, vector, N, (int)H, comb, sw);
    // update_mlp = Linear(2H, H) - SiLU - Linear(H, 3H)  (:440-444)
    if ((r = plain_sgemm(1, comb, u1t, b1, z, h, nullptr, N, (int)H, (int)(2 * H), sw, st))) return r;
    if ((r = plain_sgemm(0, h, u2t, b2, a, nullptr, nullptr, N, (int)(3 * H), (int)H, sw, st))) return r;
    MOD_LAUNCH(upd_finish_kernel, N * H, st, scalar, vector, a, mixing, N, (int)H, scalar_out, vector_out, sw);
    return MLFF_OK;
}

int mlff_painn_update_backward(int32_t hidden, int32_t n_atoms, const float* scalar, const float* vector,
                               const float* w1, const float* b1, const float* w2, const float* b2,
                               const float* mixing, const float* grad_scalar_out, const float* grad_vector_out,
                               float* grad_scalar, float* grad_vector, float* grad_w1, float* grad_b1,
                               float* grad_w2, float* grad_b2, float* grad_mixing, void* workspace,
                               size_t workspace_bytes, mlff_stream_t stream) {
    int r = check_mod(hidden, 0, n_atoms);
    if (r) return r;
    if (n_atoms < 1 || !scalar || !vector || !w1 || !b1 || !w2 || !b2 || !mixing || !grad_scalar_out ||
        !grad_vector_out || !grad_scalar || !grad_vector || !grad_w1 || !grad_b1 || !grad_w2 || !grad_b2 ||
        !grad_mixing || !workspace) {
        set_error("painn_update_backward: missing argument");
        return MLFF_ERR_INVALID;
    }
    const int64_t H = hidden, N = n_atoms;
    const ModLayout L = upd_layout(H, N, true);
    if (workspace_bytes < L.total) {
        set_error("workspace %zu bytes < %zu needed (with_backward)", workspace_bytes, L.total);
        return MLFF_ERR_WORKSPACE;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Status* sw = at<Status>(workspace, L.st);
    MLFF_CUDA(cudaMemsetAsync(sw, 0, sizeof(Status), st));
    float *u1t = at<float>(workspace, L.a[0]), *u2t = at<float>(workspace, L.a[1]);
    float *comb = at<float>(workspace, L.a[2]), *z = at<float>(workspace, L.a[3]);
    float *h = at<float>(workspace, L.a[4]), *a = at<float>(workspace, L.a[5]);
    float *ga = at<float>(workspace, L.a[6]), *gz = at<float>(workspace, L.a[7]);
    float *gcomb = at<float>(workspace, L.a[8]), *part = at<float>(workspace, L.a[9]);
    float* gmix = at<float>(workspace, L.a[10]);
    // the forward pass, recomputed
    MOD_LAUNCH(mod_transpose_kernel, 2 * H * H, st, w1, u1t, H, 2 * H, sw);
    MOD_LAUNCH(mod_transpose_kernel, 3 * H * H, st, w2, u2t, 3 * H, H, sw);
    MOD_LAUNCH(upd_comb_kernel, N * H, st, scalar, vector, N, (int)H, comb, sw);
    if ((r = plain_sgemm(1, comb, u1t, b1, z, h, nullptr, N, (int)H, (int)(2 * H), sw, st))) return r;
    if ((r = plain_sgemm(0, h, u2t, b2, a, nullptr, nullptr, N, (int)(3 * H), (int)H, sw, st))) return r;
    // gates and mixing; through the MLP; the combined input's adjoint
    MOD_LAUNCH(upd_finish_bwd_kernel, N * H, st, vector, a, mixing, grad_scalar_out, grad_vector_out, N, (int)H, ga,
               grad_scalar, grad_vector, sw);
    upd_mix_bwd_kernel<<<MIX_BLOCKS, 256, 0, st>>>(vector, a, grad_vector_out, N, (int)H, gmix, sw);
    MLFF_LAUNCH_CHECK("upd_mix_bwd_kernel");
    upd_mix_sum_kernel<<<1, 32, 0, st>>>(gmix, MIX_BLOCKS, grad_mixing, sw);
    MLFF_LAUNCH_CHECK("upd_mix_sum_kernel");
    if ((r = plain_sgemm(2, ga, w2, nullptr, gz, nullptr, z, N, (int)H, (int)(3 * H), sw, st))) return r;
    if ((r = plain_sgemm(0, gz, w1, nullptr, gcomb, nullptr, nullptr, N, (int)(2 * H), (int)H, sw, st))) return r;
    MOD_LAUNCH(upd_comb_bwd_kernel, N * H, st, vector, comb, gcomb, N, (int)H, grad_scalar, grad_vector, sw);
    // parameter gradients
    if ((r = gemm_tn({ga, h}, (int)(3 * H), (int)H, (int)(3 * H), (int)H, N, grad_w2, grad_b2, false, part, sw, st)))
        return r;
    if ((r = gemm_tn({gz, comb}, (int)H, (int)(2 * H), (int)H, (int)(2 * H), N, grad_w1, grad_b1, false, part, sw, st)))
        return r;
    return MLFF_OK;
}

}  // extern "C"
