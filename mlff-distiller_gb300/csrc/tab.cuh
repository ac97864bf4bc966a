// Tabulated edge filters (tab.cu): layout constants and launchers.
#pragma once
#include "common.cuh"
#include "workspace.h"

namespace mlff {

// The filter of a layer (Linear - SiLU - Linear of the radial basis,
// student_model.py:318-322,350) is a function of the distance alone.  Its
// table holds, for TAB_NI equal intervals of [0, cutoff] and every output
// channel, the degree-5 polynomial through the filter's float64 values at
// the interval's 6 Chebyshev nodes, in the local coordinate t in [-1, 1].
constexpr int TAB_NI = 96;
constexpr int TAB_DEG = 5;
constexpr int TAB_NC = TAB_DEG + 1;
// One interval of one 32-channel slice: the 18 coefficients of a channel's
// (phi_s, phi_v1, phi_v2) as four float4 rows and one float2 row of 32 lanes,
// so that a warp (lane = channel) reads them with conflict-free 16-byte
// loads.  phi_s and phi_v1 are interleaved (s0 a0 s1 a1 | s2 a2 s3 a3 | s4 a4
// s5 a5 | b0 b1 b2 b3 | b4 b5): the pairs are the operands of the two-wide
// FP32 fused multiply-adds.
constexpr int TAB_ROW = 32 * 3 * TAB_NC;            // floats: 576
constexpr int TAB_ROW_BYTES = TAB_ROW * 4;          // 2304, a multiple of 256
constexpr int TAB_SLICES = H / 32;
constexpr int64_t TAB_SLICE = (int64_t)TAB_NI * TAB_ROW;    // floats of a slice
constexpr int64_t TAB_LAYER = TAB_SLICES * TAB_SLICE;       // floats of a layer
// Accuracy of the table where it is worst (the ends of the intervals),
// relative 2-norms over all intervals and channels of (filter, derivative).
// TAB_TOL_D_FP32: as accurate as the FP32 evaluation; TAB_TOL_D_TC: as the
// split-FP16 evaluation (its filter derivative is off by about 1e-5).
constexpr double TAB_TOL_F = 2e-7, TAB_TOL_D_FP32 = 4e-6, TAB_TOL_D_TC = 1.2e-5;
constexpr int TAB_OK_TC = 1, TAB_OK_FP32 = 2;       // flag values (0: the table is not used)

// coefficient k of filter g (0 phi_s, 1 phi_v1, 2 phi_v2) of lane `lane`
__host__ __device__ constexpr int tab_index(int g, int k) { return g < 2 ? 2 * k + g : 2 * TAB_NC + k; }
__host__ __device__ constexpr int tab_off(int lane, int g, int k) {
    return tab_index(g, k) < 16 ? (tab_index(g, k) >> 2) * 128 + lane * 4 + (tab_index(g, k) & 3)
                                : 512 + lane * 2 + (tab_index(g, k) - 16);
}

// The network at the intervals' nodes (row interval * TAB_NC + node), for the
// weight gradients: per layer z = W1 e + b1, h = silu(z) and their
// d-derivatives z', h' [nodes][H], the basis rows e and e' [nodes][RMAX].
constexpr int64_t TAB_NODES = (int64_t)TAB_NI * TAB_NC;
constexpr int64_t TAB_NODE_LAYER = TAB_NODES * (4 * H + 2 * RMAX);

// training: edges per segment of the counting sort and per partial sum
constexpr int TT_SEG = 256, TT_CHUNK = 64;

// Edge records are read in chunks of 4, up to TREC_PAD past the last edge.
constexpr int TREC_PAD = 16;

// Quad layout of node features and adjoints in the table path: per atom, the
// 4 components of channel c at floats 4c .. 4c + 3.
__host__ __device__ constexpr int quad_off(int comp, int c) { return 4 * c + comp; }

int build_tables(const mlff_dims& d, float* packed, const PackedOffsets& po, cudaStream_t st);
void table_nodes(float* node, float* weight);   // Chebyshev nodes, 1 / prod_{m != j} (node_j - node_m)
int launch_records(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                   const WsLayout& L, void* ws, int path, cudaStream_t st);
// forward pass of the plain FP32 path; X [L + 1][N][4][H] component-major
int plain_forward(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                  const WsLayout& L, void* ws, float* X, cudaStream_t st);
// the same of the fused FP32 path, X in the tables' layout
int fused_fp32_forward(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                       const WsLayout& L, void* ws, cudaStream_t st);
// forward pass with the tables: records, X, Xt, uz, ua of every layer
int table_forward(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                  const WsLayout& L, void* ws, int path, cudaStream_t st);
// a training step's energies and forces (8: in a workspace without the gradient passes' arrays)
inline bool is_train_table(int path) {
    return path == MLFF_PATH_TRAIN_TABLE || path == MLFF_PATH_TRAIN_TABLE_FORWARD;
}
// training (train_tab.cu): offsets from p on, returns the end: the arrays of
// the forward pass by pairs, and those that the gradient passes add
size_t train_forward_workspace(WsLayout& L, size_t p);
size_t train_table_workspace(WsLayout& L, const mlff_dims& d, size_t p);
struct GradCtx;
int run_train_table(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                    const WsLayout& L, void* ws, double* energy, cudaStream_t st, const GradCtx& grad);
int run_train_table_tangent(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                            const WsLayout& L, void* ws, cudaStream_t st, const GradCtx& grad, const float* G,
                            const double* S);
int read_table_flag(const float* packed, const PackedOffsets& po, int32_t* flag, cudaStream_t st);

}  // namespace mlff
