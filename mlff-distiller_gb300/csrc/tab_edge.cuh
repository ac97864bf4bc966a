// Device helpers of the table path's edge kernels.
#pragma once
#include <algorithm>
#include <type_traits>
#include "f32x2.cuh"
#include "tab.cuh"
#include "tc_layout.cuh"
#include "tc_ptx.cuh"

namespace mlff {

// dt/dd of the table's local coordinate, as the kernels use it in FP32; the
// build places its nodes with the same rounded value.
__host__ __device__ inline float tab_scale(float cutoff) { return (float)(2.0 * TAB_NI / (double)cutoff); }

// A condition that is the same in every lane, as a vote: the branch on it
// needs no divergence bookkeeping and is not turned into predicated code.
__device__ __forceinline__ bool uni(bool p) { return __any_sync(0xffffffffu, p); }

// f(integral_constant<int, r>) for a warp-uniform r < G, so that
// per-receiver sums stay in registers
template <int G, int BASE = 0, class F>
__device__ __forceinline__ void tab_switch(int r, F&& f) {
    if constexpr (G == 1) {
        f(std::integral_constant<int, BASE>{});
    } else {
        if (uni((r & (G / 2)) != 0)) tab_switch<G / 2, BASE + G / 2>(r, f);
        else tab_switch<G / 2, BASE>(r, f);
    }
}

// Sums of 16 per-lane values over the warp's lanes with 16 shuffles
// (reduce-scatter): lanes 2 i and 2 i + 1 return the sum of v[i].
__device__ __forceinline__ float reduce16(const float (&v)[16], int lane) {
    float a[8], b[4], c[2];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        a[j] = (h16 ? v[j + 8] : v[j]) + __shfl_xor_sync(0xffffffffu, h16 ? v[j] : v[j + 8], 16);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        b[j] = (h8 ? a[j + 4] : a[j]) + __shfl_xor_sync(0xffffffffu, h8 ? a[j] : a[j + 4], 8);
#pragma unroll
    for (int j = 0; j < 2; ++j)
        c[j] = (h4 ? b[j + 2] : b[j]) + __shfl_xor_sync(0xffffffffu, h4 ? b[j] : b[j + 2], 4);
    float s = (h2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h2 ? c[0] : c[1], 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// ------------------------------------------------------------ edge records
// (a load that every lane makes of the same bytes costs the shared-memory
// pipe a cycle per word, so an edge reads its first six words and a gather
// the sender alone)
struct __align__(16) TabRec {
    float t, t2;      // local coordinate, twice (an operand pair)
    float uy, uz;
    float ux;
    int32_t off;      // byte offset of the interval's row in a table slice | receiver within the group
    int32_t sender;
    int32_t pad;
};
static_assert(sizeof(TabRec) == 32, "a 16-byte and an 8-byte load");
// the intervals of two edges differ (rows are multiples of 16 bytes)
__device__ __forceinline__ bool other_row(int off, int cur) { return (unsigned)(off ^ cur) >= 4u; }

// The 18 coefficients of one channel: pairs (phi_s, phi_v1) and phi_v2.
struct Coef {
    f32x2 sa[TAB_NC];
    float b[TAB_NC];
    template <bool SMEM>
    __device__ __forceinline__ void load(const char* table, int off, int lane) {
        const char* row = table + (off & ~3);
        const float4* q = reinterpret_cast<const float4*>(row) + lane;
        const float2* q2 = reinterpret_cast<const float2*>(row + 2048) + lane;
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = SMEM ? q[32 * j] : __ldg(q + 32 * j);
        const float2 w = SMEM ? *q2 : __ldg(q2);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            sa[2 * j] = pack2(v[j].x, v[j].y);
            sa[2 * j + 1] = pack2(v[j].z, v[j].w);
        }
        b[0] = v[3].x; b[1] = v[3].y; b[2] = v[3].z; b[3] = v[3].w;
        b[4] = w.x; b[5] = w.y;
    }
};

__device__ __forceinline__ float poly(const float (&c)[TAB_NC], float t) {
    return fmaf(fmaf(fmaf(fmaf(fmaf(c[5], t, c[4]), t, c[3]), t, c[2]), t, c[1]), t, c[0]);
}
// value and d/dt
__device__ __forceinline__ void poly_d(const float (&c)[TAB_NC], float t, float& f, float& fd) {
    float p = c[5], q = c[5];
    p = fmaf(p, t, c[4]);
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        q = fmaf(q, t, p);
        p = fmaf(p, t, c[k]);
    }
    f = p;
    fd = q;
}
__device__ __forceinline__ f32x2 poly(const f32x2 (&c)[TAB_NC], f32x2 t) {
    f32x2 p = c[5];
#pragma unroll
    for (int k = 4; k >= 0; --k) p = fma2(p, t, c[k]);
    return p;
}
__device__ __forceinline__ void poly_d(const f32x2 (&c)[TAB_NC], f32x2 t, f32x2& f, f32x2& fd) {
    f32x2 p = c[5], q = c[5];
    p = fma2(p, t, c[4]);
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        q = fma2(q, t, p);
        p = fma2(p, t, c[k]);
    }
    f = p;
    fd = q;
}

// Records of a warp's edges staged through shared memory: chunks of 4 (128
// bytes), a ring of 4, two chunks ahead.
constexpr int RING = 4;
constexpr int RING_BYTES = RING * 4 * (int)sizeof(TabRec);
struct RecRing {
    unsigned char* buf;
    const TabRec* src;      // the group's first record
    int lane;
    __device__ __forceinline__ void stage(int k) const {
        if (lane < 8)
            tc::cp_async16(buf + (k & (RING - 1)) * 128 + lane * 16,
                           reinterpret_cast<const unsigned char*>(src + 4 * k) + lane * 16);
        tc::cp_async_commit();
    }
    // all but the last staged chunk have landed, for every lane
    __device__ __forceinline__ void ready() const {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
    }
    __device__ __forceinline__ const TabRec* at(int k, int u) const {
        return reinterpret_cast<const TabRec*>(buf + (k & (RING - 1)) * 128) + u;
    }
};

constexpr int FWD_NT = 640, BWD_NT = 512, SMALL_NT = 128;   // threads per CTA (small: table read from memory)
constexpr uint32_t TAB_SLICE_BYTES = TAB_SLICE * 4;      // 221,184
constexpr uint32_t TAB_RING = TAB_SLICE_BYTES + 64;       // behind the barrier, group range and counter
__host__ __device__ constexpr uint32_t tab_smem(int nt) { return TAB_RING + nt / 32 * RING_BYTES; }
static_assert(tab_smem(FWD_NT) <= 232448, "table slice and record rings in shared memory");

// The CTA's table slice into shared memory (one bulk copy of packed weights,
// before the wait for the previous kernel).
__device__ __forceinline__ uint64_t* tab_stage(unsigned char* smem, const float* tab, int slice) {
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + TAB_SLICE_BYTES);
    if (threadIdx.x == 0) {
        tc::mbar_init(bar, 1);
        tc::fence_mbar_init();
        tc::mbar_expect_tx(bar, TAB_SLICE_BYTES);
        const char* src = reinterpret_cast<const char*>(tab + slice * TAB_SLICE);
        constexpr uint32_t CH = TAB_SLICE_BYTES / 12;
        static_assert(CH % 16 == 0 && CH * 12 == TAB_SLICE_BYTES, "copy chunks");
#pragma unroll 1
        for (int i = 0; i < 12; ++i) tc::bulk_g2s(smem + i * CH, src + i * CH, CH, bar);
    }
    return bar;
}

// first group whose edges start at or after share p of nparts
__device__ __forceinline__ int group_bound(const int32_t* row_ptr, int n_atoms, int G, int ngroups, int p, int nparts) {
    if (p <= 0) return 0;
    if (p >= nparts) return ngroups;
    const int64_t target = ((int64_t)row_ptr[n_atoms] * p + nparts - 1) / nparts;
    int lo = 0, hi = ngroups;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (row_ptr[min(mid * G, n_atoms)] >= target) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Walks the groups of this CTA (SMEM: its share of the groups of slice
// blockIdx.x % 4, handed to the warps one by one; otherwise one group and
// slice per warp) and calls body(group, slice).
template <bool SMEM, class Args, class F>
__device__ __forceinline__ void for_groups(const Args& a, int G, unsigned char* smem, F&& body) {
    const int ngroups = (a.n_atoms + G - 1) / G;
    const int lane = threadIdx.x & 31;
    if constexpr (SMEM) {
        const int slice = blockIdx.x & 3;
        uint64_t* bar = tab_stage(smem, a.tab, slice);
        int* range = reinterpret_cast<int*>(smem + TAB_SLICE_BYTES + 16);   // first, end, next
        pdl_wait();
        const bool dead = a.st->code != 0;
        if (!dead) {
            if ((threadIdx.x & 31) == 0 && threadIdx.x < 64) {
                const int p = (blockIdx.x >> 2) + (threadIdx.x >> 5);
                range[threadIdx.x >> 5] = group_bound(a.row_ptr, a.n_atoms, G, ngroups, p, gridDim.x >> 2);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            range[2] = dead ? ngroups : range[0];
            // (also before returning: the copy must have landed when the CTA exits)
            if (!tc::mbar_wait(bar, 0, tc::WAIT_BUDGET)) {
                set_status(a.st, MLFF_ERR_TIMEOUT, 50);
                range[2] = ngroups;
                tc::mbar_wait(bar, 0, tc::WAIT_BUDGET);   // no copy in flight past the CTA's end
            }
        }
        __syncthreads();
        pdl_trigger();
        if (dead) return;
        const int end = range[1];
        while (true) {
            int g = 0;
            if (lane == 0) g = atomicAdd(range + 2, 1);
            g = __shfl_sync(0xffffffffu, g, 0);
            if (g >= end) break;
            body(g, slice);
        }
    } else {
        pdl_wait();
        pdl_trigger();
        if (a.st->code != 0) return;
        const int nw = (gridDim.x * blockDim.x) >> 5;
        for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < 4 * ngroups; k += nw) body(k >> 2, k & 3);
    }
}

// Grid and dynamic shared memory of a table kernel: one CTA per SM and
// slice share with the table staged, else a warp per group and slice.
template <int G, bool SMEM, int NT>
struct TabLaunch {
    static constexpr uint32_t SM = SMEM ? tab_smem(NT) : NT / 32 * RING_BYTES;
    static int grid(int n_atoms) {
        return SMEM ? std::max(4, num_sms() & ~3) : (4 * ((n_atoms + G - 1) / G) + NT / 32 - 1) / (NT / 32);
    }
    template <class K>
    static int prepare(K* kernel) {
        if (!SMEM) return MLFF_OK;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM);
        return e == cudaSuccess ? MLFF_OK : cuda_status(e, "table kernel smem attribute");
    }
};

// Receivers per group, and whether a CTA stages its table slice in shared
// memory (221 KB, one bulk copy that overlaps the kernel before when that
// leaves SMs idle).
//
// Groups share coefficient loads between receivers but choose the receiver's
// sums per edge: 2 receivers are best for inference from 1,500 atoms
// (16,858 atoms, path 5: 1 receiver 1,513 us of reverse pass, 2: 1,432, 4:
// 1,505; path 6, both passes: 2,676, 2,473, 2,498), 1 for the passes of
// training, which read more per edge (3,804 atoms: 1,246 against 1,337).
//
// After the tensor-core path's update kernels, which take one SM per 32 atoms,
// staging always pays (60 atoms: 390 against 405 us a call, 1400: 661 against
// 688); the FP32 update kernels take more SMs (path 6: 60 atoms 466 against
// 423, 500: 556 against 543, 1000: 631 against 662; a training step, 550
// atoms, 2.96 against 3.17 ms of kernels).
struct TabShape {
    int G;
    bool smem;
};
inline TabShape tab_shape(int n_atoms, int path) {
    if (is_train_table(path)) return {1, n_atoms >= 400};
    if (n_atoms >= 1500) return {2, true};
    return {1, path == MLFF_PATH_TABLE || n_atoms >= 750};
}

}  // namespace mlff
