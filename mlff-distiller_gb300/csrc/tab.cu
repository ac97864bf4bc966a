// Edge passes with tabulated filters.
//
// Evaluating the filter network per edge (103,424 FLOP per directed edge and
// layer, twice that in the reverse pass) dominated every evaluation.  The
// network's input is the distance alone, so one table per layer replaces it:
// degree-5 polynomials on 96 intervals, built from float64 values whenever
// weights are packed.  On the seeded weights the table's filter is within
// 6e-8 (2-norm, relative) and its derivative within 5e-7 of float64, as the
// FP32 evaluation of the network (1e-7, 2.4e-7); the build measures both and
// the flag it leaves decides whether the paths use the table (sharper radial
// functions than the table resolves keep the network kernels).
//
// Measured (GB300): a reverse launch on 256 molecules (16,900 atoms, 0.85 M
// edges) 0.41 ms against 0.72 + 0.07 ms of the tensor-core network kernels;
// the FP32 path on 64 molecules 11.2 -> 1.2 ms per call.
#include <algorithm>
#include <cmath>
#include <mutex>
#include "tab.cuh"
#include "tab_edge.cuh"
#include "tc_ptx.cuh"
#include "profile.h"

namespace mlff {

namespace {

// ------------------------------------------------------------ table build
struct NodeInverse {
    double v[TAB_NC][TAB_NC];   // coefficient k = sum_j v[k][j] f(node j)
    double x[TAB_NC];           // Chebyshev nodes
};

const NodeInverse& node_inverse() {
    static const NodeInverse ni = [] {
        NodeInverse r{};
        double a[TAB_NC][2 * TAB_NC];
        for (int j = 0; j < TAB_NC; ++j) r.x[j] = std::cos((2 * j + 1) * 3.14159265358979323846 / (2 * TAB_NC));
        for (int i = 0; i < TAB_NC; ++i)
            for (int k = 0; k < TAB_NC; ++k) {
                a[i][k] = k == 0 ? 1.0 : a[i][k - 1] * r.x[i];
                a[i][TAB_NC + k] = i == k ? 1.0 : 0.0;
            }
        for (int c = 0; c < TAB_NC; ++c) {   // Gauss-Jordan with partial pivoting
            int p = c;
            for (int i = c + 1; i < TAB_NC; ++i)
                if (std::fabs(a[i][c]) > std::fabs(a[p][c])) p = i;
            for (int k = 0; k < 2 * TAB_NC; ++k) std::swap(a[c][k], a[p][k]);
            const double inv = 1.0 / a[c][c];
            for (int k = 0; k < 2 * TAB_NC; ++k) a[c][k] *= inv;
            for (int i = 0; i < TAB_NC; ++i)
                if (i != c) {
                    const double m = a[i][c];
                    for (int k = 0; k < 2 * TAB_NC; ++k) a[i][k] -= m * a[c][k];
                }
        }
        for (int k = 0; k < TAB_NC; ++k)
            for (int j = 0; j < TAB_NC; ++j) r.v[k][j] = a[k][TAB_NC + j];
        return r;
    }();
    return ni;
}

// sum_k w[k] (hi[k] + lo[k]) to well beyond FP32 without FP64 units: the
// products' and sums' rounding errors collected by fused multiply-adds and
// two-sums (the compensated dot product of Ogita, Rump and Oishi, 2005).
struct Dot2 {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float w, float hi, float lo) {
        const float p = __fmul_rn(w, hi);
        const float e = __fmaf_rn(w, hi, -p);
        const float t = __fadd_rn(s, p);
        const float z = __fsub_rn(t, s);
        const float q = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(p, z));
        s = t;
        c = __fadd_rn(c, __fadd_rn(q, __fmaf_rn(w, lo, e)));
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

constexpr int TB_P = TAB_NC + 1;   // nodes and the end point t = 1

// One block per (interval, layer), thread = hidden unit x share of the points,
// then channel x filter.  The hidden units' values at the 6 nodes and the
// interval's end, and the derivative at the end, go through shared memory as
// (hi, lo) floats.  Bound by the latency of its FP64 and compensated chains:
// three shares instead of one per unit and channel, 171 -> 117 us for three
// layers.
constexpr int TB_SHARES = 3;
__global__ void __launch_bounds__(TB_SHARES * H) tab_build_kernel(const float* __restrict__ P, PackedOffsets po, int R,
                                                      float cutoff, NodeInverse ni, float* __restrict__ tab,
                                                      float* __restrict__ node, double* __restrict__ err) {
    __shared__ double e[TB_P + 1][RMAX];   // basis x cutoff at the points; its derivative at the end
    __shared__ float en[TAB_NC][RMAX];     // its derivative at the nodes
    __shared__ float hh[TB_P + 1][H], hl[TB_P + 1][H];
    __shared__ double red[TB_SHARES * H / 32][4];
    const int t = threadIdx.x % H, share = threadIdx.x / H, i = blockIdx.x, l = blockIdx.y;
    const LayerOffsets& lo = po.layer[l];
    const double scale = (double)tab_scale(cutoff);   // dt/dd
    for (int q = threadIdx.x; q < TB_P * RMAX; q += TB_SHARES * H) {
        const int pt = q / RMAX, r = q % RMAX;
        const double x = pt < TAB_NC ? ni.x[pt] : 1.0;
        const double d = ((double)(2 * i + 1) + x) / scale;
        const double rc = cutoff, arg = 3.14159265358979323846 * d / rc;
        const double fc = d < rc ? 0.5 * (cos(arg) + 1.0) : 0.0;
        const double diff = d - (double)P[po.centers + r];
        const double gm = (double)P[po.gamma + r];
        const double g = r < R ? exp(-gm * diff * diff) : 0.0;
        e[pt][r] = g * fc;
        const double dfc = d < rc ? -0.5 * (3.14159265358979323846 / rc) * sin(arg) : 0.0;
        const double gd = g * (dfc - 2.0 * gm * diff * fc);
        if (pt == TAB_NC) {
            e[TB_P][r] = gd;
        } else {
            en[pt][r] = (float)gd;
            float* o = node + l * TAB_NODE_LAYER + TAB_NODES * 4 * H + (int64_t)(i * TAB_NC + pt) * RMAX + r;
            o[0] = (float)(g * fc);
            o[TAB_NODES * RMAX] = (float)gd;
        }
    }
    __syncthreads();
    {   // hidden unit t at points p0, p0 + 1, p0 + 2 (the last: the derivative at the end)
        static_assert(TB_P + 1 <= 3 * TB_SHARES && TB_P % 3 == 1, "the end and its derivative in one share");
        const int p0 = 3 * share;
        double z[3];
        const double b = (double)P[lo.b1 + t];
#pragma unroll
        for (int q = 0; q < 3; ++q) z[q] = p0 + q < TB_P ? b : 0.0;
        float zn[3] = {0.f, 0.f, 0.f};   // the derivatives at nodes
        for (int r = 0; r < R; ++r) {
            const float w = P[lo.w1t + r * H + t];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                z[q] += (double)w * e[min(p0 + q, TB_P)][r];
                zn[q] = fmaf(w, en[min(p0 + q, TAB_NC - 1)][r], zn[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int pt = p0 + q;
            if (pt >= TB_P) break;
            const double s = 1.0 / (1.0 + exp(-z[q]));
            const double h = z[q] * s;
            hh[pt][t] = (float)h;
            hl[pt][t] = (float)(h - (double)(float)h);
            if (pt < TAB_NC) {
                float* o = node + l * TAB_NODE_LAYER + (int64_t)(i * TAB_NC + pt) * H + t;
                o[0] = (float)z[q];
                o[TAB_NODES * H] = (float)h;
                o[2 * TAB_NODES * H] = zn[q];
                o[3 * TAB_NODES * H] = dsilu_f((float)z[q]) * zn[q];
            } else if (q + 1 < 3) {
                const double hd = s * (1.0 + z[q] * (1.0 - s)) * z[q + 1];
                hh[TB_P][t] = (float)hd;
                hl[TB_P][t] = (float)(hd - (double)(float)hd);
            }
        }
    }
    __syncthreads();
    double ef = 0.0, nf = 0.0, ed = 0.0, nd = 0.0;
    float* row = tab + l * TAB_LAYER + (t >> 5) * TAB_SLICE + (int64_t)i * TAB_ROW;
    {   // channel t of filter g
        const int g = share;
        Dot2 acc[TB_P + 1];
        for (int k = 0; k < H; ++k) {
            const float w = P[lo.w2t + k * H3 + g * H + t];
#pragma unroll
            for (int pt = 0; pt <= TB_P; ++pt) acc[pt].add(w, hh[pt][k], hl[pt][k]);
        }
        const double b = (double)P[lo.b2 + g * H + t];
        double f[TAB_NC];
#pragma unroll
        for (int j = 0; j < TAB_NC; ++j) f[j] = acc[j].value() + b;
        double pf = 0.0, pd = 0.0;
#pragma unroll
        for (int k = 0; k < TAB_NC; ++k) {
            double c = 0.0;
#pragma unroll
            for (int j = 0; j < TAB_NC; ++j) c += ni.v[k][j] * f[j];
            const float cf = (float)c;
            row[tab_off(t & 31, g, k)] = cf;
            pf += (double)cf;
            pd += k * (double)cf;
        }
        const double xf = acc[TAB_NC].value() + b, xd = acc[TB_P].value();
        pd *= scale;
        ef += (pf - xf) * (pf - xf);
        nf += xf * xf;
        ed += (pd - xd) * (pd - xd);
        nd += xd * xd;
    }
    double v[4] = {ef, nf, ed, nd};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double s = 0.0;
        for (int w = 0; w < TB_SHARES * H / 32; ++w) s += red[w][t];
        err[((int64_t)l * TAB_NI + i) * 4 + t] = s;
    }
}

// flag = the strictest accuracy class every layer's table meets
__global__ void __launch_bounds__(128) tab_flag_kernel(const double* __restrict__ err, int n_layers,
                                                       int32_t* __restrict__ flag) {
    __shared__ double red[4][128];
    const int t = threadIdx.x;
    int best = TAB_OK_FP32;
    for (int l = 0; l < n_layers; ++l) {
        for (int q = 0; q < 4; ++q) red[q][t] = t < TAB_NI ? err[((int64_t)l * TAB_NI + t) * 4 + q] : 0.0;
        __syncthreads();
        for (int o = 64; o > 0; o >>= 1) {
            if (t < o)
                for (int q = 0; q < 4; ++q) red[q][t] += red[q][t + o];
            __syncthreads();
        }
        // (written so that NaN or infinite sums fail; a filter that is zero
        // everywhere passes)
        const double ef = red[0][0], nf = red[1][0], ed = red[2][0], nd = red[3][0];
        auto within = [](double e2, double n2, double tol) { return e2 <= tol * tol * n2 && n2 < 1e300; };
        const bool f_ok = within(ef, nf, TAB_TOL_F);
        if (!(f_ok && within(ed, nd, TAB_TOL_D_FP32))) best = min(best, TAB_OK_TC);
        if (!(f_ok && within(ed, nd, TAB_TOL_D_TC))) best = 0;
        __syncthreads();
    }
    if (t == 0) *flag = best;
}
static_assert(TAB_NI <= 128, "one thread per interval");

}  // namespace

int build_tables(const mlff_dims& d, float* packed, const PackedOffsets& po, cudaStream_t st) {
    double* err = reinterpret_cast<double*>(packed + po.tab_err);
    tab_build_kernel<<<dim3(TAB_NI, d.n_layers), TB_SHARES * H, 0, st>>>(packed, po, d.n_rbf, d.cutoff, node_inverse(),
                                                             packed + po.tab, packed + po.tab_node, err);
    MLFF_LAUNCH_CHECK("tab_build");
    tab_flag_kernel<<<1, 128, 0, st>>>(err, d.n_layers, reinterpret_cast<int32_t*>(packed + po.tab_flag));
    MLFF_LAUNCH_CHECK("tab_flag");
    return MLFF_OK;
}

void table_nodes(float* node, float* weight) {
    for (int j = 0; j < TAB_NC; ++j) node[j] = (float)node_inverse().x[j];
    for (int j = 0; j < TAB_NC; ++j) {
        double w = 1.0;
        for (int m = 0; m < TAB_NC; ++m)
            if (m != j) w *= node_inverse().x[j] - node_inverse().x[m];
        weight[j] = (float)(1.0 / w);
    }
}

int read_table_flag(const float* packed, const PackedOffsets& po, int32_t* flag, cudaStream_t st) {
    MLFF_CUDA(cudaMemcpyAsync(flag, packed + po.tab_flag, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    MLFF_CUDA(cudaStreamSynchronize(st));
    return MLFF_OK;
}

namespace {

// ------------------------------------------------------------ edge records
// The edges of a group of G receivers (consecutive CSR rows) in the order of
// their interval, ties in edge order: a run of edges of one interval then
// loads its 18 coefficients once.  A receiver's own edges come in the same
// order for every G, so results do not depend on it.  One warp per group,
// a stable counting sort over the intervals in shared memory; a group of up
// to 256 edges keeps its geometry in registers between the two passes.
constexpr int REC_WARPS = 4;
constexpr int REC_REG = 8;    // chunks of 32 edges kept in registers

struct RecArgs {
    const float4* geo;    // (u, d) of every edge, when the forward pass has made them (or NULL)
    const float4* pos4;
    const int32_t* atom_mol;
    const float* box;
    const uint8_t* pbc;
    const int32_t* row_ptr;
    const int32_t* col;
    const int32_t* erecv;
    int n_atoms, G, need;
    float scale;
    const int32_t* flag;
    TabRec* rec;
    int32_t* perm;        // sorted position -> edge
    Status* st;
};

struct EdgeGeo {
    int key, b, r;
    float ux, uy, uz, t;
};
__device__ __forceinline__ EdgeGeo edge_geo(const RecArgs& a, int k, int a0) {
    EdgeGeo g;
    const int i = a.erecv[k];
    g.b = a.col[k];
    g.r = i - a0;
    float d;
    if (a.geo) {   // (100,000 atoms 327 -> 195 us)
        const float4 u = a.geo[k];
        g.ux = u.x;
        g.uy = u.y;
        g.uz = u.z;
        d = u.w;
    } else {
        Box bx;
        bx.periodic = 0;
        if (a.pbc != nullptr && a.box != nullptr) {
            const int m = a.atom_mol[i];
            bx.periodic = a.pbc[m] ? 1 : 0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                bx.L[q] = bx.periodic ? a.box[3 * m + q] : 1.0f;
                bx.invL[q] = __fdiv_rn(1.0f, bx.L[q]);
            }
        }
        const float3 v = edge_vector(a.pos4[g.b], a.pos4[i], bx);
        d = pair_distance(v.x, v.y, v.z);
        const float inv = 1.0f / (d + 1e-8f);
        g.ux = v.x * inv;
        g.uy = v.y * inv;
        g.uz = v.z * inv;
    }
    // interval and local coordinate t = 2 (d / width - i) - 1, one rounding
    g.key = min((int)(0.5f * a.scale * d), TAB_NI - 1);
    g.t = fmaf(d, a.scale, -(float)(2 * g.key + 1));
    return g;
}

__global__ void __launch_bounds__(REC_WARPS * 32) tab_records_kernel(RecArgs a) {
    pdl_wait();
    pdl_trigger();
    __shared__ int hist[REC_WARPS][128];
    if (a.st->code != 0) return;
    if (*a.flag < a.need) {   // the weights' tables are not accurate enough for this path
        if (threadIdx.x == 0) set_status(a.st, MLFF_ERR_UNSUPPORTED, -1);
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int* hw = hist[w];
    const int ngroups = (a.n_atoms + a.G - 1) / a.G;
    const unsigned lt = (1u << lane) - 1u;
    for (int g = blockIdx.x * REC_WARPS + w; g < ngroups; g += gridDim.x * REC_WARPS) {
        const int a0 = g * a.G, e0 = a.row_ptr[a0], e1 = a.row_ptr[min(a0 + a.G, a.n_atoms)];
        for (int q = lane; q < 128; q += 32) hw[q] = 0;
        __syncwarp();
        auto count = [&](int key) {
            const unsigned peers = __match_any_sync(0xffffffffu, key);
            if ((peers & lt) == 0) hw[key] += __popc(peers);
            __syncwarp();
        };
        // exclusive scan of the interval counts (4 per lane; slot 127 takes the padding lanes)
        auto scan = [&]() {
            int c[4], s = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                c[q] = hw[4 * lane + q];
                s += c[q];
            }
            int incl = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            int base = incl - s;
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                hw[4 * lane + q] = base;
                base += c[q];
            }
            __syncwarp();
        };
        auto place = [&](int k, const EdgeGeo& e) {
            const unsigned peers = __match_any_sync(0xffffffffu, e.key);
            const int at = hw[e.key];
            __syncwarp();
            if (k < e1) {
                const int p = e0 + at + __popc(peers & lt);
                float4* o = reinterpret_cast<float4*>(a.rec + p);
                o[0] = make_float4(e.t, e.t, e.uy, e.uz);
                o[1] = make_float4(e.ux, __int_as_float(e.key * TAB_ROW_BYTES | e.r), __int_as_float(e.b), 0.f);
                a.perm[p] = k;
            }
            if ((peers & lt) == 0) hw[e.key] = at + __popc(peers);
            __syncwarp();
        };
        EdgeGeo none{};
        none.key = 127;
        if (e1 - e0 <= 32 * REC_REG) {
            EdgeGeo e[REC_REG];
#pragma unroll
            for (int j = 0; j < REC_REG; ++j) {
                const int k = e0 + 32 * j + lane;
                e[j] = k < e1 ? edge_geo(a, k, a0) : none;
            }
#pragma unroll
            for (int j = 0; j < REC_REG; ++j)
                if (e0 + 32 * j < e1) count(e[j].key);
            scan();
#pragma unroll
            for (int j = 0; j < REC_REG; ++j)
                if (e0 + 32 * j < e1) place(e0 + 32 * j + lane, e[j]);
        } else {
            for (int k0 = e0; k0 < e1; k0 += 32) {
                const int k = k0 + lane;
                count(k < e1 ? edge_geo(a, k, a0).key : 127);
            }
            scan();
            for (int k0 = e0; k0 < e1; k0 += 32) {
                const int k = k0 + lane;
                place(k, k < e1 ? edge_geo(a, k, a0) : none);
            }
        }
        if (g == ngroups - 1 && lane < TREC_PAD) {   // records read past the end: sender 0, interval 0
            float4* o = reinterpret_cast<float4*>(a.rec + e1 + lane);
            o[0] = make_float4(0.f, 0.f, 0.f, 0.f);
            o[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}
static_assert(TAB_NI < 127, "slot 127 holds the padding lanes");
static_assert(TAB_ROW_BYTES % 16 == 0, "the receiver in the low bits of a row's offset");

// ----------------------------------------------------------- edge kernels
struct TabArgs {
    const TabRec* rec;
    const int32_t* row_ptr;
    int n_atoms;
    const float* tab;      // the layer's table
    const float* X;        // layer input: layer 0 s [N][H], later layers quads [N][H][4]; or pairs
    float* Xt;             // forward: X + messages, component-major [N][4][H]
    const float4* xtbar;   // reverse: dE/dXt, quads
    float* xbar;           // reverse: dE/dX, component-major
    float* part;           // reverse: per slice and sorted edge (dE/dd, dE/du), [4][cap][4]
    int64_t cap;
    int eacc_init;         // reverse: 1 = part is written, 0 = added to
    Status* st;
};

template <int G, bool SMEM, bool L0, int NT>
__global__ void __launch_bounds__(NT, SMEM ? 1 : 4) tab_fwd_kernel(TabArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    RecRing ring{smem + (SMEM ? TAB_RING : 0) + (threadIdx.x >> 5) * RING_BYTES, nullptr, lane};
    for_groups<SMEM>(a, G, smem, [&](int g, int slice) {
        const char* table = SMEM ? reinterpret_cast<const char*>(smem)
                                 : reinterpret_cast<const char*>(a.tab + slice * TAB_SLICE);
        const int ch = 32 * slice + lane;
        const int a0 = g * G;
        const int e0 = a.row_ptr[a0], n = a.row_ptr[min(a0 + G, a.n_atoms)] - e0;
        f32x2 acc01[G];                 // sums of (s, v_x)
        float acc2[G], acc3[G];         // v_y, v_z
#pragma unroll
        for (int r = 0; r < G; ++r) {
            acc01[r] = pack2(0.f, 0.f);
            acc2[r] = acc3[r] = 0.f;
        }
        const float4* X4 = reinterpret_cast<const float4*>(a.X) + ch;
        const float* X1 = a.X + ch;
        if (n > 0) {
            Coef c;
            int cur = -1;
            float4 xa[2], xb[2];        // sender features of two edges each, in flight
            auto gather = [&](float4 (&x)[2], int k, int u0) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int64_t j = ring.at(k, u0 + u)->sender;
                    if (L0) x[u].x = __ldg(X1 + j * H);
                    else x[u] = __ldg(X4 + j * H);
                }
            };
            auto edge = [&](const TabRec* rp, const float4& x) {
                const float4 ra = reinterpret_cast<const float4*>(rp)[0];
                const float2 rb = reinterpret_cast<const float2*>(rp)[2];
                const int off = __float_as_int(rb.y);
                if (uni(other_row(off, cur))) {
                    c.load<SMEM>(table, off, lane);
                    cur = off;
                }
                float fs, f1;
                f32x2 sa;
                if (L0) {   // v = 0: phi_v1 does not enter
                    const float s[TAB_NC] = {lo2(c.sa[0]), lo2(c.sa[1]), lo2(c.sa[2]), lo2(c.sa[3]), lo2(c.sa[4]),
                                             lo2(c.sa[5])};
                    fs = poly(s, ra.x);
                } else {
                    sa = poly(c.sa, pack2(ra.x, ra.y));
                    f1 = hi2(sa);
                }
                const float f2 = poly(c.b, ra.x);
                auto add = [&](f32x2& s01, float& s2, float& s3) {
                    if (L0) {
                        s01 = fma2(pack2(x.x, rb.x), pack2(fs, f2), s01);
                        s2 = fmaf(ra.z, f2, s2);
                        s3 = fmaf(ra.w, f2, s3);
                    } else {
                        s01 = pack2(lo2(s01), fmaf(rb.x, f2, hi2(s01)));
                        s01 = fma2(pack2(x.x, x.y), sa, s01);
                        s2 = fmaf(x.z, f1, fmaf(ra.z, f2, s2));
                        s3 = fmaf(x.w, f1, fmaf(ra.w, f2, s3));
                    }
                };
                tab_switch<G>(off, [&](auto r) {
                    constexpr int R = decltype(r)::value;
                    add(acc01[R], acc2[R], acc3[R]);
                });
            };
            ring.src = a.rec + e0;
            tc::cp_async_wait_all();    // the previous group's last copies have landed, its records are read
            __syncwarp();
            ring.stage(0);
            ring.stage(1);
            ring.ready();
            ring.stage(2);
            gather(xa, 0, 0);
            const int full = n >> 2, left = n & 3;
#pragma unroll 1
            for (int k = 0; k < full; ++k) {
                gather(xb, k, 2);
                edge(ring.at(k, 0), xa[0]);
                edge(ring.at(k, 1), xa[1]);
                ring.ready();           // chunk k + 1 (past the end: other records, not used)
                gather(xa, k + 1, 0);
                edge(ring.at(k, 2), xb[0]);
                edge(ring.at(k, 3), xb[1]);
                ring.stage(k + 3);      // into the slot of chunk k - 1
            }
            gather(xb, full, 2);
#pragma unroll 1
            for (int u = 0; u < left; ++u) {
                edge(ring.at(full, u), xa[0]);
                xa[0] = xa[1];
                xa[1] = xb[0];
            }
        }
#pragma unroll
        for (int r = 0; r < G; ++r) {
            if (a0 + r >= a.n_atoms) break;
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (L0) b.x = X1[(int64_t)(a0 + r) * H];
            else b = X4[(int64_t)(a0 + r) * H];
            float* o = a.Xt + (int64_t)(a0 + r) * 4 * H + ch;
            o[0] = b.x + lo2(acc01[r]);
            o[H] = b.y + hi2(acc01[r]);
            o[2 * H] = b.z + acc2[r];
            o[3 * H] = b.w + acc3[r];
        }
    });
    tc::cp_async_wait_all();
}

// Per edge (receiver i, sender j), channel c of the slice:
//   dE/dX_i += dE/dXt_j (phi_s, phi_v1)          (the sender side's gather:
//                                                 the reverse edge has the same filter)
//   dE/dd    = sum_c q0 phi_s' + q1 phi_v1' + q2 phi_v2'
//   dE/du_k  = sum_c dE/dXt_i.v_k phi_v2
// with q0 = dE/dXt_i.s X_j.s, q1 = dE/dXt_i.v . X_j.v, q2 = dE/dXt_i.v . u.
// The four channel sums of 4 edges are reduced over the lanes together (16
// shuffles); the four slices' shares are added by tab_combine_kernel.
// PAIRS: X in the tensor-core forward pass's pair layout (layer 0 too).
template <int G, bool SMEM, bool L0, bool PAIRS, int NT>
__global__ void __launch_bounds__(NT, SMEM ? 1 : 4) tab_bwd_kernel(TabArgs a, float scale) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    RecRing ring{smem + (SMEM ? TAB_RING : 0) + (threadIdx.x >> 5) * RING_BYTES, nullptr, lane};
    for_groups<SMEM>(a, G, smem, [&](int g, int slice) {
        const char* table = SMEM ? reinterpret_cast<const char*>(smem)
                                 : reinterpret_cast<const char*>(a.tab + slice * TAB_SLICE);
        const int ch = 32 * slice + lane;
        const int a0 = g * G;
        const int e0 = a.row_ptr[a0], n = a.row_ptr[min(a0 + G, a.n_atoms)] - e0;
        f32x2 acc01[G];
        float acc2[G], acc3[G];
        float4 ta[G];
        const float4* T4 = a.xtbar + ch;
        const float4* X4 = reinterpret_cast<const float4*>(a.X) + ch;
        const float2* X2 = reinterpret_cast<const float2*>(a.X) + ch;
        const float* X1 = PAIRS ? a.X + 2 * ch : a.X + ch;
#pragma unroll
        for (int r = 0; r < G; ++r) {
            ta[r] = T4[(int64_t)min(a0 + r, a.n_atoms - 1) * H];
            acc01[r] = pack2(0.f, 0.f);
            acc2[r] = acc3[r] = 0.f;
        }
        if (n > 0) {
            // lane 2 i holds sum i = 4 edge + quantity of a chunk after the reduction
            const int si = lane >> 1;
            const bool even = (lane & 1) == 0;
            const float mul = (si & 3) == 0 ? scale : 1.0f;   // dE/dd: the table's derivative is in t
            float* dst = a.part + ((int64_t)slice * a.cap + e0) * 4 + si;
            Coef c;
            int cur = -1;
            float4 xa[2], ya[2], xb[2], yb[2];   // sender features and adjoints of two edges each, in flight
            auto gather = [&](float4 (&x)[2], float4 (&y)[2], int k, int u0) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int64_t j = ring.at(k, u0 + u)->sender;
                    if (L0) {
                        x[u].x = __ldg(X1 + j * (PAIRS ? 4 * H : H));
                    } else {
                        if (PAIRS) {
                            const float2 p = __ldg(X2 + j * 2 * H), q = __ldg(X2 + j * 2 * H + H);
                            x[u] = make_float4(p.x, p.y, q.x, q.y);
                        } else {
                            x[u] = __ldg(X4 + j * H);
                        }
                        y[u] = __ldg(T4 + j * H);
                    }
                }
            };
            auto edge = [&](const TabRec* rp, const float4& x, const float4& y, float* v) {
                const float4 ra = reinterpret_cast<const float4*>(rp)[0];
                const float2 rb = reinterpret_cast<const float2*>(rp)[2];
                const int off = __float_as_int(rb.y);
                if (uni(other_row(off, cur))) {
                    c.load<SMEM>(table, off, lane);
                    cur = off;
                }
                float f2, d2, ds;
                f32x2 sa, da;
                if (L0) {
                    const float s[TAB_NC] = {lo2(c.sa[0]), lo2(c.sa[1]), lo2(c.sa[2]), lo2(c.sa[3]), lo2(c.sa[4]),
                                             lo2(c.sa[5])};
                    float fs;
                    poly_d(s, ra.x, fs, ds);
                } else {
                    poly_d(c.sa, pack2(ra.x, ra.y), sa, da);
                }
                poly_d(c.b, ra.x, f2, d2);
                auto add = [&](const float4& ti, f32x2& s01, float& s2, float& s3) {
                    const float q0 = ti.x * x.x;
                    const float q2 = fmaf(ti.y, rb.x, fmaf(ti.z, ra.z, ti.w * ra.w));
                    if (L0) {
                        v[0] = fmaf(q0, ds, q2 * d2);
                    } else {
                        const float q1 = fmaf(ti.y, x.y, fmaf(ti.z, x.z, ti.w * x.w));
                        v[0] = fmaf(q0, lo2(da), fmaf(q1, hi2(da), q2 * d2));
                        s01 = fma2(pack2(y.x, y.y), sa, s01);
                        s2 = fmaf(y.z, hi2(sa), s2);
                        s3 = fmaf(y.w, hi2(sa), s3);
                    }
                    v[1] = ti.y * f2;
                    v[2] = ti.z * f2;
                    v[3] = ti.w * f2;
                };
                tab_switch<G>(off, [&](auto r) {
                    constexpr int R = decltype(r)::value;
                    add(ta[R], acc01[R], acc2[R], acc3[R]);
                });
            };
            ring.src = a.rec + e0;
            tc::cp_async_wait_all();
            __syncwarp();
            ring.stage(0);
            ring.stage(1);
            ring.ready();
            ring.stage(2);
            gather(xa, ya, 0, 0);
            const int full = n >> 2, left = n & 3;
#pragma unroll 1
            for (int k = 0; k < full; ++k) {
                float prev = 0.f;
                if (even && !a.eacc_init) prev = *dst;
                float v[16];
                gather(xb, yb, k, 2);
                edge(ring.at(k, 0), xa[0], ya[0], v);
                edge(ring.at(k, 1), xa[1], ya[1], v + 4);
                ring.ready();
                gather(xa, ya, k + 1, 0);
                edge(ring.at(k, 2), xb[0], yb[0], v + 8);
                edge(ring.at(k, 3), xb[1], yb[1], v + 12);
                ring.stage(k + 3);
                const float s = reduce16(v, lane);
                if (even) *dst = fmaf(s, mul, prev);
                dst += 16;
            }
            if (uni(left != 0)) {
                const bool mine = even && (si >> 2) < left;
                float prev = 0.f;
                if (mine && !a.eacc_init) prev = *dst;
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = 0.f;
                edge(ring.at(full, 0), xa[0], ya[0], v);
                if (uni(left > 1)) edge(ring.at(full, 1), xa[1], ya[1], v + 4);
                if (uni(left > 2)) {
                    gather(xb, yb, full, 2);
                    edge(ring.at(full, 2), xb[0], yb[0], v + 8);
                }
                const float s = reduce16(v, lane);
                if (mine) *dst = fmaf(s, mul, prev);
            }
        }
        if (!L0) {
#pragma unroll
            for (int r = 0; r < G; ++r) {
                if (a0 + r >= a.n_atoms) break;
                float* o = a.xbar + (int64_t)(a0 + r) * 4 * H + ch;
                o[0] = ta[r].x + lo2(acc01[r]);
                o[H] = ta[r].y + hi2(acc01[r]);
                o[2 * H] = ta[r].z + acc2[r];
                o[3 * H] = ta[r].w + acc3[r];
            }
        }
    });
    tc::cp_async_wait_all();
}

// edge_acc[perm[p]] = the four slices' (dE/dd, dE/du) of sorted edge p
__global__ void __launch_bounds__(256) tab_combine_kernel(const float4* __restrict__ part,
                                                          const int32_t* __restrict__ perm, int64_t cap,
                                                          const int32_t* __restrict__ row_ptr, int n_atoms,
                                                          float4* __restrict__ eacc, const Status* st) {
    pdl_wait();
    pdl_trigger();
    if (st->code != 0) return;
    const int E = row_ptr[n_atoms];
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < E; p += gridDim.x * blockDim.x) {
        const float4 a = part[p], b = part[cap + p], c = part[2 * cap + p], d = part[3 * cap + p];
        eacc[perm[p]] = make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y), (a.z + b.z) + (c.z + d.z),
                                    (a.w + b.w) + (c.w + d.w));
    }
}

// ------------------------------------------------------------- launchers
template <int G, bool SMEM, bool L0>
int launch_fwd_t(const TabArgs& a, cudaStream_t st) {
    constexpr int NT = SMEM ? FWD_NT : SMALL_NT;
    using TL = TabLaunch<G, SMEM, NT>;
    static std::once_flag once;
    static int err = MLFF_OK;
    std::call_once(once, [] { err = TL::prepare(tab_fwd_kernel<G, SMEM, L0, NT>); });
    if (err) return err;
    MLFF_LAUNCH_PDL("tab_fwd", (tab_fwd_kernel<G, SMEM, L0, NT>), TL::grid(a.n_atoms), NT, TL::SM, st, a);
    return MLFF_OK;
}
template <int G, bool SMEM, bool L0, bool PAIRS>
int launch_bwd_t(const TabArgs& a, float scale, cudaStream_t st) {
    constexpr int NT = SMEM ? BWD_NT : SMALL_NT;
    using TL = TabLaunch<G, SMEM, NT>;
    static std::once_flag once;
    static int err = MLFF_OK;
    std::call_once(once, [] { err = TL::prepare(tab_bwd_kernel<G, SMEM, L0, PAIRS, NT>); });
    if (err) return err;
    MLFF_LAUNCH_PDL("tab_bwd", (tab_bwd_kernel<G, SMEM, L0, PAIRS, NT>), TL::grid(a.n_atoms), NT, TL::SM, st, a, scale);
    return MLFF_OK;
}

template <bool L0>
int launch_fwd(const TabShape& s, const TabArgs& a, cudaStream_t st) {
    if (s.G == 2) return launch_fwd_t<2, true, L0>(a, st);
    if (s.smem) return launch_fwd_t<1, true, L0>(a, st);
    return launch_fwd_t<1, false, L0>(a, st);
}
template <bool L0, bool PAIRS>
int launch_bwd(const TabShape& s, const TabArgs& a, float scale, cudaStream_t st) {
    if (s.G == 2) return launch_bwd_t<2, true, L0, PAIRS>(a, scale, st);
    if constexpr (!PAIRS)   // (after the tensor-core forward pass tab_shape always stages)
        if (!s.smem) return launch_bwd_t<1, false, L0, PAIRS>(a, scale, st);
    return launch_bwd_t<1, true, L0, PAIRS>(a, scale, st);
}

}  // namespace

namespace {

TabArgs tab_args(const WsLayout& L, void* ws) {
    TabArgs a{};
    a.rec = ws_ptr<TabRec>(ws, L.trec);
    a.row_ptr = ws_ptr<int32_t>(ws, L.row_ptr);
    a.n_atoms = L.N;
    a.part = ws_ptr<float>(ws, L.tpart);
    a.cap = L.cap;
    a.st = ws_ptr<Status>(ws, L.status);
    return a;
}

}  // namespace

int launch_records(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                   const WsLayout& L, void* ws, int path, cudaStream_t st) {
    ProfScope prof(PK_NEIGHBORS, st);
    const TabShape shape = tab_shape(L.N, path);
    const int ngroups = (L.N + shape.G - 1) / shape.G;
    const int grid = std::max(1, std::min((ngroups + REC_WARPS - 1) / REC_WARPS, num_sms() * 16));
    const RecArgs ra{path == MLFF_PATH_TABLE ? ws_ptr<float4>(ws, L.geo) : nullptr, ws_ptr<float4>(ws, L.pos4), ws_ptr<int32_t>(ws, L.atom_mol), sys.box, sys.pbc,
                     ws_ptr<int32_t>(ws, L.row_ptr), ws_ptr<int32_t>(ws, L.col), ws_ptr<int32_t>(ws, L.erecv), L.N,
                     shape.G, path == MLFF_PATH_TABLE ? TAB_OK_TC : TAB_OK_FP32, tab_scale(d.cutoff),
                     reinterpret_cast<const int32_t*>(P + po.tab_flag), ws_ptr<TabRec>(ws, L.trec),
                     ws_ptr<int32_t>(ws, L.tperm), ws_ptr<Status>(ws, L.status)};
    MLFF_LAUNCH_PDL("tab_records", tab_records_kernel, grid, REC_WARPS * 32, 0, st, ra);
    return MLFF_OK;
}

int table_forward(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                  const WsLayout& L, void* ws, int path, cudaStream_t st) {
    const int64_t NX = (int64_t)L.N * 4 * H;
    const TabShape shape = tab_shape(L.N, path);
    int r;
    if ((r = launch_embed(d, P, po, sys, L, ws, st))) return r;
    if ((r = launch_records(d, P, po, sys, L, ws, path, st))) return r;
    TabArgs a = tab_args(L, ws);
    for (int l = 0; l < d.n_layers; ++l) {
        a.tab = P + po.tab + l * TAB_LAYER;
        a.X = ws_ptr<float>(ws, L.X) + l * NX;
        a.Xt = ws_ptr<float>(ws, L.Xt) + l * NX;
        {
            ProfScope prof(PK_EDGE_FWD, st);
            if ((r = l == 0 ? launch_fwd<true>(shape, a, st) : launch_fwd<false>(shape, a, st))) return r;
        }
        if ((r = launch_upd32_fwd(P, po.layer[l], L, ws, l, st))) return r;
    }
    return MLFF_OK;
}

// The FP32 path with tabulated filters (MLFF_PATH_TABLE_FP32; the training
// paths: its reverse pass).
int run_table(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys, const WsLayout& L,
              void* ws, const mlff_outputs& out, int path, cudaStream_t st, const VerletFuse* vf) {
    int r;
    if (is_train_table(path)) {
        // A training step's energies and forces: the fused FP32 path's forward
        // pass, bit for bit.  The loss divides by |F| and the gradients by |v|,
        // so another forward pass, as exact, moves them by up to 5e-5.
        if ((r = launch_embed(d, P, po, sys, L, ws, st))) return r;
        if ((r = launch_records(d, P, po, sys, L, ws, path, st))) return r;
        r = fused_fp32_forward(d, P, po, sys, L, ws, st);
    } else {
        r = table_forward(d, P, po, sys, L, ws, path, st);
    }
    if (r) return r;
    const bool want_grad = out.forces != nullptr || out.virial != nullptr;
    if ((r = launch_readout(d, P, po, sys, L, ws, out, want_grad ? 1 : 0, st))) return r;
    if (!want_grad) return MLFF_OK;
    return run_table_reverse(d, P, po, sys, L, ws, out, path, st, vf);
}

// Reverse pass and forces.  MLFF_PATH_TABLE comes here after the tensor-core
// forward pass (X in the pair layout; the records are made now, in the E
// tiles' space): its energies are those of the split-FP16 evaluation, and the
// reverse pass, half of a call's time with the network evaluated per edge,
// reads the tables.
int run_table_reverse(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                      const WsLayout& L, void* ws, const mlff_outputs& out, int path, cudaStream_t st,
                      const VerletFuse* vf) {
    const int64_t NX = (int64_t)L.N * 4 * H;
    const TabShape shape = tab_shape(L.N, path);
    const bool tc = path == MLFF_PATH_TABLE;
    const float scale = tab_scale(d.cutoff);
    int r;
    if (tc && (r = launch_records(d, P, po, sys, L, ws, path, st))) return r;
    TabArgs a = tab_args(L, ws);
    float* xbo = ws_ptr<float>(ws, L.xbar);
    float* xtb = xbo + NX;
    for (int l = d.n_layers - 1; l >= 0; --l) {
        r = tc ? launch_update_bwd_tc(P, po.layer[l], L, ws, l, xbo, xtb, st)
               : launch_upd32_bwd(P, po.layer[l], L, ws, l, xbo, xtb, st);
        if (r) return r;
        a.tab = P + po.tab + l * TAB_LAYER;
        a.X = ws_ptr<float>(ws, L.X) + l * NX;
        a.xtbar = reinterpret_cast<const float4*>(xtb);
        a.xbar = xbo;
        a.eacc_init = l == d.n_layers - 1 ? 1 : 0;
        ProfScope prof(PK_EDGE_BWD, st);
        if (tc) r = l == 0 ? launch_bwd<true, true>(shape, a, scale, st) : launch_bwd<false, true>(shape, a, scale, st);
        else r = l == 0 ? launch_bwd<true, false>(shape, a, scale, st) : launch_bwd<false, false>(shape, a, scale, st);
        if (r) return r;
    }
    {
        ProfScope prof(PK_FORCES, st);
        const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((L.cap + 255) / 256, num_sms() * 8));
        MLFF_LAUNCH_PDL("tab_combine", tab_combine_kernel, blocks, 256, 0, st, ws_ptr<float4>(ws, L.tpart),
                        ws_ptr<int32_t>(ws, L.tperm), L.cap, a.row_ptr, L.N, ws_ptr<float4>(ws, L.edge_acc), a.st);
    }
    return launch_forces(d, sys, L, ws, out, st, vf);
}

}  // namespace mlff
