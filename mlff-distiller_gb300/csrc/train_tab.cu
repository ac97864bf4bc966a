// Parameter gradients through the tabulated filters (training).
//
// Energy term: sum_b w_b dE_b/dtheta.  Force and stress terms: the
// derivative of grad_theta sum_b E_b along positions moved by -G and cells
// strained by S (forward mode over the reverse pass, as the plain path's
// Dual instantiation).  Here every array has a value plane and, for the
// second, a tangent plane behind it, so that a GEMM of both is one GEMM over
// twice the rows.
//
// A filter value interpolates the filter's values at its interval's nodes.
// So the filter's weight gradient needs the network at the 576 nodes only:
//   fbar(node j)[c] = sum over the interval's edges of L_j(t) fbar_e[c]
// (L_j the Lagrange polynomials, whose sums stay as well conditioned as the
// edges' own, unlike sums of powers of t; the tangent of f interpolates the
// nodes' f' = df/dd instead of differentiating L_j, which would amplify the
// rounding of the nodes' values) followed by the network's reverse pass over
// 576 rows, instead of GEMMs over every edge and layer.  The edges are sorted
// by interval once per call (a stable counting sort) and summed in chunks of
// 64 in a fixed order, so repeated calls give the same bits.
//
// The value forward pass is the plain path's own (plain_forward).  Gradients
// of the force term pass through the second derivative of |v|, ~1/|v|, which
// turns a last-bit change of v into 1e-5 of a gradient; those of the mixing
// matrices cancel to 1e-6.  Errors against float64 are then the plain path's
// own instead of others as large (of 40 random steps of 8 molecules, 10 had a
// tensor 1.5 times further off with a table forward pass, 3 with this one).
//
// Measured (64 molecules of 10..120 atoms, 184,000 edges, energy + force
// terms): 48.3 -> 11.9 ms a step against the plain and Dual passes, whose
// weight gradients (20 ms) and GEMMs (19 ms) run over every edge; 8 molecules
// 15.2 -> 7.7 ms (launches and host), energy term of 100 molecules 14.0 -> 5.7
// ms.
#include <algorithm>
#include <mutex>
#include "common.cuh"
#include "dual.cuh"
#include "gemm.cuh"
#include "tab.cuh"
#include "tab_edge.cuh"
#include "workspace.h"
#include "profile.h"

namespace mlff {

namespace {

constexpr int SEG = TT_SEG;          // edges per segment of the counting sort
constexpr int CHUNK = TT_CHUNK;      // edges per partial sum
constexpr int NODES = TAB_NI * TAB_NC;

inline int blocks_for(int64_t n, int threads = 256) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, num_sms() * 8));
}

// ---------------------------------------------------------- edge tangents
// Per edge in CSR order: value (u, t), interval, and the tangents (u', t') of
// the direction (positions -G, strain S); the tangents in the records' order
// too.
struct MapArgs {
    const TabRec* rec;
    const int32_t* perm;
    const int32_t* row_ptr;
    const int32_t* col;
    const int32_t* erecv;
    const float4* pos4;
    const int32_t* atom_mol;
    const float* box;
    const uint8_t* pbc;
    const float* G;          // [N][3] or NULL
    const double* S;         // [B][9] or NULL
    float scale;
    int n_atoms, dual;
    float4* geo;             // [cap] (u, t)
    int32_t* key;            // [cap]
    float4* geo_t;           // [cap] (u', t')
    float4* rec_t;           // [cap + TREC_PAD], sorted order
    const Status* st;
};

__global__ void __launch_bounds__(256) edge_maps_kernel(MapArgs a) {
    if (a.st->code != 0) return;
    const int E = a.row_ptr[a.n_atoms];
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < E; p += gridDim.x * blockDim.x) {
        const int k = a.perm[p];
        const float4 ra = reinterpret_cast<const float4*>(a.rec + p)[0], rb = reinterpret_cast<const float4*>(a.rec + p)[1];
        a.geo[k] = make_float4(rb.x, ra.z, ra.w, ra.x);
        a.key[k] = __float_as_int(rb.y) / TAB_ROW_BYTES;
        if (!a.dual) continue;
        const int i = a.erecv[k], j = a.col[k], m = a.atom_mol[i];
        Box bx;
        bx.periodic = (a.pbc != nullptr && a.box != nullptr && a.pbc[m]) ? 1 : 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            bx.L[q] = bx.periodic ? a.box[3 * m + q] : 1.0f;
            bx.invL[q] = __fdiv_rn(1.0f, bx.L[q]);
        }
        const float3 r = edge_vector(a.pos4[j], a.pos4[i], bx);
        float tx = 0.f, ty = 0.f, tz = 0.f;
        if (a.G) {   // a position direction leaves the image shift alone: r' = -(G_j - G_i)
            tx = a.G[3 * i] - a.G[3 * j];
            ty = a.G[3 * i + 1] - a.G[3 * j + 1];
            tz = a.G[3 * i + 2] - a.G[3 * j + 2];
        }
        if (a.S) {
            const double* S = a.S + 9 * m;
            tx += (float)(S[0] * r.x + S[1] * r.y + S[2] * r.z);
            ty += (float)(S[3] * r.x + S[4] * r.y + S[5] * r.z);
            tz += (float)(S[6] * r.x + S[7] * r.y + S[8] * r.z);
        }
        const float d = pair_distance(r.x, r.y, r.z);
        const float dt = d > 0.f ? (r.x * tx + r.y * ty + r.z * tz) / d : 0.f;   // 0 at the origin, as torch.norm
        // u = r / (d + 1e-8): u' = r' inv - r inv^2 d'
        const float inv = 1.0f / (d + 1e-8f), q = dt * inv * inv;
        const float4 u = make_float4(tx * inv - r.x * q, ty * inv - r.y * q, tz * inv - r.z * q, dt * a.scale);
        a.geo_t[k] = u;
        a.rec_t[p] = u;
    }
    if (a.dual && blockIdx.x == 0 && threadIdx.x < TREC_PAD) a.rec_t[E + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// --------------------------------------------- edges sorted by interval
// counts[interval][segment]; one warp per segment of SEG edges
__global__ void __launch_bounds__(128) sort_count_kernel(const int32_t* __restrict__ key,
                                                         const int32_t* __restrict__ row_ptr, int n_atoms, int nseg,
                                                         int32_t* __restrict__ counts, const Status* st) {
    __shared__ int hist[4][128];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int E = st->code != 0 ? 0 : row_ptr[n_atoms];
    const unsigned lt = (1u << lane) - 1u;
    for (int sg = blockIdx.x * 4 + w; sg < nseg; sg += gridDim.x * 4) {
        for (int q = lane; q < 128; q += 32) hist[w][q] = 0;
        __syncwarp();
        for (int k0 = sg * SEG; k0 < min(E, (sg + 1) * SEG); k0 += 32) {
            const int k = k0 + lane, kk = k < E ? key[k] : 127;
            const unsigned peers = __match_any_sync(0xffffffffu, kk);
            if ((peers & lt) == 0) hist[w][kk] += __popc(peers);
            __syncwarp();
        }
        for (int q = lane; q < TAB_NI; q += 32) counts[(int64_t)q * nseg + sg] = hist[w][q];
        __syncwarp();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[(int64_t)TAB_NI * nseg] = 0;
}

__global__ void __launch_bounds__(128) sort_place_kernel(const int32_t* __restrict__ key,
                                                         const int32_t* __restrict__ row_ptr, int n_atoms, int nseg,
                                                         const int32_t* __restrict__ offs, int32_t* __restrict__ order,
                                                         const Status* st) {
    __shared__ int next[4][128];
    if (st->code != 0) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int E = row_ptr[n_atoms];
    const unsigned lt = (1u << lane) - 1u;
    for (int sg = blockIdx.x * 4 + w; sg * SEG < E; sg += gridDim.x * 4) {
        for (int q = lane; q < TAB_NI; q += 32) next[w][q] = offs[(int64_t)q * nseg + sg];
        __syncwarp();
        for (int k0 = sg * SEG; k0 < min(E, (sg + 1) * SEG); k0 += 32) {
            const int k = k0 + lane, kk = k < E ? key[k] : 127;
            const unsigned peers = __match_any_sync(0xffffffffu, kk);
            const int at = next[w][kk];
            __syncwarp();
            if (k < E) order[at + __popc(peers & lt)] = k;
            if ((peers & lt) == 0) next[w][kk] = at + __popc(peers);
            __syncwarp();
        }
    }
}

// cst[i]: first chunk of interval i; cst[NI]: their number
__global__ void chunk_starts_kernel(const int32_t* __restrict__ offs, int nseg, int32_t* __restrict__ cst,
                                    const Status* st) {
    if (st->code != 0) {
        if (threadIdx.x <= TAB_NI) cst[threadIdx.x] = 0;
        return;
    }
    __shared__ int n[TAB_NI];
    if (threadIdx.x < TAB_NI)
        n[threadIdx.x] = (offs[(int64_t)(threadIdx.x + 1) * nseg] - offs[(int64_t)threadIdx.x * nseg] + CHUNK - 1) / CHUNK;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int i = 0; i < TAB_NI; ++i) {
            cst[i] = s;
            s += n[i];
        }
        cst[TAB_NI] = s;
    }
}

// ------------------------------------------------------- table adjoint
struct AdjArgs {
    const int32_t* order;
    const int32_t* offs;     // [NI * nseg + 1]
    const int32_t* cst;
    int nseg;
    const int32_t* col;
    const int32_t* erecv;
    const float4* geo;
    const float4* geo_t;
    const float* X;          // layer 0: s [N][H]; later layers quads
    const float* X_t;
    const float4* xtbar;     // quads
    const float4* xtbar_t;
    float* part;             // [chunk][18 (DUAL: 36)][H]
    float inv_scale;         // d' = t' / scale
    float node[TAB_NC];      // Chebyshev nodes
    float weight[TAB_NC];    // 1 / prod_{m != j} (node_j - node_m)
};

__device__ __forceinline__ void lagrange(const AdjArgs& a, float t, float (&L)[TAB_NC]) {
    float p[TAB_NC], q = 1.f;   // products over the nodes before j, then those after
#pragma unroll
    for (int j = 0; j < TAB_NC; ++j) {
        p[j] = q;
        q *= t - a.node[j];
    }
    q = 1.f;
#pragma unroll
    for (int j = TAB_NC - 1; j >= 0; --j) {
        L[j] = p[j] * q * a.weight[j];
        q *= t - a.node[j];
    }
}

// One block per chunk of edges of one interval, thread = channel: fbar_e =
// (ta.s x.s, ta.v . x.v, ta.v . u) (receiver adjoint ta, sender features x)
// times L_j(t).  DUAL: the adjoints of f (L_j fbar') and of f' = df/dd
// (L_j d' fbar) of the tangent f' d'.  Bound
// by the row gathers (4 KB per edge, 8 KB with tangents), four edges ahead.
template <bool DUAL, bool L0>
__global__ void __launch_bounds__(H) table_adjoint_kernel(AdjArgs a) {
    __shared__ int s_i[CHUNK], s_j[CHUNK];
    __shared__ float4 s_g[CHUNK], s_t[DUAL ? CHUNK : 1];
    __shared__ float s_l[CHUNK][TAB_NC];
    const int chunk = blockIdx.x, c = threadIdx.x;
    if (chunk >= a.cst[TAB_NI]) return;
    int lo = 0, hi = TAB_NI - 1;   // last interval whose first chunk is at or before this one
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.cst[mid] <= chunk) lo = mid;
        else hi = mid - 1;
    }
    const int p0 = a.offs[(int64_t)lo * a.nseg] + (chunk - a.cst[lo]) * CHUNK;
    const int n = min(CHUNK, a.offs[(int64_t)(lo + 1) * a.nseg] - p0);
    if (c < CHUNK) {
        const int k = a.order[p0 + min(c, n - 1)];
        s_i[c] = a.erecv[k];
        s_j[c] = a.col[k];
        s_g[c] = a.geo[k];
        if (DUAL) s_t[c] = a.geo_t[k];
        float l[TAB_NC];
        lagrange(a, s_g[c].w, l);
#pragma unroll
        for (int j = 0; j < TAB_NC; ++j) s_l[c][j] = l[j];
    }
    __syncthreads();
    float acc[3][TAB_NC], acd[DUAL ? 3 : 1][TAB_NC];
#pragma unroll
    for (int g = 0; g < 3; ++g)
#pragma unroll
        for (int k = 0; k < TAB_NC; ++k) acc[g][k] = acd[DUAL ? g : 0][k] = 0.f;
    const float4* T4 = a.xtbar + c;
    const float4* T4t = a.xtbar_t + c;
    const float4* X4 = reinterpret_cast<const float4*>(a.X) + c;
    const float4* X4t = reinterpret_cast<const float4*>(a.X_t) + c;
    const float* X1 = a.X + c;
#pragma unroll 4
    for (int e = 0; e < n; ++e) {
        const int64_t i = s_i[e], j = s_j[e];
        const float4 g = s_g[e];
        const float4 ta = __ldg(T4 + i * H);
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (L0) x.x = __ldg(X1 + j * H);
        else x = __ldg(X4 + j * H);
        float fb[3] = {ta.x * x.x, L0 ? 0.f : fmaf(ta.y, x.y, fmaf(ta.z, x.z, ta.w * x.w)),
                       fmaf(ta.y, g.x, fmaf(ta.z, g.y, ta.w * g.z))};
        if constexpr (!DUAL) {
#pragma unroll
            for (int k = 0; k < TAB_NC; ++k) {
                const float lk = s_l[e][k];
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if (!(L0 && f == 1)) acc[f][k] = fmaf(fb[f], lk, acc[f][k]);
            }
        } else {
            const float4 gt = s_t[e];
            const float dt = gt.w * a.inv_scale;
            const float4 tt = __ldg(T4t + i * H);
            float4 xt = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!L0) xt = __ldg(X4t + j * H);
            const float ft[3] = {
                fmaf(tt.x, x.x, ta.x * xt.x),
                L0 ? 0.f : fmaf(tt.y, x.y, fmaf(tt.z, x.z, tt.w * x.w)) + fmaf(ta.y, xt.y, fmaf(ta.z, xt.z, ta.w * xt.w)),
                fmaf(tt.y, g.x, fmaf(tt.z, g.y, tt.w * g.z)) + fmaf(ta.y, gt.x, fmaf(ta.z, gt.y, ta.w * gt.z))};
#pragma unroll
            for (int k = 0; k < TAB_NC; ++k) {
                const float lk = s_l[e][k];
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if (!(L0 && f == 1)) {
                        acc[f][k] = fmaf(ft[f], lk, acc[f][k]);
                        acd[f][k] = fmaf(fb[f] * dt, lk, acd[f][k]);
                    }
            }
        }
    }
    constexpr int ROWS = (DUAL ? 6 : 3) * TAB_NC;
    float* o = a.part + (int64_t)chunk * ROWS * H + c;
#pragma unroll
    for (int g = 0; g < 3; ++g)
#pragma unroll
        for (int k = 0; k < TAB_NC; ++k) {
            o[(g * TAB_NC + k) * H] = acc[g][k];
            if (DUAL) o[((3 + g) * TAB_NC + k) * H] = acd[DUAL ? g : 0][k];
        }
}

// Sums of the chunks' shares: out [NODES][3H], with two planes (DUAL) the
// adjoints of f' behind them.  Grid (interval, plane x filter x node).
__global__ void __launch_bounds__(H) node_adjoint_kernel(const float* __restrict__ part, const int32_t* __restrict__ cst,
                                                         int rows, float* __restrict__ out, const Status* st) {
    if (st->code != 0) return;
    const int i = blockIdx.x, row = blockIdx.y, c = threadIdx.x;
    const int plane = row / (3 * TAB_NC), g = row / TAB_NC % 3, j = row % TAB_NC;
    // two chains of compensated sums (Knuth's two-sum): the FP64 units are too
    // few for a sum per chunk
    float s[2] = {0.f, 0.f}, lo[2] = {0.f, 0.f};
    const float* p = part + (int64_t)row * H + c;
    const int64_t stride = (int64_t)rows * H;
    const int q1 = cst[i + 1];
    for (int q = cst[i]; q < q1; q += 8) {   // 8 loads in flight
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = q + u < q1 ? p[(q + u) * stride] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float t = __fadd_rn(s[u & 1], x[u]), z = __fsub_rn(t, s[u & 1]);
            lo[u & 1] = __fadd_rn(lo[u & 1],
                                  __fadd_rn(__fsub_rn(s[u & 1], __fsub_rn(t, z)), __fsub_rn(x[u], z)));
            s[u & 1] = t;
        }
    }
    out[(int64_t)plane * NODES * H3 + (int64_t)(i * TAB_NC + j) * H3 + g * H + c] =
        (float)(((double)s[0] + (double)s[1]) + ((double)lo[0] + (double)lo[1]));
}

// Adjoints of the network's hidden layer at the nodes, in place: of z =
// W1 e + b1 from hb = dE/dh, and (DUAL) with hd = dE/dh', h' = silu'(z) z':
//   zbar = hb silu'(z) + hd silu''(z) z',   zbar' = hd silu'(z)
template <bool DUAL>
__global__ void node_zbar_kernel(const float* __restrict__ z, const float* __restrict__ zd, float* __restrict__ hb,
                                 const Status* st) {
    if (st->code != 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NODES * H; i += gridDim.x * blockDim.x) {
        const float zz = z[i], d = dsilu_f(zz);
        float v = hb[i] * d;
        if (DUAL) {
            const float hd = hb[NODES * H + i];
            v = fmaf(hd, d2silu_f(zz) * zd[i], v);
            hb[NODES * H + i] = hd * d;
        }
        hb[i] = v;
    }
}

// ----------------------------------------------------- edge passes
enum { PASS_ADJ = 0, PASS_DUAL_FWD = 1, PASS_DUAL_ADJ = 2 };
struct PassArgs {
    const TabRec* rec;
    const float4* rec_t;
    const int32_t* row_ptr;
    int n_atoms;
    const float* tab;
    const float* A;          // value rows gathered: X (layer 0: s rows) or dE/dXt quads
    const float* A_t;        // their tangents (quads; layer 0 forward: none, they are zero)
    float* out;              // component-major rows
    Status* st;
};

// PASS_ADJ       out_i = A_i + sum_j A_j (phi_s, phi_v1)
// PASS_DUAL_ADJ  out_i = A'_i + sum_j A'_j (phi_s, phi_v1) + A_j (phi_s, phi_v1)'
// PASS_DUAL_FWD  the tangent of X_i + sum_j X_j (phi_s, phi_v1) + u phi_v2
// over receiver i's edges, sender j; the same walk as the table path's edge
// kernels.
template <int MODE, int G, bool SMEM, bool L0, int NT>
__global__ void __launch_bounds__(NT, SMEM ? 1 : 4) tab_pass_kernel(PassArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr bool DUAL = MODE != PASS_ADJ, FWD = MODE == PASS_DUAL_FWD;
    const int lane = threadIdx.x & 31;
    RecRing ring{smem + (SMEM ? TAB_RING : 0) + (threadIdx.x >> 5) * RING_BYTES, nullptr, lane};
    for_groups<SMEM>(a, G, smem, [&](int g, int slice) {
        const char* table = SMEM ? reinterpret_cast<const char*>(smem)
                                 : reinterpret_cast<const char*>(a.tab + slice * TAB_SLICE);
        const int ch = 32 * slice + lane;
        const int a0 = g * G;
        const int e0 = a.row_ptr[a0], n = a.row_ptr[min(a0 + G, a.n_atoms)] - e0;
        float acc[G][4];
#pragma unroll
        for (int r = 0; r < G; ++r)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[r][k] = 0.f;
        const float4* A4 = reinterpret_cast<const float4*>(a.A) + ch;
        const float4* T4 = reinterpret_cast<const float4*>(a.A_t) + ch;
        const float* A1 = a.A + ch;
        if (n > 0) {
            Coef c;
            int cur = -1;
            struct In {
                float4 x, xt, gt;
            };
            In ia[2], ib[2];
            auto gather = [&](In (&x)[2], int k, int u0) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int64_t j = ring.at(k, u0 + u)->sender;
                    if (FWD && L0) {
                        x[u].x = make_float4(__ldg(A1 + j * H), 0.f, 0.f, 0.f);
                        x[u].xt = make_float4(0.f, 0.f, 0.f, 0.f);
                    } else {
                        x[u].x = __ldg(A4 + j * H);
                        if (DUAL) x[u].xt = __ldg(T4 + j * H);
                    }
                    if (DUAL) x[u].gt = __ldg(a.rec_t + e0 + 4 * k + u0 + u);
                }
            };
            auto edge = [&](const TabRec* rp, const In& in) {
                const float4 ra = reinterpret_cast<const float4*>(rp)[0];
                const float2 rb = reinterpret_cast<const float2*>(rp)[2];
                const int off = __float_as_int(rb.y);
                if (uni(other_row(off, cur))) {
                    c.load<SMEM>(table, off, lane);
                    cur = off;
                }
                f32x2 sa, da;
                float m[4];
                if constexpr (!DUAL) {
                    sa = poly(c.sa, pack2(ra.x, ra.y));
                    m[0] = in.x.x * lo2(sa);
                    m[1] = in.x.y * hi2(sa);
                    m[2] = in.x.z * hi2(sa);
                    m[3] = in.x.w * hi2(sa);
                } else {
                    poly_d(c.sa, pack2(ra.x, ra.y), sa, da);
                    const float ds = lo2(da) * in.gt.w, d1 = hi2(da) * in.gt.w;   // phi' t'
                    m[0] = fmaf(in.xt.x, lo2(sa), in.x.x * ds);
                    m[1] = fmaf(in.xt.y, hi2(sa), in.x.y * d1);
                    m[2] = fmaf(in.xt.z, hi2(sa), in.x.z * d1);
                    m[3] = fmaf(in.xt.w, hi2(sa), in.x.w * d1);
                    if (FWD) {
                        float f2, d2;
                        poly_d(c.b, ra.x, f2, d2);
                        d2 *= in.gt.w;
                        m[1] = fmaf(in.gt.x, f2, fmaf(rb.x, d2, m[1]));
                        m[2] = fmaf(in.gt.y, f2, fmaf(ra.z, d2, m[2]));
                        m[3] = fmaf(in.gt.z, f2, fmaf(ra.w, d2, m[3]));
                    }
                }
                tab_switch<G>(off, [&](auto r) {
                    constexpr int R = decltype(r)::value;
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[R][k] += m[k];
                });
            };
            ring.src = a.rec + e0;
            tc::cp_async_wait_all();
            __syncwarp();
            ring.stage(0);
            ring.stage(1);
            ring.ready();
            ring.stage(2);
            gather(ia, 0, 0);
            const int full = n >> 2, left = n & 3;
#pragma unroll 1
            for (int k = 0; k < full; ++k) {
                gather(ib, k, 2);
                edge(ring.at(k, 0), ia[0]);
                edge(ring.at(k, 1), ia[1]);
                ring.ready();
                gather(ia, k + 1, 0);
                edge(ring.at(k, 2), ib[0]);
                edge(ring.at(k, 3), ib[1]);
                ring.stage(k + 3);
            }
            gather(ib, full, 2);
#pragma unroll 1
            for (int u = 0; u < left; ++u) {
                edge(ring.at(full, u), ia[0]);
                ia[0] = ia[1];
                ia[1] = ib[0];
            }
        }
#pragma unroll
        for (int r = 0; r < G; ++r) {
            if (a0 + r >= a.n_atoms) break;
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!(FWD && L0)) b = DUAL ? T4[(int64_t)(a0 + r) * H] : A4[(int64_t)(a0 + r) * H];
            float* o = a.out + (int64_t)(a0 + r) * 4 * H + ch;
            o[0] = b.x + acc[r][0];
            o[H] = b.y + acc[r][1];
            o[2 * H] = b.z + acc[r][2];
            o[3 * H] = b.w + acc[r][3];
        }
    });
    tc::cp_async_wait_all();
}

template <int MODE, int G, bool SMEM, bool L0>
int launch_pass_t(const PassArgs& a, cudaStream_t st) {
    constexpr int NT = SMEM ? BWD_NT : SMALL_NT;
    using TL = TabLaunch<G, SMEM, NT>;
    static std::once_flag once;
    static int err = MLFF_OK;
    std::call_once(once, [] { err = TL::prepare(tab_pass_kernel<MODE, G, SMEM, L0, NT>); });
    if (err) return err;
    MLFF_LAUNCH_PDL("tab_pass", (tab_pass_kernel<MODE, G, SMEM, L0, NT>), TL::grid(a.n_atoms), NT, TL::SM, st, a);
    return MLFF_OK;
}
template <int MODE, bool L0>
int launch_pass(const PassArgs& a, cudaStream_t st) {
    ProfScope prof(PK_PLAIN_EDGE, st);
    const TabShape s = tab_shape(a.n_atoms, MLFF_PATH_TRAIN_TABLE);
    if (s.smem) return launch_pass_t<MODE, 1, true, L0>(a, st);
    return launch_pass_t<MODE, 1, false, L0>(a, st);
}

// ------------------------------------------------------ per-atom kernels
// (thread = atom and channel; planes of n = N rows: value, then tangent)

// comb = [s, |v|] and its tangent from Xt rows; with uz also h = silu(z) and
// its tangent (the inputs of the update MLP's two layers)
template <bool DUAL>
__global__ void node_inputs_kernel(const float* __restrict__ Xt, const float* __restrict__ Xt_t,
                                   const float* __restrict__ uz, const float* __restrict__ uz_t, int n_atoms,
                                   int want_value, float* __restrict__ comb, float* __restrict__ h, const Status* st) {
    if (st->code != 0) return;
    const int64_t total = (int64_t)n_atoms * H;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i / H;
        const int c = (int)(i % H);
        const float* x = Xt + a * 4 * H + c;
        const float v0 = x[H], v1 = x[2 * H], v2 = x[3 * H];
        const float n = pair_distance(v0, v1, v2);
        if (want_value) {
            comb[a * 2 * H + c] = x[0];
            comb[a * 2 * H + H + c] = n;
            if (uz) h[i] = silu_f(uz[i]);
        }
        if (DUAL) {
            const float* y = Xt_t + a * 4 * H + c;
            float* ct = comb + (want_value ? (int64_t)n_atoms * 2 * H : 0) + a * 2 * H + c;
            ct[0] = y[0];
            ct[H] = n > 0.f ? (v0 * y[H] + v1 * y[2 * H] + v2 * y[3 * H]) / n : 0.f;
            if (uz) h[(int64_t)n_atoms * H + i] = dsilu_f(uz[i]) * uz_t[i];
        }
    }
}

// h' = silu'(z) z'
__global__ void dsilu_mul_kernel(const float* __restrict__ z, const float* __restrict__ zt, int64_t n,
                                 float* __restrict__ out, const Status* st) {
    if (st->code != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = dsilu_f(z[i]) * zt[i];
}

// tangent of s + ds, v g1 + (M v) g2; out quads or (last layer) rows
__global__ void update_out_tangent_kernel(const float* __restrict__ Xt, const float* __restrict__ Xt_t,
                                          const float* __restrict__ ua, const float* __restrict__ ua_t,
                                          const float* __restrict__ mix_g, int n_atoms, int quads,
                                          float* __restrict__ out, const Status* st) {
    if (st->code != 0) return;
    float M[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) M[q] = mix_g[q];
    const int64_t total = (int64_t)n_atoms * H;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i / H;
        const int c = (int)(i % H);
        const float *x = Xt + a * 4 * H + c, *y = Xt_t + a * 4 * H + c, *u = ua + a * H3 + c, *ut = ua_t + a * H3 + c;
        float v[3], w[3], o[4];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            v[q] = x[(1 + q) * H];
            w[q] = y[(1 + q) * H];
        }
        o[0] = y[0] + ut[0];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float mv = M[3 * q] * v[0] + M[3 * q + 1] * v[1] + M[3 * q + 2] * v[2];
            const float mw = M[3 * q] * w[0] + M[3 * q + 1] * w[1] + M[3 * q + 2] * w[2];
            o[1 + q] = (w[q] * u[H] + v[q] * ut[H]) + (mw * u[2 * H] + mv * ut[2 * H]);
        }
        if (quads) {
            reinterpret_cast<float4*>(out + a * 4 * H)[c] = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) out[a * 4 * H + q * H + c] = o[q];
        }
    }
}

// reverse of the gates and the mixing: abar = dE/d(ds, g1, g2) and its tangent
template <bool DUAL>
__global__ void update_abar_kernel(const float* __restrict__ Xt, const float* __restrict__ Xt_t,
                                   const float* __restrict__ xb, const float* __restrict__ xb_t,
                                   const float* __restrict__ mix_g, int n_atoms, float* __restrict__ abar,
                                   const Status* st) {
    if (st->code != 0) return;
    float M[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) M[q] = mix_g[q];
    const int64_t total = (int64_t)n_atoms * H;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i / H;
        const int c = (int)(i % H);
        const float *x = Xt + a * 4 * H + c, *b = xb + a * 4 * H + c;
        float g1 = 0.f, g2 = 0.f, g1t = 0.f, g2t = 0.f;
        float v[3], w[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            v[q] = x[(1 + q) * H];
            if (DUAL) w[q] = Xt_t[a * 4 * H + (1 + q) * H + c];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float vb = b[(1 + q) * H];
            const float mv = M[3 * q] * v[0] + M[3 * q + 1] * v[1] + M[3 * q + 2] * v[2];
            g1 = fmaf(vb, v[q], g1);
            g2 = fmaf(vb, mv, g2);
            if (DUAL) {
                const float vbt = xb_t[a * 4 * H + (1 + q) * H + c];
                const float mw = M[3 * q] * w[0] + M[3 * q + 1] * w[1] + M[3 * q + 2] * w[2];
                g1t = fmaf(vbt, v[q], fmaf(vb, w[q], g1t));
                g2t = fmaf(vbt, mv, fmaf(vb, mw, g2t));
            }
        }
        float* o = abar + a * H3 + c;
        o[0] = b[0];
        o[H] = g1;
        o[2 * H] = g2;
        if (DUAL) {
            o += (int64_t)n_atoms * H3;
            o[0] = xb_t[a * 4 * H + c];
            o[H] = g1t;
            o[2 * H] = g2t;
        }
    }
}

// in place: zbar = hbar silu'(z) and its tangent
template <bool DUAL>
__global__ void zbar_kernel(const float* __restrict__ z, const float* __restrict__ zt, int64_t n,
                            float* __restrict__ hb, const Status* st) {
    if (st->code != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float zz = z[i], d = dsilu_f(zz), h = hb[i];
        hb[i] = h * d;
        if (DUAL) hb[n + i] = fmaf(hb[n + i], d, h * d2silu_f(zz) * zt[i]);
    }
}

// dE/dXt = (sb + cs, xb g1 + M^T xb g2 + cn v / |v|) and its tangent, quads
template <bool DUAL>
__global__ void update_in_adjoint_kernel(const float* __restrict__ Xt, const float* __restrict__ Xt_t,
                                         const float* __restrict__ ua, const float* __restrict__ ua_t,
                                         const float* __restrict__ xb, const float* __restrict__ xb_t,
                                         const float* __restrict__ cb, const float* __restrict__ mix_g, int n_atoms,
                                         float4* __restrict__ out, float4* __restrict__ out_t, const Status* st) {
    if (st->code != 0) return;
    float M[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) M[q] = mix_g[q];
    const int64_t total = (int64_t)n_atoms * H;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i / H;
        const int c = (int)(i % H);
        const float *x = Xt + a * 4 * H + c, *b = xb + a * 4 * H + c, *u = ua + a * H3 + c, *k = cb + a * 2 * H + c;
        float v[3], vb[3], o[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            v[q] = x[(1 + q) * H];
            vb[q] = b[(1 + q) * H];
        }
        const float g1 = u[H], g2 = u[2 * H], n = pair_distance(v[0], v[1], v[2]);
        const float sc = n > 0.f ? k[H] / n : 0.f;   // d|v|/dv = v / |v|, 0 at v = 0
        float mb[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            mb[q] = M[q] * vb[0] + M[3 + q] * vb[1] + M[6 + q] * vb[2];
            o[q] = vb[q] * g1 + mb[q] * g2 + sc * v[q];
        }
        out[i] = make_float4(b[0] + k[0], o[0], o[1], o[2]);
        if (DUAL) {
            const float *y = Xt_t + a * 4 * H + c, *bt = xb_t + a * 4 * H + c, *ut = ua_t + a * H3 + c;
            const float* kt = cb + ((int64_t)n_atoms + a) * 2 * H + c;
            float w[3], vbt[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                w[q] = y[(1 + q) * H];
                vbt[q] = bt[(1 + q) * H];
            }
            const float nt = n > 0.f ? (v[0] * w[0] + v[1] * w[1] + v[2] * w[2]) / n : 0.f;
            const float sct = n > 0.f ? (kt[H] - sc * nt) / n : 0.f;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float mbt = M[q] * vbt[0] + M[3 + q] * vbt[1] + M[6 + q] * vbt[2];
                o[q] = (vbt[q] * g1 + vb[q] * ut[H]) + (mbt * g2 + mb[q] * ut[2 * H]) + (sct * v[q] + sc * w[q]);
            }
            out_t[i] = make_float4(bt[0] + kt[0], o[0], o[1], o[2]);
        }
    }
}

// mixing matrix: dM_ij = sum_{a,c} xb_{v_i} g2 v_j (DUAL: its tangent),
// per-block partials, then a fixed-order sum
template <bool DUAL>
__global__ void __launch_bounds__(256) mix_adjoint_kernel(const float* __restrict__ Xt, const float* __restrict__ Xt_t,
                                                          const float* __restrict__ ua, const float* __restrict__ ua_t,
                                                          const float* __restrict__ xb, const float* __restrict__ xb_t,
                                                          int n_atoms, float* __restrict__ part, const Status* st) {
    __shared__ float red[8][9];
    if (st->code != 0) return;
    float acc[9] = {};
    const int64_t total = (int64_t)n_atoms * H;
    for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const int64_t a = i / H;
        const int c = (int)(i % H);
        const float *x = Xt + a * 4 * H + c, *b = xb + a * 4 * H + c;
        const float g2 = ua[a * H3 + 2 * H + c];
        float v[3], w[3], gt = 0.f;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            v[q] = x[(1 + q) * H];
            if (DUAL) w[q] = Xt_t[a * 4 * H + (1 + q) * H + c];
        }
        if (DUAL) gt = ua_t[a * H3 + 2 * H + c];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const float vb = b[(1 + r) * H];
            if (!DUAL) {
                const float t = vb * g2;
#pragma unroll
                for (int q = 0; q < 3; ++q) acc[3 * r + q] = fmaf(t, v[q], acc[3 * r + q]);
            } else {
                const float t = vb * g2, tt = fmaf(xb_t[a * 4 * H + (1 + r) * H + c], g2, vb * gt);
#pragma unroll
                for (int q = 0; q < 3; ++q) acc[3 * r + q] = fmaf(tt, v[q], fmaf(t, w[q], acc[3 * r + q]));
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = acc[k];
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
        part[blockIdx.x * 9 + threadIdx.x] = s;
    }
}
__global__ void mix_sum_kernel(const float* __restrict__ part, int blocks, int acc, float* __restrict__ out,
                               const Status* st) {
    if (st->code != 0) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;   // warp = entry
    double s = 0.0;
    for (int b = lane; b < blocks; b += 32) s += (double)part[b * 9 + w];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[w] = (acc ? out[w] : 0.f) + (float)s;
}

// energy head: h1' = silu'(z1) z1' ; a2 = w w3 silu'(z2) (and tangent), the
// rows w h2 (value) or h2' (tangent) of head_w3's gradient
__global__ void head_mid_kernel(const float* __restrict__ z2, const float* __restrict__ z2t,
                                const float* __restrict__ w3, const double* __restrict__ w,
                                const int32_t* __restrict__ atom_mol, int n_atoms, float* __restrict__ a2,
                                float* __restrict__ h2w, float* __restrict__ wcol, const Status* st) {
    if (st->code != 0) return;
    const int64_t total = (int64_t)n_atoms * 32;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i / 32;
        const int o = (int)(i % 32);
        const float ww = w ? (float)w[atom_mol[a]] : 1.0f, z = z2[i], d = dsilu_f(z);
        a2[i] = ww * w3[o] * d;
        if (z2t) {
            a2[total + i] = w3[o] * d2silu_f(z) * z2t[i];
            h2w[i] = d * z2t[i];
        } else {
            h2w[i] = ww * silu_f(z);
            if (o == 0) wcol[a] = ww;
        }
    }
}
// adjoint rows (s part, then zeros) from the head's dE/ds
__global__ void head_seed_kernel(const float* __restrict__ sbar, int64_t rows, float* __restrict__ xbar,
                                 const Status* st) {
    if (st->code != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows * 4 * H;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = i / (4 * H);
        const int q = (int)(i % (4 * H));
        xbar[i] = q < H ? sbar[a * H + q] : 0.f;
    }
}

// dEmb[z] = sum of the adjoint's s rows of the atoms of species z: blocks of
// (species, share of the atoms); each finds its atoms by ballots, sums their
// rows in atom order
constexpr int EMB_SPLIT = 16;
__global__ void __launch_bounds__(H) embed_part_kernel(const int64_t* __restrict__ Z, const float* __restrict__ xbar,
                                                       int n_atoms, int n_species, float* __restrict__ part,
                                                       const Status* st) {
    __shared__ int list[H];
    __shared__ int cnt[4];
    if (st->code != 0) return;
    const int z = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int per = (n_atoms + EMB_SPLIT - 1) / EMB_SPLIT;
    const int b0 = blockIdx.y * per, b1 = min(n_atoms, b0 + per);
    float s = 0.f;
    for (int a0 = b0; a0 < b1; a0 += H) {
        const int a = a0 + t;
        const bool hit = a < b1 && Z[a] == z;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) cnt[w] = __popc(m);
        __syncthreads();
        int base = 0;
        for (int q = 0; q < w; ++q) base += cnt[q];
        if (hit) list[base + __popc(m & ((1u << lane) - 1u))] = a;
        const int n = cnt[0] + cnt[1] + cnt[2] + cnt[3];
        __syncthreads();
#pragma unroll 8
        for (int q = 0; q < n; ++q) s += xbar[(int64_t)list[q] * 4 * H + t];
        __syncthreads();
    }
    part[((int64_t)blockIdx.y * n_species + z) * H + t] = s;
}
__global__ void embed_sum_kernel(const float* __restrict__ part, int64_t n, int acc, float* __restrict__ out,
                                 const Status* st) {
    if (st->code != 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < EMB_SPLIT; ++q) s += part[q * n + i];
        out[i] = acc ? out[i] + s : s;
    }
}

// layer inputs 0 .. n_layers - 1 from component-major rows to the gather
// layout: layer 0 the s rows alone, the others quads
__global__ void rows_to_gather_kernel(const float* __restrict__ rows, int n_atoms, int n_layers, float* __restrict__ X,
                                      const Status* st) {
    if (st->code != 0) return;
    const int64_t per = (int64_t)n_atoms * H, total = per * n_layers;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t l = i / per, k = i % per, a = k / H;
        const int c = (int)(k % H);
        const float* x = rows + l * per * 4 + a * 4 * H + c;
        if (l == 0) X[k] = x[0];
        else reinterpret_cast<float4*>(X + l * per * 4)[k] = make_float4(x[0], x[H], x[2 * H], x[3 * H]);
    }
}

#define TT_LAUNCH(kernel, n, ...)                           \
    do {                                                    \
        kernel<<<blocks_for(n), 256, 0, st>>>(__VA_ARGS__); \
        MLFF_LAUNCH_CHECK(#kernel);                         \
    } while (0)

// The whole pass.  DUAL false: gradients written, seeded with w (grad.w);
// DUAL true: their tangent along (-G, S) added, unit seeds.
template <bool DUAL>
int run_train(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys, const WsLayout& L,
              void* ws, double* energy, cudaStream_t st, const GradCtx& grad, const float* G, const double* S) {
    const int N = L.N;
    const int64_t NX = (int64_t)N * 4 * H, NH = (int64_t)N * H;
    const int planes = DUAL ? 2 : 1;
    const int64_t rows = (int64_t)planes * N;
    Status* status = ws_ptr<Status>(ws, L.status);
    const int32_t* row_ptr = ws_ptr<int32_t>(ws, L.row_ptr);
    const int32_t *col = ws_ptr<int32_t>(ws, L.col), *erecv = ws_ptr<int32_t>(ws, L.erecv);
    // per layer arrays: values first, then tangents
    float *X = ws_ptr<float>(ws, L.X), *X_t = X + (int64_t)(L.L + 1) * NX;
    float *Xt = ws_ptr<float>(ws, L.Xt), *Xt_t = Xt + (int64_t)L.L * NX;
    float *uz = ws_ptr<float>(ws, L.uz), *uz_t = uz + (int64_t)L.L * NH;
    float *ua = ws_ptr<float>(ws, L.ua), *ua_t = ua + (int64_t)L.L * N * H3;
    float *xb = ws_ptr<float>(ws, L.xbar), *xb_t = xb + NX;        // dE/dX rows
    float4 *tb = ws_ptr<float4>(ws, L.txtbar), *tb_t = tb + NH;    // dE/dXt quads
    float *comb = ws_ptr<float>(ws, L.comb), *hbuf = ws_ptr<float>(ws, L.uh), *abar = ws_ptr<float>(ws, L.abar);
    float *hb = ws_ptr<float>(ws, L.thb), *cb = ws_ptr<float>(ws, L.tcb), *gpart = ws_ptr<float>(ws, L.gpart);
    float4 *geo = ws_ptr<float4>(ws, L.geo), *geo_t = ws_ptr<float4>(ws, L.tgeo_t), *rec_t = ws_ptr<float4>(ws, L.trec_t);
    int32_t *key = ws_ptr<int32_t>(ws, L.tkey), *order = ws_ptr<int32_t>(ws, L.torder);
    int32_t *offs = ws_ptr<int32_t>(ws, L.toffs), *cst = ws_ptr<int32_t>(ws, L.tcst);
    const int nseg = (int)((L.cap + SEG - 1) / SEG);
    const float scale = tab_scale(d.cutoff);
    const bool acc = DUAL;
    int r;

    // Value forward pass (records, X, Xt, uz, ua of every layer): the plain
    // path's, bit for bit (see the head of the file).
    if ((r = launch_records(d, P, po, sys, L, ws, MLFF_PATH_TRAIN_TABLE, st))) return r;
    {
        float* rowsX = ws_ptr<float>(ws, L.prows);   // [L + 1][N][4][H]
        if ((r = plain_forward(d, P, po, sys, L, ws, rowsX, st))) return r;
        TT_LAUNCH(rows_to_gather_kernel, (int64_t)L.L * NH, rowsX, N, L.L, X, status);
        MLFF_CUDA(cudaMemcpyAsync(X + L.L * NX, rowsX + L.L * NX, sizeof(float) * NX, cudaMemcpyDeviceToDevice, st));
    }
    {
        ProfScope prof(PK_OTHER, st);
        const MapArgs m{ws_ptr<TabRec>(ws, L.trec), ws_ptr<int32_t>(ws, L.tperm), row_ptr, col, erecv,
                        ws_ptr<float4>(ws, L.pos4), ws_ptr<int32_t>(ws, L.atom_mol), sys.box, sys.pbc, G, S, scale, N,
                        DUAL ? 1 : 0, geo, key, geo_t, rec_t, status};
        TT_LAUNCH(edge_maps_kernel, L.cap, m);
        const int sb = std::max(1, std::min((nseg + 3) / 4, num_sms() * 16));
        sort_count_kernel<<<sb, 128, 0, st>>>(key, row_ptr, N, nseg, offs, status);
        MLFF_LAUNCH_CHECK("sort_count");
        if ((r = launch_scan(offs, (int64_t)TAB_NI * nseg + 1, ws_ptr<int32_t>(ws, L.tscan), st))) return r;
        sort_place_kernel<<<sb, 128, 0, st>>>(key, row_ptr, N, nseg, offs, order, status);
        MLFF_LAUNCH_CHECK("sort_place");
        chunk_starts_kernel<<<1, 128, 0, st>>>(offs, nseg, cst, status);
        MLFF_LAUNCH_CHECK("chunk_starts");
    }
    if constexpr (DUAL) {   // tangent forward pass
        for (int l = 0; l < L.L; ++l) {
            const LayerOffsets& lo = po.layer[l];
            const PassArgs pa{ws_ptr<TabRec>(ws, L.trec), rec_t, row_ptr, N, P + po.tab + l * TAB_LAYER, X + l * NX,
                              X_t + l * NX, Xt_t + l * NX, status};
            if ((r = l == 0 ? launch_pass<PASS_DUAL_FWD, true>(pa, st) : launch_pass<PASS_DUAL_FWD, false>(pa, st)))
                return r;
            TT_LAUNCH(node_inputs_kernel<true>, NH, Xt + l * NX, Xt_t + l * NX, nullptr, nullptr, N, 0, comb, nullptr,
                      status);
            if ((r = gemm_nn(0, comb, P + lo.u1t, nullptr, uz_t + l * NH, nullptr, nullptr, N, nullptr, H, 2 * H, status,
                             st))) return r;
            TT_LAUNCH(dsilu_mul_kernel, NH, uz + l * NH, uz_t + l * NH, NH, hbuf, status);
            if ((r = gemm_nn(0, hbuf, P + lo.u2t, nullptr, ua_t + l * N * H3, nullptr, nullptr, N, nullptr, H3, H,
                             status, st))) return r;
            TT_LAUNCH(update_out_tangent_kernel, NH, Xt + l * NX, Xt_t + l * NX, ua + (int64_t)l * N * H3,
                      ua_t + (int64_t)l * N * H3, P + lo.mix, N, l + 1 < L.L, X_t + (l + 1) * NX, status);
        }
    } else {
        mlff_outputs out{energy, nullptr, nullptr, nullptr};
        if ((r = launch_readout(d, P, po, sys, L, ws, out, 0, st))) return r;
    }
    {   // energy head: activations, adjoints and gradients
        ProfScope prof(PK_READOUT, st);
        const float *XL = X + L.L * NX, *XL_t = X_t + L.L * NX;
        float* z1 = ws_ptr<float>(ws, L.thead);         // [planes][N][64] each: z1, h1, hb1
        float *h1 = z1 + 2LL * N * 64, *b1 = h1 + 2LL * N * 64;
        float *z2 = b1 + 2LL * N * 64, *a2 = z2 + 2LL * N * 32, *h2w = a2 + 2LL * N * 32, *wcol = h2w + (int64_t)N * 32;
        float *z1t = z1 + (int64_t)N * 64, *h1t = h1 + (int64_t)N * 64, *z2t = z2 + (int64_t)N * 32;
        if ((r = gemm_nn(1, XL, P + po.head_w1t, P + po.head_b1, z1, h1, nullptr, N, nullptr, 64, H, status, st, 4 * H)))
            return r;
        if ((r = gemm_nn(0, h1, P + po.head_w2t, P + po.head_b2, z2, nullptr, nullptr, N, nullptr, 32, 64, status, st)))
            return r;
        if (DUAL) {
            if ((r = gemm_nn(0, XL_t, P + po.head_w1t, nullptr, z1t, nullptr, nullptr, N, nullptr, 64, H, status, st,
                             4 * H))) return r;
            TT_LAUNCH(dsilu_mul_kernel, (int64_t)N * 64, z1, z1t, (int64_t)N * 64, h1t, status);
            if ((r = gemm_nn(0, h1t, P + po.head_w2t, nullptr, z2t, nullptr, nullptr, N, nullptr, 32, 64, status, st)))
                return r;
        }
        TT_LAUNCH(head_mid_kernel, (int64_t)N * 32, z2, DUAL ? z2t : nullptr, P + po.head_w3, grad.w,
                  ws_ptr<int32_t>(ws, L.atom_mol), N, a2, h2w, wcol, status);
        if ((r = gemm_nn(0, a2, P + po.head_w2, nullptr, b1, nullptr, nullptr, rows, nullptr, 64, 32, status, st)))
            return r;
        TT_LAUNCH(zbar_kernel<DUAL>, (int64_t)N * 64, z1, z1t, (int64_t)N * 64, b1, status);
        // dE/ds through cb ([planes][N][H])
        if ((r = gemm_nn(0, b1, P + po.head_w1, nullptr, cb, nullptr, nullptr, rows, nullptr, H, 64, status, st)))
            return r;
        TT_LAUNCH(head_seed_kernel, rows * 4 * H, cb, rows, xb, status);
        auto set = [&](const float* A, const float* B, int64_t pa, int64_t pb) {
            return DUAL ? GemmRows{A + pa, B, A, B + pb} : GemmRows{A, B};
        };
        const mlff_grads& g = grad.g;
        if (g.head_w1 || g.head_b1) {
            GemmRows x = DUAL ? GemmRows{b1 + (int64_t)N * 64, XL, b1, XL_t} : GemmRows{b1, XL};
            if ((r = gemm_tn(x, 64, 4 * H, 64, H, N, g.head_w1, g.head_b1, acc, gpart, status, st))) return r;
        }
        if (g.head_w2 || g.head_b2)
            if ((r = gemm_tn(set(a2, h1, (int64_t)N * 32, (int64_t)N * 64), 32, 64, 32, 64, N, g.head_w2, g.head_b2, acc,
                             gpart, status, st))) return r;
        if (g.head_w3)
            if ((r = gemm_tn({h2w, nullptr}, 32, 1, 32, 0, N, nullptr, g.head_w3, acc, gpart, status, st))) return r;
        if (!DUAL && g.head_b3)
            if ((r = gemm_tn({wcol, nullptr}, 1, 1, 1, 0, N, nullptr, g.head_b3, acc, gpart, status, st))) return r;
    }
    float* nodes = ws_ptr<float>(ws, L.tnode);          // [NODES][3H], then [NODES][H]
    float* node_zb = nodes + 2LL * NODES * H3;         // [planes][NODES][H]
    for (int l = L.L - 1; l >= 0; --l) {
        const LayerOffsets& lo = po.layer[l];
        const mlff_grads& g = grad.g;
        const float *xt = Xt + l * NX, *xt_t = Xt_t + l * NX, *z = uz + l * NH, *zt = uz_t + l * NH;
        const float *u = ua + (int64_t)l * N * H3, *u_t = ua_t + (int64_t)l * N * H3;
        TT_LAUNCH(update_abar_kernel<DUAL>, NH, xt, xt_t, xb, xb_t, P + lo.mix, N, abar, status);
        TT_LAUNCH(node_inputs_kernel<DUAL>, NH, xt, xt_t, z, zt, N, 1, comb, hbuf, status);
        if (g.update_w2[l] || g.update_b2[l]) {
            GemmRows x = DUAL ? GemmRows{abar + (int64_t)N * H3, hbuf, abar, hbuf + NH} : GemmRows{abar, hbuf};
            if ((r = gemm_tn(x, H3, H, H3, H, N, g.update_w2[l], g.update_b2[l], acc, gpart, status, st))) return r;
        }
        if (g.mixing[l]) {
            float* part = ws_ptr<float>(ws, L.gmix);
            mix_adjoint_kernel<DUAL><<<GRAD_MIX_BLOCKS, 256, 0, st>>>(xt, xt_t, u, u_t, xb, xb_t, N, part, status);
            MLFF_LAUNCH_CHECK("mix_adjoint");
            mix_sum_kernel<<<1, 9 * 32, 0, st>>>(part, GRAD_MIX_BLOCKS, acc ? 1 : 0, g.mixing[l], status);
            MLFF_LAUNCH_CHECK("mix_sum");
        }
        if ((r = gemm_nn(0, abar, P + lo.u2, nullptr, hb, nullptr, nullptr, rows, nullptr, H, H3, status, st))) return r;
        TT_LAUNCH(zbar_kernel<DUAL>, NH, z, zt, NH, hb, status);
        if (g.update_w1[l] || g.update_b1[l]) {
            GemmRows x = DUAL ? GemmRows{hb + NH, comb, hb, comb + (int64_t)N * 2 * H} : GemmRows{hb, comb};
            if ((r = gemm_tn(x, H, 2 * H, H, 2 * H, N, g.update_w1[l], g.update_b1[l], acc, gpart, status, st))) return r;
        }
        if ((r = gemm_nn(0, hb, P + lo.u1, nullptr, cb, nullptr, nullptr, rows, nullptr, 2 * H, H, status, st))) return r;
        TT_LAUNCH(update_in_adjoint_kernel<DUAL>, NH, xt, xt_t, u, u_t, xb, xb_t, cb, P + lo.mix, N, tb, tb_t, status);
        // filter network: table adjoint, then the network's reverse pass at the nodes
        if (g.filter_w1[l] || g.filter_b1[l] || g.filter_w2[l] || g.filter_b2[l]) {
            float* apart = ws_ptr<float>(ws, L.tadj);
            AdjArgs aa{order, offs, cst, nseg, col, erecv, geo, geo_t, X + l * NX, X_t + l * NX, tb, tb_t, apart,
                             1.0f / scale, {}, {}};
            table_nodes(aa.node, aa.weight);
            const int nblk = (int)(L.cap / CHUNK + TAB_NI + 1);
            {
                ProfScope prof(PK_PLAIN_EDGE, st);
                if (l == 0) table_adjoint_kernel<DUAL, true><<<nblk, H, 0, st>>>(aa);
                else table_adjoint_kernel<DUAL, false><<<nblk, H, 0, st>>>(aa);
                MLFF_LAUNCH_CHECK("table_adjoint");
                node_adjoint_kernel<<<dim3(TAB_NI, planes * 3 * TAB_NC), H, 0, st>>>(apart, cst, planes * 3 * TAB_NC, nodes,
                                                                                     status);
                MLFF_LAUNCH_CHECK("node_adjoint");
            }
            // z, h, z', h' [NODES][H], e, e' [NODES][RMAX]
            const float* nz = P + po.tab_node + (int64_t)l * TAB_NODE_LAYER;
            const float *nh = nz + (int64_t)NODES * H, *nzd = nh + (int64_t)NODES * H, *nhd = nzd + (int64_t)NODES * H;
            const float *ne = nhd + (int64_t)NODES * H, *ned = ne + (int64_t)NODES * RMAX;
            if (g.filter_w2[l] || g.filter_b2[l]) {
                GemmRows x = DUAL ? GemmRows{nodes, nh, nodes + (int64_t)NODES * H3, nhd} : GemmRows{nodes, nh};
                if ((r = gemm_tn(x, H3, H, H3, H, NODES, g.filter_w2[l], g.filter_b2[l], acc, gpart, status, st)))
                    return r;
            }
            if (g.filter_w1[l] || g.filter_b1[l]) {
                if ((r = gemm_nn(0, nodes, P + lo.w2, nullptr, node_zb, nullptr, nullptr, (int64_t)planes * NODES,
                                 nullptr, H, H3, status, st))) return r;
                TT_LAUNCH(node_zbar_kernel<DUAL>, (int64_t)NODES * H, nz, nzd, node_zb, status);
                GemmRows x = DUAL ? GemmRows{node_zb, ne, node_zb + (int64_t)NODES * H, ned} : GemmRows{node_zb, ne};
                if ((r = gemm_tn(x, H, RMAX, H, d.n_rbf, NODES, g.filter_w1[l], g.filter_b1[l], acc, gpart, status,
                                 st))) return r;
            }
        }
        // dE/dX of the layer's input
        if (l > 0 || g.embedding) {
            PassArgs pa{ws_ptr<TabRec>(ws, L.trec), rec_t, row_ptr, N, P + po.tab + l * TAB_LAYER,
                        reinterpret_cast<const float*>(tb), reinterpret_cast<const float*>(tb_t), nullptr, status};
            if constexpr (DUAL) {
                pa.out = xb_t;
                if ((r = launch_pass<PASS_DUAL_ADJ, false>(pa, st))) return r;
            }
            if (!DUAL || l > 0) {
                pa.out = xb;
                if ((r = launch_pass<PASS_ADJ, false>(pa, st))) return r;
            }
        }
    }
    if (grad.g.embedding) {
        ProfScope prof(PK_OTHER, st);
        float* part = ws_ptr<float>(ws, L.temb);
        embed_part_kernel<<<dim3(d.n_species, EMB_SPLIT), H, 0, st>>>(sys.Z, DUAL ? xb_t : xb, N, d.n_species, part, status);
        MLFF_LAUNCH_CHECK("embed_part");
        const int64_t n = (int64_t)d.n_species * H;
        TT_LAUNCH(embed_sum_kernel, n, part, n, acc ? 1 : 0, grad.g.embedding, status);
    }
    return MLFF_OK;
}

}  // namespace

static size_t take_bytes(size_t& p, size_t bytes) {
    const size_t q = p;
    p += (bytes + 255) & ~size_t(255);
    return q;
}

size_t train_forward_workspace(WsLayout& L, size_t p) {
    const int64_t pairs = L.cap / 2 + 1;   // filters by pair of atoms
    L.erbf = take_bytes(p, sizeof(float) * pairs * RMAX);
    L.fh = take_bytes(p, sizeof(float) * pairs * H);
    L.ff = take_bytes(p, sizeof(float) * pairs * H3);
    L.pgeo = take_bytes(p, sizeof(float4) * L.cap);
    return p;
}

size_t train_table_workspace(WsLayout& L, const mlff_dims& d, size_t p) {
    auto take = [&](size_t bytes) { return take_bytes(p, bytes); };
    const int64_t N = L.N, nseg = (L.cap + SEG - 1) / SEG;
    const int64_t nscan = (int64_t)TAB_NI * nseg + 1;
    L.txtbar = take(sizeof(float4) * 2 * N * H);
    L.comb = take(sizeof(float) * 2 * N * 2 * H);
    L.uh = take(sizeof(float) * 2 * N * H);
    L.abar = take(sizeof(float) * 2 * N * H3);
    L.thb = take(sizeof(float) * 2 * N * H);
    L.tcb = take(sizeof(float) * 2 * N * 2 * H);
    L.gpart = take(sizeof(float) * std::max({gemm_tn_floats(H3, H), gemm_tn_floats(H, 2 * H), gemm_tn_floats(64, H),
                                             gemm_tn_floats(32, 64), gemm_tn_floats(H, RMAX), gemm_tn_floats(32, 0)}));
    L.gmix = take(sizeof(float) * GRAD_MIX_BLOCKS * 9);
    L.geo = take(sizeof(float4) * L.cap);
    L.tgeo_t = take(sizeof(float4) * L.cap);
    L.trec_t = take(sizeof(float4) * (L.cap + TREC_PAD));
    L.tkey = take(4 * L.cap);
    L.torder = take(4 * L.cap);
    L.toffs = take(4 * nscan);
    L.tscan = take(4 * ((nscan + 1023) / 1024 + 2));
    L.tcst = take(4 * (TAB_NI + 1));
    L.thead = take(sizeof(float) * N * (2 * 64 * 3 + 2 * 32 * 2 + 32 + 1));
    L.tadj = take(sizeof(float) * (L.cap / CHUNK + TAB_NI + 1) * 6 * TAB_NC * H);
    // the value forward pass
    L.prows = take(sizeof(float) * (L.L + 1) * N * 4 * H);
    L.fz = take(sizeof(float) * (L.cap / 2 + 1) * H);
    L.tnode = take(sizeof(float) * 2 * NODES * (H3 + H));
    L.temb = take(sizeof(float) * EMB_SPLIT * (size_t)d.n_species * H);
    return p;
}

int run_train_table(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                    const WsLayout& L, void* ws, double* energy, cudaStream_t st, const GradCtx& grad) {
    return run_train<false>(d, P, po, sys, L, ws, energy, st, grad, nullptr, nullptr);
}
int run_train_table_tangent(const mlff_dims& d, const float* P, const PackedOffsets& po, const mlff_system& sys,
                            const WsLayout& L, void* ws, cudaStream_t st, const GradCtx& grad, const float* G,
                            const double* S) {
    return run_train<true>(d, P, po, sys, L, ws, nullptr, st, grad, G, S);
}

}  // namespace mlff
