// k_scalar.cu -- scalar Laplace stiffness and load vector, FP64 throughout.
//
// FE::assemblyLaplace (feddlib/core/FE/FE_def.hpp:2437-2500):
//     K_ab = |det B| sum_q w_q grad phi_a . grad phi_b
// FE::assemblyRHS with a constant source (FE_def.hpp:7303-7400):
//     b_a  = |det B| f sum_q w_q phi_a(q)
// For affine elements both orders' integrals are combinations of the products
//     D_ij = V L_i . L_j = C_i . C_j / (6 |det B|)
// of the barycentric gradients L_i = C_i / det B (C_1..C_3 the cofactor columns,
// C_0 = -(C_1 + C_2 + C_3), V = |det B| / 6): P1 K_ij = D_ij, and with
// int lambda_i lambda_j = V (1 + d_ij) / 20 for P2
//     vertices i, j:           3/5 D_ii, -1/5 D_ij
//     vertex i, edge (j, k):   (4/5 d_ij - 1/5) D_ik + (4/5 d_ik - 1/5) D_ij
//     edges (i, j), (k, l):    4/5 ((1 + d_ik) D_jl + (1 + d_il) D_jk
//                                   + (1 + d_jk) D_il + (1 + d_jl) D_ik).
// The load factors m_a = sum_q w_q phi_a are exact for the reference's rules (1
// point for P1, 5 points for P2).
//
// The FP64 pipe takes 20 cycles per warp instruction, whatever the number of
// active lanes, so what counts is FP64 warp instructions: the element kernel
// forms its entries in few of them, and the row kernel adds an incidence's
// entries and load for several nodes at once (a warp's 32 lanes hold six P1 or
// two P2 nodes).  Element and row kernel, us, before (one warp per node, P2 by
// the reference gradients' integrals) and after: 16^3 x 6 tets P1 10.3 + 19.9
// and 8.2 + 9.5, P2 35.6 + 45.2 and 15.8 + 19.0; 40^3 x 6 P2 281 + 559 and
// 168 + 185 (252 with the element's values stored one by one).
#include "kernels.cuh"

namespace fedd {
namespace {


__device__ __forceinline__ int lap_packed(int n, int a, int b) {
    if (a > b) { int t = a; a = b; b = t; }
    return a * n - (a * (a - 1)) / 2 + (b - a);
}

__host__ __device__ constexpr int lap_edge(int a, int end) {  // vertices of P2 node 4 + a: 01 12 02 03 13 23
    constexpr int E[6][2] = {{0, 1}, {1, 2}, {0, 2}, {0, 3}, {1, 3}, {2, 3}};
    return E[a][end];
}

// WANT_K: the stiffness (packed upper triangle); the load always
template <int NPE, bool WANT_K>
__global__ void __launch_bounds__(64) k_lap_elem(const double *__restrict__ xyz, const int32_t *__restrict__ conn,
                                                 int64_t ne, double f, const double *__restrict__ mfac, double *stage,
                                                 int *err, int64_t e_begin, int64_t e_end) {
    constexpr int STRIDE = NPE == 4 ? kLapStrideP1 : kLapStrideP2;
    constexpr int NK = NPE * (NPE + 1) / 2;
    int64_t e = e_begin + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= e_end) return;
    const int32_t n0 = conn[e], n1 = conn[ne + e], n2 = conn[2 * ne + e], n3 = conn[3 * ne + e];
    double x0 = xyz[3 * (int64_t)n0], y0 = xyz[3 * (int64_t)n0 + 1], z0 = xyz[3 * (int64_t)n0 + 2];
    double B[9] = {xyz[3 * (int64_t)n1] - x0, xyz[3 * (int64_t)n2] - x0, xyz[3 * (int64_t)n3] - x0,
                   xyz[3 * (int64_t)n1 + 1] - y0, xyz[3 * (int64_t)n2 + 1] - y0, xyz[3 * (int64_t)n3 + 1] - y0,
                   xyz[3 * (int64_t)n1 + 2] - z0, xyz[3 * (int64_t)n2 + 2] - z0, xyz[3 * (int64_t)n3 + 2] - z0};
    double C[9];
    C[0] = B[4] * B[8] - B[5] * B[7]; C[1] = B[5] * B[6] - B[3] * B[8]; C[2] = B[3] * B[7] - B[4] * B[6];
    if (WANT_K) {
        C[3] = B[2] * B[7] - B[1] * B[8]; C[4] = B[0] * B[8] - B[2] * B[6]; C[5] = B[1] * B[6] - B[0] * B[7];
        C[6] = B[1] * B[5] - B[2] * B[4]; C[7] = B[2] * B[3] - B[0] * B[5]; C[8] = B[0] * B[4] - B[1] * B[3];
    }
    const double det = B[0] * C[0] + B[1] * C[1] + B[2] * C[2];
    if (det == 0.0) set_dev_error(err, kDevBadDet);
    const double ad = fabs(det);
    const double fa = ad * f;
    double *S = stage + e * STRIDE;
    if (WANT_K) {
        double G[4][3], D[4][4];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            G[1][k] = C[3 * k];
            G[2][k] = C[3 * k + 1];
            G[3][k] = C[3 * k + 2];
            G[0][k] = -(G[1][k] + G[2][k] + G[3][k]);
        }
        // P2: a fifth of D.  Row 0 from G_0 like the others: as minus the sum of their
        // entries (7.5 us instead of 8.2 at 16^3 x 6 tets P1) it loses the square of
        // an element's height over its base, 5e-9 of D_00 at 1000
        const double w = (NPE == 4 ? 1.0 : 0.2) / (6.0 * ad);
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const double g0 = w * G[a][0], g1 = w * G[a][1], g2 = w * G[a][2];
#pragma unroll
            for (int b = a; b < 4; b++) D[a][b] = D[b][a] = g0 * G[b][0] + g1 * G[b][1] + g2 * G[b][2];
        }
        // values in pairs: the stores of a warp are not contiguous
        double even = 0.0;
        auto put = [&](int t, double v) {
            if (t & 1) *reinterpret_cast<double2 *>(S + t - 1) = make_double2(even, v);
            else even = v;
        };
        int t = 0;
#pragma unroll
        for (int a = 0; a < NPE; a++)
#pragma unroll
            for (int b = a; b < NPE; b++, t++) {
                double v;
                if (NPE == 4) {
                    v = D[a & 3][b & 3];
                } else if (b < 4) {
                    v = a == b ? 3.0 * D[a & 3][a & 3] : -D[a & 3][b & 3];
                } else if (a < 4) {
                    const int j = lap_edge(b >= 4 ? b - 4 : 0, 0), k = lap_edge(b >= 4 ? b - 4 : 0, 1);
                    v = a == j ? 3.0 * D[a & 3][k] - D[a & 3][j]
                               : (a == k ? 3.0 * D[a & 3][j] - D[a & 3][k] : -(D[a & 3][j] + D[a & 3][k]));
                } else {
                    const int i = lap_edge(a >= 4 ? a - 4 : 0, 0), j = lap_edge(a >= 4 ? a - 4 : 0, 1);
                    const int k = lap_edge(b >= 4 ? b - 4 : 0, 0), l = lap_edge(b >= 4 ? b - 4 : 0, 1);
                    double s = (i == k ? 2.0 : 1.0) * D[j][l] + (j == l ? 2.0 : 1.0) * D[i][k];
                    s += (i == l ? 2.0 : 1.0) * D[j][k] + (j == k ? 2.0 : 1.0) * D[i][l];
                    v = 4.0 * s;
                }
                put(t, v);
            }
#pragma unroll
        for (int a = 0; a < NPE; a++) put(NK + a, fa * mfac[a]);
        if ((NK + NPE) & 1) S[NK + NPE - 1] = even;
        return;
    }
#pragma unroll
    for (int a = 0; a < NPE; a++) S[NK + a] = fa * mfac[a];
}

// Several nodes per warp, NPE + 1 lanes each: lane b < NPE adds column b of the
// node's row of each incidence, lane NPE its load (to the word behind the
// columns), four incidences read ahead; FP64 accumulation in shared memory, in
// incidence order.
template <int NPE>
__global__ void __launch_bounds__(128) k_lap_rows(const int64_t *__restrict__ inc_ptr, const uint32_t *__restrict__ inc,
                                                  const uint8_t *__restrict__ slots, const int64_t *__restrict__ adj_ptr,
                                                  const double *__restrict__ stage, double *vals, double *load,
                                                  int64_t nnodes, int max_adj) {
    constexpr int STRIDE = NPE == 4 ? kLapStrideP1 : kLapStrideP2;
    constexpr int NK = NPE * (NPE + 1) / 2, W = NPE + 1, NODES = 32 / W, AHEAD = 4;
    extern __shared__ double dacc[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, s = lane / W, b = lane - W * s;
    const int64_t n = (blockIdx.x * (int64_t)(blockDim.x >> 5) + w) * NODES + s;
    const bool in = s < NODES && n < nnodes;
    double *acc = dacc + (size_t)(w * (NODES + 1) + s) * (max_adj + 1);  // the last one: lanes without a node
    const int64_t a0 = in ? adj_ptr[n] : 0, i0 = in ? inc_ptr[n] : 0;
    const int K = in ? (int)(adj_ptr[n + 1] - a0) : 0, m = in ? (int)(inc_ptr[n + 1] - i0) : 0;
    for (int c = b; c <= K; c += W) acc[c] = 0.0;
    int mm = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mm = max(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    __syncwarp();
    for (int t0 = 0; t0 < mm; t0 += AHEAD) {
        double v[AHEAD];
        int at[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            v[k] = 0.0;
            at[k] = 0;
            if (t0 + k < m) {
                const int64_t i = i0 + t0 + k;
                const uint32_t ea = __ldg(inc + i);
                const int a = (int)(ea & 15u);
                v[k] = __ldg(stage + (int64_t)(ea >> 4) * STRIDE + (b < NPE ? lap_packed(NPE, a, b) : NK + a));
                at[k] = b < NPE ? __ldg(slots + i * kSlotStride + b) : K;
            }
        }
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            if (t0 + k < mm) {
                if (t0 + k < m) acc[at[k]] += v[k];
                __syncwarp();
            }
        }
    }
    if (!in) return;
    for (int c = b; c < K; c += W) vals[a0 + c] = acc[c];
    if (load && b == NPE) load[n] = acc[K];
}

// the load alone: one thread per node, its entries in incidence order
template <int NPE>
__global__ void __launch_bounds__(128) k_lap_load(const int64_t *__restrict__ inc_ptr, const uint32_t *__restrict__ inc,
                                                  const double *__restrict__ stage, double *load, int64_t nnodes) {
    constexpr int STRIDE = NPE == 4 ? kLapStrideP1 : kLapStrideP2;
    constexpr int NK = NPE * (NPE + 1) / 2;
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nnodes) return;
    const int64_t i1 = inc_ptr[n + 1];
    double r = 0.0;
#pragma unroll 4
    for (int64_t i = inc_ptr[n]; i < i1; i++) {
        const uint32_t ea = __ldg(inc + i);
        r += __ldg(stage + (int64_t)(ea >> 4) * STRIDE + NK + (ea & 15u));
    }
    load[n] = r;
}

template <int NPE>
__global__ void k_lap_dense(const double *__restrict__ stage, int64_t first, int64_t count, double *Ke, double *re) {
    constexpr int STRIDE = NPE == 4 ? kLapStrideP1 : kLapStrideP2;
    constexpr int NK = NPE * (NPE + 1) / 2;
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= count * (NPE * NPE + NPE)) return;
    int64_t e = t / (NPE * NPE + NPE);
    int k = (int)(t - e * (NPE * NPE + NPE));
    const double *S = stage + (first + e) * STRIDE;
    if (k < NPE * NPE)
        Ke[e * NPE * NPE + k] = S[lap_packed(NPE, k / NPE, k % NPE)];
    else
        re[e * NPE + (k - NPE * NPE)] = S[NK + (k - NPE * NPE)];
}

}  // namespace

// Host FP64 table for the Laplace stage: the load factors m[10].
void lap_make_tables(int order, std::vector<double> &out) {
    out.assign(kLapTab, 0.0);
    if (order == 1) {
        for (int a = 0; a < 4; a++) out[a] = (1.0 / 6.0) * 0.25;  // one point, phi = 1/4
        return;
    }
    Rule r = make_rule(5);
    for (int q = 0; q < r.n; q++) {
        double ph[10];
        basis_phi(2, r.pts[q], ph);
        for (int a = 0; a < 10; a++) out[a] += r.w[q] * ph[a];
    }
}

void launch_lap_elem(const double *xyz, const int32_t *conn, int64_t ne, int order, const double *d_tables, double f,
                     bool want_k, double *stage, int *d_err, cudaStream_t s, LaunchCounter &lc, int64_t e_begin,
                     int64_t e_end) {
    if (e_end < 0) e_end = ne;
    const int64_t count = e_end - e_begin;
    if (count <= 0) return;
    auto kern = order == 1 ? (want_k ? k_lap_elem<4, true> : k_lap_elem<4, false>)
                           : (want_k ? k_lap_elem<10, true> : k_lap_elem<10, false>);
    kern<<<ceil_div(count, 64), 64, 0, s>>>(xyz, conn, ne, f, d_tables, stage, d_err, e_begin, e_end);
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_lap_rows(const Graph &g, const double *stage, int order, double *vals, double *load, int64_t nnodes,
                     cudaStream_t s, LaunchCounter &lc) {
    if (nnodes <= 0) return;
    if (!vals) {
        auto kern = order == 1 ? k_lap_load<4> : k_lap_load<10>;
        kern<<<ceil_div(nnodes, 128), 128, 0, s>>>(g.inc_ptr.p, g.inc.p, stage, load, nnodes);
    } else {
        const int warps = 4, nodes = order == 1 ? 32 / 5 : 32 / 11;
        const size_t smem = (size_t)warps * (nodes + 1) * (g.max_adj + 1) * sizeof(double);
        auto kern = order == 1 ? k_lap_rows<4> : k_lap_rows<10>;
        if (smem > 48 * 1024) allow_dynamic_smem(kern);
        kern<<<ceil_div(nnodes, warps * nodes), 32 * warps, smem, s>>>(g.inc_ptr.p, g.inc.p, g.slots.p, g.adj_ptr.p, stage,
                                                                      vals, load, nnodes, g.max_adj);
    }
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_lap_dense(const double *stage, int order, int64_t first, int64_t count, double *Ke, double *re,
                      cudaStream_t s) {
    if (count == 0) return;
    const int per = order == 1 ? 20 : 110;
    if (order == 1)
        k_lap_dense<4><<<ceil_div(count * per, 256), 256, 0, s>>>(stage, first, count, Ke, re);
    else
        k_lap_dense<10><<<ceil_div(count * per, 256), 256, 0, s>>>(stage, first, count, Ke, re);
    FEDD_CUDA(cudaGetLastError());
}

}  // namespace fedd
