// k_hyper.cu -- P2 elasticity / hyperelasticity: element stage (two elements
// per warp, FP32) and row stage (warp per node, deterministic gather).
//
// Element math follows the AceGen kernels FEDDLib calls for
// "LinearElasticity" (skr1, NeoHookQuadraticTets.f, 4-point rule code 18),
// "NonLinearElasticity" (skr2, NeoHookQuadraticTets2.f, 5-point rule code 19)
// and "NonLinearElasticity2" (skr3, NeoHookQuadraticTets3.f, code 19),
// restated from their strain energies (skr1: :27-32, 481-483; skr2: :28-30,
// 490-512; skr3: :25-31, 491-496) with FEDDLib's sign conventions
// (AssembleFE_LinElas_def.hpp:117-121, 167):
//     K = det B sum_q w_q G_a . A(F_q) . G_b,   r = -det B sum_q w_q P(F_q) G_a
// written for any law Psi(I1, J, I4a, I4b) through invariant derivatives:
//     K_(ai)(bj) = sum_kl psi_kl D_k[a,i] D_l[b,j] + d_ij (2 psi_1 G_a.G_b
//                  + sum_f 2 psi_4f (a_f.G_a)(a_f.G_b))
//                  + (psi_J / J) (c_a,i c_b,j - c_b,i c_a,j)
//     D_1 = 2 F G,  D_J = c = cof(F) G,  D_4f = 2 (F a_f)(a_f . G).
// The geometry (B^-1, det B) comes from the mesh's table, formed in FP64;
// everything else is FP32.
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "mlp_dev.cuh"

namespace fedd {
namespace {

constexpr int kWarps = 4;

// Staged element rows, 32 floats each: word elem_col(a, c) of the rows 3 a + i
// holds column c; columns 0-29 are (b, j) = 3 b + j, 30 the row's residual entry,
// 31 zero.  The nodes b are in the order 0-5, 8, 9, 6, 7 (elem_node), and a
// row's eight 16-byte chunks are rotated by elem_rot(a): with these two the
// 8-byte stores of the element kernel's tiles, (A, B) and transposed, fall on
// sixteen different bank pairs.
__device__ __forceinline__ int elem_node(int b) { return b < 6 ? b : b ^ 14; }
constexpr unsigned kElemRot = 06273375140;  // three bits per node
__device__ __forceinline__ int elem_rot(int a) { return (int)(kElemRot >> (3 * a)) & 7; }
__device__ __forceinline__ int elem_col(int a, int c) {
    const int k = c < 30 ? 3 * elem_node(c / 3) + c % 3 : c;
    return 4 * (((k >> 2) + elem_rot(a)) & 7) + (k & 3);
}

// shared to global memory by the bulk copy engine (16-byte multiples), one thread's groups
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_store(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(__cvta_generic_to_global(dst)),
                 "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- laws ----------------------------------------------------------------
__device__ __forceinline__ void nh_matrix(int kind, float mu, float lam, float J, QPDerivs &d) {
    float iJ = 1.0f / J;
    d.d1[0] = 0.5f * mu;
    if (kind == kLawSKR2) {
        float lnJ = logf(J);
        d.d1[1] = (lam * lnJ - mu) * iJ;
        d.d2[4] = (mu + lam - lam * lnJ) * iJ * iJ;
    } else {  // skr1 (also the matrix of the fibre law and of the surrogate)
        d.d1[1] = -mu * iJ + 0.5f * lam * (J - iJ);
        d.d2[4] = mu * iJ * iJ + 0.5f * lam * (1.0f + iJ * iJ);
    }
}

__device__ __forceinline__ void fibre_terms(float k1, float k2, float I4, float &d1, float &d2) {
    float e = I4 - 1.0f;
    if (e > 0.0f) {
        float ex = expf(k2 * e * e);
        d1 = k1 * e * ex;
        d2 = k1 * ex * (1.0f + 2.0f * k2 * e * e);
    } else {
        d1 = 0.0f;
        d2 = 0.0f;
    }
}

// skr3, the isochoric split (NeoHookQuadraticTets3.f:25-31, 491-496, where
// v(208), v(214) and v(561) are the derivatives below with respect to
// I3 = J^2): Psi = mu/2 (J^-2/3 I1 - 3) + kappa/2 (J - 1)^2 with
// mu = E / (2 (1 + nu)), kappa = E / (3 (1 - 2 nu)).
__device__ __forceinline__ void skr3_terms(float mu, float kappa, float I1, float J, QPDerivs &d) {
    const float c = 1.0f / cbrtf(J);  // J^-1/3
    const float j23 = c * c, j53 = j23 / J, j83 = j53 * j23 * c;
    d.d1[0] = 0.5f * mu * j23;
    d.d1[1] = -(mu / 3.0f) * I1 * j53 + kappa * (J - 1.0f);
    d.d2[1] = -(mu / 3.0f) * j53;
    d.d2[4] = (5.0f * mu / 9.0f) * I1 * j83 + kappa;
}

// plain law at given invariants (used by the fused element stage, the
// plain-law QP kernel and the fallback of the surrogate)
__device__ __forceinline__ void law_plain(const LawParams &L, const float *inv, QPDerivs &d) {
#pragma unroll
    for (int k = 0; k < 4; k++) d.d1[k] = 0.0f;
#pragma unroll
    for (int k = 0; k < 10; k++) d.d2[k] = 0.0f;
    if (L.kind == kLawSKR3) {
        skr3_terms(L.mu, L.lam, inv[0], inv[1], d);
        return;
    }
    int kind = L.kind == kLawSKR2 ? kLawSKR2 : kLawSKR1;
    nh_matrix(kind, L.mu, L.lam, inv[1], d);
    if (L.kind == kLawAniso || L.kind == kLawMLP) {
        fibre_terms(L.k1, L.k2, inv[2], d.d1[2], d.d2[7]);
        fibre_terms(L.k1, L.k2, inv[3], d.d1[3], d.d2[9]);
    }
}

__device__ __forceinline__ float det3(const float *F) {
    return F[0] * (F[4] * F[8] - F[5] * F[7]) - F[1] * (F[3] * F[8] - F[5] * F[6]) + F[2] * (F[3] * F[7] - F[4] * F[6]);
}

__device__ __forceinline__ void cof3(const float *F, float *C) {
    C[0] = F[4] * F[8] - F[5] * F[7];
    C[1] = F[5] * F[6] - F[3] * F[8];
    C[2] = F[3] * F[7] - F[4] * F[6];
    C[3] = F[2] * F[7] - F[1] * F[8];
    C[4] = F[0] * F[8] - F[2] * F[6];
    C[5] = F[1] * F[6] - F[0] * F[7];
    C[6] = F[1] * F[5] - F[2] * F[4];
    C[7] = F[2] * F[3] - F[0] * F[5];
    C[8] = F[0] * F[4] - F[1] * F[3];
}

// ---- element stage ----------------------------------------------------
// A warp takes a batch of consecutive elements, two at a time:
//   phase 1  the geometry table's entries, one element of the batch per lane;
// then for each pair of elements:
//   phase Q  lane (element, q < nq): F_q, cof F_q and the law's derivatives at
//            F_q, folded with the weight w_q det B into the scalars below;
//   phase V  a lane per (element, point q) and every few pairs of nodes a:
//            G = B^-T grad phi_a(q), c = cof(F_q) G, f = F_q G, the fibre
//            projections a_f . G and the nodes' residual contributions at q;
//   phase K  a half warp per element, one lane per 2 x 2 tile of node pairs
//            (2 A + x, 2 B + y), A <= B (15 tiles), so a record read from
//            shared memory serves two blocks; each 3 x 3 block sums over q in
//            registers
//              K_(ai)(bj) += gamma G_a.G_b d_ij + alpha c_ai c_bj
//                            - beta c_bi c_aj + (law-specific terms)
//            with gamma = 2 s psi_1, beta = s psi_J / J,
//            alpha = s (psi_JJ + psi_J / J), s = w_q det B;
//   epilogue both triangles into a shared-memory image of the elements' rows,
//            which one bulk copy takes to the stage.
constexpr int kQS = 52;    // floats per quadrature-point record: 13 chunks of 16 B, so the records
                           // of q = 0..4 start in different bank groups
// quadrature-point record: F 0-8, cof F 9-17, (gamma alpha beta kappa) 20,
// (phi1 phi2 chi1 chi2) 24, F a1 28, F a2 32, s psi_kl 36-45, residual
// scalars (-2 s psi_1, -s psi_J, -2 s psi_4a, -2 s psi_4b) 48
constexpr int kQScal = 20, kQFib = 24, kQFa1 = 28, kQFa2 = 32, kQHess = 36, kQRes = 48;
// node records of a point, two nodes 2 m and 2 m + 1 side by side: planes of the
// five pairs' 16-byte chunks  c0 c0' c1 c1' | c2 c2' G0 G0' | G1 G1' G2 G2' |
// g1 g1' g2 g2' with fibres | f0 f0' f1 f1' | f2 f2' - - where the law's blocks
// have f.  So two nodes' values are the operands of one packed instruction.
constexpr int kVPlane = 20;
constexpr int kImage = kElemStride;  // floats of an element's image
constexpr int kPairWords = 2 * kImage + 16 + 5 * kQS;
// words between the points' node records and between their residual
// contributions, by the banks of phase V's stores (ch planes)
__host__ __device__ constexpr int vpoint(int ch, int nq) {
    return nq == 4 ? (ch <= 4 ? 80 : ch == 5 ? 112 : 144) : (ch == 3 ? 76 : ch <= 5 ? 108 : 120);
}
__host__ __device__ constexpr int rpoint(int nq) { return nq == 4 ? 44 : 33; }
static_assert(5 * kQS + 8 * (vpoint(6, 4) + rpoint(4)) <= 2 * kImage && 5 * kQS + 10 * (vpoint(6, 5) + rpoint(5)) <= 2 * kImage,
              "the phase buffers alias the images");

// lane of a half warp -> tile (A << 4 | B); lane 15 repeats lane 14's and stores nothing
__constant__ uint8_t c_tile_lane[16] = {0x00, 0x01, 0x02, 0x03, 0x04, 0x11, 0x12, 0x13,
                                        0x14, 0x22, 0x23, 0x24, 0x33, 0x34, 0x44, 0x44};

// the scalars of one quadrature point that every block reads
template <int LAW>
struct PointScalars {
    float4 s;          // gamma alpha beta kappa
    float4 fib;        // phi1 phi2 chi1 chi2
    float fa1[3], fa2[3];
    float h[10];       // s psi_kl (surrogate)
    __device__ __forceinline__ void load(const float *Qq) {
        constexpr bool kFibre = (LAW == kLawAniso || LAW == kLawMLP || LAW == kLawMLPF);
        s = *reinterpret_cast<const float4 *>(Qq + kQScal);
        if (kFibre) {
            fib = *reinterpret_cast<const float4 *>(Qq + kQFib);
            const float4 x = *reinterpret_cast<const float4 *>(Qq + kQFa1);
            const float4 y = *reinterpret_cast<const float4 *>(Qq + kQFa2);
            fa1[0] = x.x; fa1[1] = x.y; fa1[2] = x.z;
            fa2[0] = y.x; fa2[1] = y.y; fa2[2] = y.z;
        }
        if (LAW == kLawMLP) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float4 z = *reinterpret_cast<const float4 *>(Qq + kQHess + 4 * k);
                if (4 * k < 10) h[4 * k] = z.x;
                if (4 * k + 1 < 10) h[4 * k + 1] = z.y;
                if (4 * k + 2 < 10) h[4 * k + 2] = z.z;
                if (4 * k + 3 < 10) h[4 * k + 3] = z.w;
            }
        }
    }
};

// a pair of nodes' record at a quadrature point
struct NodePair {
    float2 c[3], G[3], g1, g2, f[3];
};

// the blocks (a, b) and (a, b') of the row node a (record A's component X) and
// the node pair of B at one quadrature point: K += the blocks' integrands
template <int LAW, int X>
__device__ __forceinline__ void block_update(float2 *K, const NodePair &A, const NodePair &B, const PointScalars<LAW> &P) {
    constexpr bool kFibre = (LAW == kLawAniso || LAW == kLawMLP || LAW == kLawMLPF);
    constexpr bool kFullHess = (LAW == kLawMLP);
    constexpr bool kCross = (LAW == kLawSKR3);
    auto of = [](float2 v) { return X ? v.y : v.x; };
    const float ca[3] = {of(A.c[0]), of(A.c[1]), of(A.c[2])};
    const float2 dot = fma2(both(of(A.G[2])), B.G[2], fma2(both(of(A.G[0])), B.G[0], mul2(both(of(A.G[1])), B.G[1])));
    float2 t[3];
    float n[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        t[j] = mul2(both(P.s.y), B.c[j]);
        n[j] = -P.s.z * ca[j];
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) K[3 * i + j] = fma2(B.c[i], both(n[j]), fma2(both(ca[i]), t[j], K[3 * i + j]));
    if (kCross) {  // psi_1J (D_1 (x) D_J + D_J (x) D_1), D_1 = 2 f
        float2 kf[3], kc[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            kf[j] = mul2(both(P.s.w), B.f[j]);
            kc[j] = mul2(both(P.s.w), B.c[j]);
        }
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                K[3 * i + j] = fma2(both(of(A.f[i])), kc[j], fma2(both(ca[i]), kf[j], K[3 * i + j]));
    }
    if (kFibre) {
        const float a1 = of(A.g1), a2 = of(A.g2);
        const float2 g1 = mul2(both(a1), B.g1), g2 = mul2(both(a2), B.g2);
        const float2 dg = fma2(both(P.fib.x), g1, fma2(both(P.fib.y), g2, mul2(both(P.s.x), dot)));
        if (!kFullHess) {  // psi_4f4f D_4f (x) D_4f, D_4f = 2 (a_f . G) F a_f
            const float2 x1 = mul2(both(P.fib.z), g1), x2 = mul2(both(P.fib.w), g2);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const float2 y1 = mul2(x1, both(P.fa1[i])), y2 = mul2(x2, both(P.fa2[i]));
#pragma unroll
                for (int j = 0; j < 3; j++)
                    K[3 * i + j] = fma2(y2, both(P.fa2[j]), fma2(y1, both(P.fa1[j]), K[3 * i + j]));
            }
            if (LAW == kLawMLPF) {  // psi_4a4b (D_4a (x) D_4b + D_4b (x) D_4a), 4 s psi_4a4b in s.w
                const float2 c12 = mul2(both(P.s.w * a1), B.g2), c21 = mul2(both(P.s.w * a2), B.g1);
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const float2 y1 = mul2(c12, both(P.fa1[i])), y2 = mul2(c21, both(P.fa2[i]));
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        K[3 * i + j] = fma2(y2, both(P.fa1[j]), fma2(y1, both(P.fa2[j]), K[3 * i + j]));
                }
            }
        } else {  // the full Hessian: sum_kl s psi_kl D_k[a] (x) D_l[b]
#pragma unroll
            for (int y = 0; y < 2; y++) {
                auto ob = [&](float2 v) { return y ? v.y : v.x; };
                float Da[4][3], Db[4][3];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    Da[0][i] = 2.0f * of(A.f[i]);
                    Db[0][i] = 2.0f * ob(B.f[i]);
                    Da[1][i] = ca[i];
                    Db[1][i] = ob(B.c[i]);
                    Da[2][i] = 2.0f * a1 * P.fa1[i];
                    Db[2][i] = 2.0f * ob(B.g1) * P.fa1[i];
                    Da[3][i] = 2.0f * a2 * P.fa2[i];
                    Db[3][i] = 2.0f * ob(B.g2) * P.fa2[i];
                }
                const float *h = P.h;
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const float E0 = h[0] * Db[0][j] + h[1] * Db[1][j] + h[2] * Db[2][j] + h[3] * Db[3][j];
                    const float E1 = h[1] * Db[0][j] + h[4] * Db[1][j] + h[5] * Db[2][j] + h[6] * Db[3][j];
                    const float E2 = h[2] * Db[0][j] + h[5] * Db[1][j] + h[7] * Db[2][j] + h[8] * Db[3][j];
                    const float E3 = h[3] * Db[0][j] + h[6] * Db[1][j] + h[8] * Db[2][j] + h[9] * Db[3][j];
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        float &k = y ? K[3 * i + j].y : K[3 * i + j].x;
                        k += Da[0][i] * E0 + Da[1][i] * E1 + Da[2][i] * E2 + Da[3][i] * E3;
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 9; k += 4) K[k] = make_float2(K[k].x + dg.x, K[k].y + dg.y);
    }
    if (!kFibre) {
#pragma unroll
        for (int k = 0; k < 9; k += 4) K[k] = fma2(both(P.s.x), dot, K[k]);
    }
}

// LAW: kLawSKR1 / kLawSKR2 / kLawSKR3 / kLawAniso (fused plain law) or
// kLawMLP (reads per-QP derivatives of the surrogate network, adds the skr1
// matrix part).  Bound by the shared-memory pipe (83 %) and latency; DRAM takes
// the rows at 75 to 90 % of the copy bandwidth.  us at
// 32^3 x 6 tets of linear elasticity, at 64^3 x 6 of skr2 and at 40^3 x 6 of the
// fibre-block surrogate: 219, 1,941 and 690 with a warp per element, one block
// per lane and pass, and an image read back by its lanes; 148, 1,564 and 593 with
// tiles and bulk stores; 125, 1,501 and 576 with conflict-free stores and a
// point's values read once for its nodes; 125, 1,330 and 558 with the next pair's
// displacements read ahead; 122, 1,151 and 479 with two nodes' values to an
// instruction and four CTAs per SM (128 registers; with five 120, 1,160 and 514,
// with three 130, 1,250 and 508).
constexpr int kElemCtas = 4;  // per SM
template <int LAW, bool HAS_U>
__global__ void __launch_bounds__(32 * kWarps, kElemCtas) k_hyper_elem(const float *__restrict__ geo,
                                                            const int32_t *__restrict__ conn, int64_t ne,
                                                            const double *__restrict__ u, LawParams L,
                                                            const QPDerivs *__restrict__ qpd,
                                                            const uint8_t *__restrict__ qpfb, float *stage,
                                                            int want_res, int *err, int64_t e_begin, int64_t e_end, int batch,
                                                            const __grid_constant__ HyperTables tab) {
    constexpr bool kFibre = (LAW == kLawAniso || LAW == kLawMLP || LAW == kLawMLPF);
    constexpr bool kF = LAW == kLawMLP || LAW == kLawSKR3;  // the blocks have f
    constexpr int CH = 3 + (kFibre ? 1 : 0) + (kF ? 2 : 0), CF = kFibre ? 4 : 3;  // planes, and the first of f
    __shared__ __align__(16) float sdphi[5][36];  // per point: grad_ref phi of the 10 nodes, zero padded
    __shared__ __align__(8) float sdpair[5][36];  // the same at 10 j + a
    __shared__ float sw[5];
    __shared__ __align__(16) float sBi[kWarps][32][12];  // B^-1, det B
    __shared__ __align__(16) float sU[kWarps][2][36];  // nodal u of the element pair of phase Q
    __shared__ __align__(16) float sBuf[kWarps][kPairWords];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = tab.nq;
    for (int i = threadIdx.x; i < 5 * 36; i += blockDim.x) {
        const int q = i / 36, k = i - 36 * q;
        (&sdphi[0][0])[i] = (q < nq && k < 30) ? (&tab.dphi[0][0][0])[30 * q + k] : 0.0f;
        if (q < nq && k < 30) sdpair[q][10 * (k % 3) + k / 3] = (&tab.dphi[0][0][0])[30 * q + k];
    }
    if (threadIdx.x < 5) sw[threadIdx.x] = (int)threadIdx.x < nq ? tab.w[threadIdx.x] : 0.0f;
    if (lane < 12) sU[w][lane / 6][30 + lane % 6] = 0.0f;
    __syncthreads();

    const int h = lane >> 4, hl = lane & 15;
    const int A = c_tile_lane[hl] >> 4, B = c_tile_lane[hl] & 15;
    // per warp: point records of an even element (QA) | V | Rq, aliased by
    // the elements' images, then the point records of the odd element (QB)
    float *QA = sBuf[w];                         // [5][kQS]
    float *V = QA + 5 * kQS;                     // [2][nq] of CH planes
    const int vp = vpoint(CH, nq), rp = rpoint(nq);
    float *Rq = V + 2 * nq * vp;                 // [2][nq][rp]: residual contributions of (node, component)
    float *QB = sBuf[w] + 2 * kImage + 16;       // [5][kQS], in other banks than QA
    float *O = sBuf[w] + h * kImage;             // this half's image
    // the tile's places in the image: the pairs of columns c of B in the rows of A, and of A in the rows of B
    // (those of the odd nodes' rows: 16 words on or back)
    int oAB[3], oBA[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const int cb = 3 * elem_node(2 * B) + 2 * c, ca = 3 * elem_node(2 * A) + 2 * c;
        oAB[c] = 192 * A + 4 * (((cb >> 2) + elem_rot(2 * A)) & 7) + (cb & 3);
        oBA[c] = 192 * B + 4 * (((ca >> 2) + elem_rot(2 * B)) & 7) + (ca & 3);
    }
    const int rcol = 32 * lane + 4 * ((7 + elem_rot(lane / 3)) & 7) + 2;  // row `lane`, columns 30 and 31

    for (int64_t e0 = e_begin + ((int64_t)blockIdx.x * kWarps + w) * batch; e0 < e_end;
         e0 += (int64_t)gridDim.x * kWarps * batch) {
        {  // phase 1: geometry, one element per lane
            int64_t e = e0 + lane;
            if (lane < batch && e < e_end) {
                float Bi[9];
                const float det = load_geometry(geo, ne, e, Bi);
#pragma unroll
                for (int k = 0; k < 9; k++) sBi[w][lane][k] = Bi[k];
                // det B, times the element's E_e / E when a modulus field is set (the
                // point weights w_q det B carry it into every block and residual term)
                sBi[w][lane][9] = L.escale ? det * L.escale[e] : det;
                if (!(det > 0.0f) && !(det < 0.0f)) set_dev_error(err, kDevBadDet);
            }
        }
        __syncwarp();
        const int nb = (int)min((int64_t)batch, e_end - e0);
        // nodal u of a pair of elements, values lane and lane + 32 of its 60: the
        // next pair's nodes are read before phase Q, their u before phase K
        int32_t un[2] = {0, 0};
        double uv[2] = {0.0, 0.0};
        auto read_nodes = [&](int t) {
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const int k = lane + 32 * m, ep = k >= 30 ? 1 : 0;
                if (k < 60 && t + ep < nb) un[m] = __ldg(conn + (int64_t)((k - 30 * ep) / 3) * ne + e0 + t + ep);
            }
        };
        auto read_u = [&]() {
#pragma unroll
            for (int m = 0; m < 2; m++) uv[m] = __ldg(u + 3 * (int64_t)un[m] + (lane + 32 * m) % 3);
        };
        if (HAS_U) {
            read_nodes(0);
            read_u();
        }
        for (int t = 0; t < nb; t += 2) {
            const int64_t el = e0 + t;
            const int pair = t + 1 < nb ? 2 : 1;
            // phase Q: one lane per (element, quadrature point), lane = ep nq + q
            {
                if (HAS_U) {
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const int k = lane + 32 * m, ep = k >= 30 ? 1 : 0;
                        if (k < 60) sU[w][ep][k - 30 * ep] = d2f_rn(uv[m]);
                    }
                    read_nodes(t + 2);
                }
                if (lane == 0) bulk_wait_read();  // the previous pair's images have left
                __syncwarp();
                const int ep = lane >= nq ? 1 : 0, q = lane - ep * nq;
                if (lane < pair * nq) {
                const float *Bq = sBi[w][t + ep];
                const float detB = Bq[9];
                float F[9];
                if (HAS_U) {
                    // H = sum_a u_a (x) grad_ref phi_a(q), nodes four at a time
                    float H[9];
#pragma unroll
                    for (int k = 0; k < 9; k++) H[k] = 0.0f;
                    const float4 *u4 = reinterpret_cast<const float4 *>(sU[w][ep]);
                    const float4 *d4 = reinterpret_cast<const float4 *>(sdphi[q]);
#pragma unroll
                    for (int g = 0; g < 3; g++) {
                        float uu[12], dd[12];
#pragma unroll
                        for (int m = 0; m < 3; m++) {
                            const float4 x = u4[3 * g + m], y = d4[3 * g + m];
                            uu[4 * m] = x.x; uu[4 * m + 1] = x.y; uu[4 * m + 2] = x.z; uu[4 * m + 3] = x.w;
                            dd[4 * m] = y.x; dd[4 * m + 1] = y.y; dd[4 * m + 2] = y.z; dd[4 * m + 3] = y.w;
                        }
#pragma unroll
                        for (int n = 0; n < 4; n++)
#pragma unroll
                            for (int i = 0; i < 3; i++)
#pragma unroll
                                for (int c = 0; c < 3; c++) H[3 * i + c] = fmaf(uu[3 * n + i], dd[3 * n + c], H[3 * i + c]);
                    }
                    // F = I + H B^-1
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int k = 0; k < 3; k++)
                            F[3 * i + k] = (i == k ? 1.0f : 0.0f) + H[3 * i] * Bq[k] + H[3 * i + 1] * Bq[3 + k] +
                                           H[3 * i + 2] * Bq[6 + k];
                } else {
#pragma unroll
                    for (int k = 0; k < 9; k++) F[k] = (k % 4 == 0) ? 1.0f : 0.0f;
                }
                float C[9];
                cof3(F, C);
                const float J = F[0] * C[0] + F[1] * C[1] + F[2] * C[2];
                if (!(J > 0.0f)) set_dev_error(err, kDevBadDet);
                float Fa1[3] = {0.0f, 0.0f, 0.0f}, Fa2[3] = {0.0f, 0.0f, 0.0f}, inv[4];
                inv[0] = 0.0f;
#pragma unroll
                for (int k = 0; k < 9; k++) inv[0] = fmaf(F[k], F[k], inv[0]);
                inv[1] = J;
                inv[2] = inv[3] = 1.0f;
                if (kFibre) {
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        Fa1[i] = F[3 * i] * L.a1[0] + F[3 * i + 1] * L.a1[1] + F[3 * i + 2] * L.a1[2];
                        Fa2[i] = F[3 * i] * L.a2[0] + F[3 * i + 1] * L.a2[1] + F[3 * i + 2] * L.a2[2];
                    }
                    inv[2] = Fa1[0] * Fa1[0] + Fa1[1] * Fa1[1] + Fa1[2] * Fa1[2];
                    inv[3] = Fa2[0] * Fa2[0] + Fa2[1] * Fa2[1] + Fa2[2] * Fa2[2];
                }
                QPDerivs d;
                if (LAW == kLawMLP || LAW == kLawMLPF) {
                    const int64_t qi = (el + ep) * nq + q;
                    if (qpfb[qi]) {
                        law_plain(L, inv, d);
                    } else {
                        d = qpd[qi];
                        QPDerivs m;
#pragma unroll
                        for (int k = 0; k < 10; k++) m.d2[k] = 0.0f;
                        nh_matrix(kLawSKR1, L.mu, L.lam, J, m);
                        d.d1[0] += m.d1[0];
                        d.d1[1] += m.d1[1];
                        d.d2[4] += m.d2[4];
                    }
                } else {
                    law_plain(L, inv, d);
                }
                const float s = sw[q] * detB;
                const float psiJ_J = d.d1[1] / J;
                float *Qq = (ep ? QB : QA) + q * kQS;
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    Qq[k] = F[k];
                    Qq[9 + k] = C[k];
                }
                const float beta = s * psiJ_J;
                const float alpha = LAW == kLawMLP ? beta : s * (d.d2[4] + psiJ_J);
                // the fourth scalar: 2 s psi_1J (skr3) or 4 s psi_4a4b (the fibre-block surrogate)
                *reinterpret_cast<float4 *>(Qq + kQScal) =
                    make_float4(2.0f * s * d.d1[0], alpha, beta, LAW == kLawMLPF ? 4.0f * s * d.d2[8] : 2.0f * s * d.d2[1]);
                *reinterpret_cast<float4 *>(Qq + kQRes) =
                    make_float4(-2.0f * s * d.d1[0], -s * d.d1[1], -2.0f * s * d.d1[2], -2.0f * s * d.d1[3]);
                if (kFibre) {
                    *reinterpret_cast<float4 *>(Qq + kQFib) =
                        make_float4(2.0f * s * d.d1[2], 2.0f * s * d.d1[3], 4.0f * s * d.d2[7], 4.0f * s * d.d2[9]);
                    *reinterpret_cast<float4 *>(Qq + kQFa1) = make_float4(Fa1[0], Fa1[1], Fa1[2], 0.0f);
                    *reinterpret_cast<float4 *>(Qq + kQFa2) = make_float4(Fa2[0], Fa2[1], Fa2[2], 0.0f);
                }
                if (LAW == kLawMLP) {
#pragma unroll
                    for (int k = 0; k < 10; k++) Qq[kQHess + k] = s * d.d2[k];
                }
                }
            }
            __syncwarp();
            // phase V: a lane works at one (element, point q) on every 4th pair of nodes (every 3rd with five
            // points); the strides put no two of a quarter warp's stores on one bank
            {
                const int parts = nq == 4 ? 4 : 3, qq = lane / parts, ep = qq >= nq ? 1 : 0, q = qq - ep * nq;
                if (qq < nq * pair) {
                const float *Qq = (ep ? QB : QA) + q * kQS;
                float FC[20], Bi[12];
#pragma unroll
                for (int m = 0; m < 5; m++) {
                    const float4 x = reinterpret_cast<const float4 *>(Qq)[m];
                    FC[4 * m] = x.x; FC[4 * m + 1] = x.y; FC[4 * m + 2] = x.z; FC[4 * m + 3] = x.w;
                }
#pragma unroll
                for (int m = 0; m < 3; m++) {
                    const float4 x = reinterpret_cast<const float4 *>(sBi[w][t + ep])[m];
                    Bi[4 * m] = x.x; Bi[4 * m + 1] = x.y; Bi[4 * m + 2] = x.z; Bi[4 * m + 3] = x.w;
                }
                const float4 rs = *reinterpret_cast<const float4 *>(Qq + kQRes);
                float4 x1, x2;  // F a1, F a2
                if (kFibre) {
                    x1 = *reinterpret_cast<const float4 *>(Qq + kQFa1);
                    x2 = *reinterpret_cast<const float4 *>(Qq + kQFa2);
                }
                float *Vq = V + qq * vp, *rq = Rq + qq * rp;
                for (int m = lane - parts * qq; m < 5; m += parts) {
                    float2 d[3], G[3], c[3], f[3];
#pragma unroll
                    for (int j = 0; j < 3; j++) d[j] = *reinterpret_cast<const float2 *>(&sdpair[q][10 * j + 2 * m]);
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        G[k] = fma2(both(Bi[6 + k]), d[2], fma2(both(Bi[k]), d[0], mul2(both(Bi[3 + k]), d[1])));
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        c[i] = fma2(both(FC[9 + 3 * i + 2]), G[2], fma2(both(FC[9 + 3 * i]), G[0], mul2(both(FC[9 + 3 * i + 1]), G[1])));
                        f[i] = fma2(both(FC[3 * i + 2]), G[2], fma2(both(FC[3 * i]), G[0], mul2(both(FC[3 * i + 1]), G[1])));
                    }
                    float2 ag1 = both(0.0f), ag2 = ag1;
                    if (kFibre) {
                        ag1 = fma2(both(L.a1[2]), G[2], fma2(both(L.a1[0]), G[0], mul2(both(L.a1[1]), G[1])));
                        ag2 = fma2(both(L.a2[2]), G[2], fma2(both(L.a2[0]), G[0], mul2(both(L.a2[1]), G[1])));
                    }
                    auto put = [&](int plane, float2 x, float2 y) {
                        *reinterpret_cast<float4 *>(Vq + kVPlane * plane + 4 * m) = make_float4(x.x, x.y, y.x, y.y);
                    };
                    put(0, c[0], c[1]);
                    put(1, c[2], G[0]);
                    put(2, G[1], G[2]);
                    if (kFibre) put(3, ag1, ag2);
                    if (kF) {
                        put(CF, f[0], f[1]);
                        put(CF + 1, f[2], f[2]);
                    }
                    if (want_res) {
                        float2 r[3];
#pragma unroll
                        for (int i = 0; i < 3; i++) r[i] = fma2(both(rs.x), f[i], mul2(both(rs.y), c[i]));
                        if (kFibre) {
                            const float2 h1 = mul2(both(rs.z), ag1), h2 = mul2(both(rs.w), ag2);
                            const float z1[3] = {x1.x, x1.y, x1.z}, z2[3] = {x2.x, x2.y, x2.z};
#pragma unroll
                            for (int i = 0; i < 3; i++) {
                                const float2 e = fma2(h1, both(z1[i]), mul2(h2, both(z2[i])));
                                r[i] = make_float2(r[i].x + e.x, r[i].y + e.y);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            rq[6 * m + i] = r[i].x;
                            rq[6 * m + 3 + i] = r[i].y;
                        }
                    }
                }
                }
            }
            __syncwarp();
            if (HAS_U && t + 2 < nb) read_u();
            // phase K: the tile's four blocks, summed over the points in registers
            float2 K[2][9];  // [x]: the blocks (2 A + x, 2 B) and (2 A + x, 2 B + 1)
#pragma unroll
            for (int k = 0; k < 18; k++) (&K[0][0])[k] = make_float2(0.0f, 0.0f);
            const float *Qh = h ? QB : QA, *Vh = V + h * nq * vp;
#pragma unroll 1
            for (int q = 0; q < nq; q++) {
                PointScalars<LAW> P;
                P.load(Qh + q * kQS);
                const float *Vq = Vh + q * vp;
                auto record = [&](int m, NodePair &R) {
                    auto get = [&](int plane, float2 &x, float2 &y) {
                        const float4 v = *reinterpret_cast<const float4 *>(Vq + kVPlane * plane + 4 * m);
                        x = make_float2(v.x, v.y);
                        y = make_float2(v.z, v.w);
                    };
                    get(0, R.c[0], R.c[1]);
                    get(1, R.c[2], R.G[0]);
                    get(2, R.G[1], R.G[2]);
                    if (kFibre) get(3, R.g1, R.g2);
                    if (kF) {
                        get(CF, R.f[0], R.f[1]);
                        R.f[2] = *reinterpret_cast<const float2 *>(Vq + kVPlane * (CF + 1) + 4 * m);
                    }
                };
                NodePair ra, rb;
                record(A, ra);
                record(B, rb);
                block_update<LAW, 0>(K[0], ra, rb, P);
                block_update<LAW, 1>(K[1], ra, rb, P);
            }
            auto value = [&](int x, int y, int k) { return y ? K[x][k].y : K[x][k].x; };
            float r0 = 0.0f, r1 = 0.0f;
            if (want_res && lane < 30)
                for (int q = 0; q < nq; q++) {
                    r0 += Rq[rp * q + lane];
                    r1 += Rq[rp * (nq + q) + lane];
                }
            if (A == B) {  // the lower block of a tile on the diagonal is the upper one transposed
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) K[1][3 * i + j].x = K[0][3 * j + i].y;
            }
            __syncwarp();  // the phase buffers are dead: the images overwrite them
            if (hl < 15 && h < pair) {
#pragma unroll
                for (int r = 0; r < 6; r++)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const int u = 2 * c, v = 2 * c + 1;  // columns of the tile
                        *reinterpret_cast<float2 *>(O + (r < 3 ? oAB[c] : oAB[c] ^ 16) + 32 * r) =
                            make_float2(value(r / 3, u / 3, 3 * (r % 3) + u % 3), value(r / 3, v / 3, 3 * (r % 3) + v % 3));
                        if (A != B)
                            *reinterpret_cast<float2 *>(O + (r < 3 ? oBA[c] : oBA[c] ^ 16) + 32 * r) =
                                make_float2(value(u / 3, r / 3, 3 * (u % 3) + r % 3), value(v / 3, r / 3, 3 * (v % 3) + r % 3));
                    }
            }
            if (lane < 30) {
                *reinterpret_cast<float2 *>(sBuf[w] + rcol) = make_float2(r0, 0.0f);
                if (pair == 2) *reinterpret_cast<float2 *>(sBuf[w] + kImage + rcol) = make_float2(r1, 0.0f);
            }
            fence_async_shared();
            __syncwarp();
            if (lane == 0) bulk_store(stage + el * kElemStride, sBuf[w], (uint32_t)(pair * kElemStride * sizeof(float)));
        }
        __syncwarp();
    }
    if (lane == 0) bulk_wait_all();
}

// ---- row stage ----------------------------------------------------------
// One warp per node: walks the node's incidences in ascending element order,
// adds row a of each staged element matrix into shared-memory rows (FP32,
// one owner lane per value and incidence), then writes the node's three CSR
// rows once, converting to FP64.  The three values each lane needs from an
// incidence are streamed into a per-warp shared-memory ring with cp.async,
// kHRing - 1 incidences ahead of the arithmetic.
constexpr int kHRing = 4;
constexpr int kHStage = 100;  // floats per ring slot: three rows of 32 (values, residual entry, zero) | slot map 16 B
constexpr int kHSlots = 96;

// stage incidence t (of m) of a node into ring slot `slot` (a constant after
// unrolling): lanes 0-23 the three rows 3 a + i of the element matrix (96
// contiguous floats, each row's chunks rotated by elem_rot(a)), lane 24 the
// slot map; each lane's destination is ring slot + 4 lane.  Every call
// commits one group, empty past the node's last incidence, so the wait counts
// hold.
__device__ __forceinline__ void hyper_stage(float *dst_lane, int slot, int t, int m, const IncList &il,
                                            const uint8_t *__restrict__ slots_node,
                                            const float *__restrict__ stage_row, int lane) {
    if (t < m) {  // warp-uniform: every lane takes part in the shuffle
        const uint32_t ea = m <= 32 ? __shfl_sync(0xffffffffu, il.lo, t & 31) : incidence_at(il, t);
        const int a = (int)(ea & 15u);
        const void *src = lane < 24 ? static_cast<const void *>(stage_row + (size_t)(ea >> 4) * kElemStride + 96 * a +
                                                                4 * ((lane + (kElemRot >> (3 * a))) & 7u))
                                    : static_cast<const void *>(slots_node + t * kSlotStride);
        if (lane < 25) cp_async16(dst_lane + slot * kHStage, src);
    }
    cp_async_commit();
}

// The node's accumulators are one run of 9 K floats in the order of its CSR
// values (three rows of 3 K), so the write-out is a linear copy: pairs of
// values as 16-byte stores, the run shifted by one word when the values start
// at an odd multiple of 8 bytes.  Behind it lane 30 keeps the node's residual
// (column 30 of the element's rows), which the same updates accumulate, and
// lane 31 a scratch word.  The kernel is bound by latency and the shared-memory
// pipe (76 %) together: 1,915 us at 64^3 x 6 tets and 257 us at 32^3 x 6 (75 %
// of the copy bandwidth in DRAM bytes), against 2,160 and 285 us with three
// planes of fixed stride, 8-byte stores, a separate residual sum and eight
// warps per CTA (1,944 and 265 us since the stage's chunks are rotated).  Slower: reading the rows straight into registers without the
// ring (334 us at 32^3), a ring running on across the nodes of a warp's run
// (298), the hardware FP32 -> FP64 conversion in place of f2d_exact (294).
constexpr int kHPad = 8;  // words besides the 9 K
__global__ void __launch_bounds__(128) k_hyper_rows(const int64_t *__restrict__ inc_ptr,
                                                    const uint32_t *__restrict__ inc,
                                                    const uint8_t *__restrict__ slots,
                                                    const int64_t *__restrict__ adj_ptr,
                                                    const float *__restrict__ stage,
                                                    double *vals, double *res, int64_t nnodes, int words,
                                                    int64_t n_begin) {
    extern __shared__ __align__(16) float sacc[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    float *ring = sacc + (size_t)w * (kHRing * kHStage + words);
    float *mem = ring + kHRing * kHStage;
    const bool lw = lane < 30;
    const int b = lw ? lane / 3 : 0, j = lw ? lane - 3 * (lane / 3) : 0;
    float *dst_lane = ring + 4 * lane;
    const uint8_t *pS = reinterpret_cast<const uint8_t *>(ring + kHSlots) + b;
    const float *pV = ring + (lw ? 3 * elem_node(b) + j : lane), *stage_row = stage + 32 * (lane >> 3);
    for (int64_t n = n_begin + (int64_t)blockIdx.x * nw + w; n < nnodes; n += (int64_t)gridDim.x * nw) {
        const int64_t i0 = inc_ptr[n], i1 = inc_ptr[n + 1];
        const int m = (int)(i1 - i0);
        const IncList il = load_incidences(inc, i0, m, lane);
        const uint8_t *slots_node = slots + i0 * kSlotStride;
#pragma unroll
        for (int t = 0; t < kHRing - 1; t++) hyper_stage(dst_lane, t, t, m, il, slots_node, stage_row, lane);
        const int64_t a0 = adj_ptr[n];
        const int K = (int)(adj_ptr[n + 1] - a0), len = 9 * K;
        double *out = vals + 9 * a0;
        const int shift = (int)((reinterpret_cast<uintptr_t>(out) >> 3) & 1);
        float *acc = mem + shift;
        for (int c = 4 * lane; c < len + kHPad; c += 128)
            *reinterpret_cast<float4 *>(mem + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        const int st = lw ? 3 * K : (lane == 30 ? 1 : 0), mul = lw ? 3 : 0;
        float *d0 = acc + (lw ? j : (lane == 30 ? len : len + 3));
        for (int t0 = 0; t0 < m; t0 += kHRing) {
#pragma unroll
            for (int rs = 0; rs < kHRing; rs++) {
                const int t = t0 + rs;
                if (t >= m) break;
                cp_async_wait<kHRing - 2>();
                // the slot's copies are visible to the warp, and every lane is
                // done with the slot consumed in the previous step, refilled next
                __syncwarp();
                hyper_stage(dst_lane, (rs + kHRing - 1) % kHRing, t + kHRing - 1, m, il, slots_node, stage_row, lane);
                float *dst = d0 + mul * pS[4 * rs * kHStage];
                dst[0] += pV[rs * kHStage];
                dst[st] += pV[rs * kHStage + 32];
                dst[2 * st] += pV[rs * kHStage + 64];
            }
        }
        cp_async_wait<0>();
        __syncwarp();
        if (len > 0) {
            if (shift && lane == 31) st_cs(out, f2d_exact(acc[0]));
            const int pairs = (len - shift) >> 1;
            for (int c = lane; c < pairs; c += 32) {
                const float2 x = *reinterpret_cast<const float2 *>(mem + 2 * shift + 2 * c);
                __stcs(reinterpret_cast<double2 *>(out + shift) + c, make_double2(f2d_exact(x.x), f2d_exact(x.y)));
            }
            if (((len - shift) & 1) && lane == 30) st_cs(out + len - 1, f2d_exact(acc[len - 1]));
        }
        if (res && lane < 3) res[3 * n + lane] = f2d_exact(acc[len + lane]);
        __syncwarp();
    }
}

// ---- surrogate path: invariants at every quadrature point ---------------
__global__ void k_hyper_invariants(const float *__restrict__ geo, const int32_t *__restrict__ conn, int64_t ne,
                                   const double *__restrict__ u, LawParams L, float *inv, int *err, int64_t e_begin,
                                   int64_t e_end, const __grid_constant__ HyperTables tab) {
    int64_t e = e_begin + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= e_end) return;
    float Bi[9];
    load_geometry(geo, ne, e, Bi);
    float ue[30];
#pragma unroll
    for (int a = 0; a < 10; a++) {
        int32_t node = conn[(int64_t)a * ne + e];
#pragma unroll
        for (int i = 0; i < 3; i++) ue[3 * a + i] = u ? d2f_rn(u[3 * (int64_t)node + i]) : 0.0f;
    }
    const int nq = tab.nq;
    for (int q = 0; q < nq; q++) {
        float Hr[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float h = 0.0f;
#pragma unroll
                for (int a = 0; a < 10; a++) h = fmaf(ue[3 * a + i], tab.dphi[q][a][c], h);
                Hr[3 * i + c] = h;
            }
        float F[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int k = 0; k < 3; k++)
                F[3 * i + k] = (i == k ? 1.0f : 0.0f) + Hr[3 * i] * Bi[k] + Hr[3 * i + 1] * Bi[3 + k] +
                               Hr[3 * i + 2] * Bi[6 + k];
        float I1 = 0.0f;
#pragma unroll
        for (int k = 0; k < 9; k++) I1 = fmaf(F[k], F[k], I1);
        float J = det3(F);
        if (!(J > 0.0f)) set_dev_error(err, kDevBadDet);
        float f1 = 0.0f, f2 = 0.0f;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            float a1 = F[3 * i] * L.a1[0] + F[3 * i + 1] * L.a1[1] + F[3 * i + 2] * L.a1[2];
            float a2 = F[3 * i] * L.a2[0] + F[3 * i + 1] * L.a2[1] + F[3 * i + 2] * L.a2[2];
            f1 = fmaf(a1, a1, f1);
            f2 = fmaf(a2, a2, f2);
        }
        float4 v = make_float4(I1, J, f1, f2);
        reinterpret_cast<float4 *>(inv)[e * nq + q] = v;
    }
}

// ---- the residual alone -------------------------------------------------
// A call for the residual alone (FEDDLib's "Rhs" call, a line search) needs
// no tangents: one thread per element takes the element kernel's residual
// operations in the same order, so the values are those of the call that
// assembles both, and one thread per node adds the node's entries in the row
// kernel's order.  Bound by the gathers of connectivity and displacements and
// by latency (168 registers, 12 warps per SM): 48 and 18 us at 41 x 29 x 35 x 6
// tets in file order, 5 points, against 394 and 285 us of the matrix stages.
constexpr int kHyperRes = 40;  // floats per element: (r_a, 0) of local node a as one 16-byte word

template <int LAW>
__global__ void __launch_bounds__(128) k_hyper_residual(const float *__restrict__ geo, const int32_t *__restrict__ conn,
                                                        int64_t ne, const double *__restrict__ u, LawParams L,
                                                        const QPDerivs *__restrict__ qpd,
                                                        const uint8_t *__restrict__ qpfb, float *__restrict__ stage,
                                                        int *err, const __grid_constant__ HyperTables tab) {
    constexpr bool kFibre = LAW == kLawAniso || LAW == kLawMLP;
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    float Bi[9];
    float det = load_geometry(geo, ne, e, Bi);
    det = L.escale ? det * L.escale[e] : det;
    if (!(det > 0.0f) && !(det < 0.0f)) set_dev_error(err, kDevBadDet);
    float r[30];
#pragma unroll
    for (int k = 0; k < 30; k++) r[k] = 0.0f;
    if (u) {
        float ue[30];
#pragma unroll
        for (int n = 0; n < 10; n++) {
            const double *up = u + 3 * (int64_t)conn[(int64_t)n * ne + e];
#pragma unroll
            for (int i = 0; i < 3; i++) ue[3 * n + i] = d2f_rn(up[i]);
        }
        const int nq = tab.nq;
#pragma unroll 1
        for (int q = 0; q < nq; q++) {
            float H[9], F[9], C[9];
#pragma unroll
            for (int k = 0; k < 9; k++) H[k] = 0.0f;
#pragma unroll
            for (int n = 0; n < 10; n++)
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int c = 0; c < 3; c++) H[3 * i + c] = fmaf(ue[3 * n + i], tab.dphi[q][n][c], H[3 * i + c]);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int k = 0; k < 3; k++)
                    F[3 * i + k] = (i == k ? 1.0f : 0.0f) + H[3 * i] * Bi[k] + H[3 * i + 1] * Bi[3 + k] +
                                   H[3 * i + 2] * Bi[6 + k];
            cof3(F, C);
            const float J = F[0] * C[0] + F[1] * C[1] + F[2] * C[2];
            if (!(J > 0.0f)) set_dev_error(err, kDevBadDet);
            float Fa1[3] = {0.0f, 0.0f, 0.0f}, Fa2[3] = {0.0f, 0.0f, 0.0f}, inv[4];
            inv[0] = 0.0f;
#pragma unroll
            for (int k = 0; k < 9; k++) inv[0] = fmaf(F[k], F[k], inv[0]);
            inv[1] = J;
            inv[2] = inv[3] = 1.0f;
            if (kFibre) {
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    Fa1[i] = F[3 * i] * L.a1[0] + F[3 * i + 1] * L.a1[1] + F[3 * i + 2] * L.a1[2];
                    Fa2[i] = F[3 * i] * L.a2[0] + F[3 * i + 1] * L.a2[1] + F[3 * i + 2] * L.a2[2];
                }
                inv[2] = Fa1[0] * Fa1[0] + Fa1[1] * Fa1[1] + Fa1[2] * Fa1[2];
                inv[3] = Fa2[0] * Fa2[0] + Fa2[1] * Fa2[1] + Fa2[2] * Fa2[2];
            }
            QPDerivs d;
            if (LAW == kLawMLP && !qpfb[e * nq + q]) {
                QPDerivs m;
                nh_matrix(kLawSKR1, L.mu, L.lam, J, m);
#pragma unroll
                for (int k = 0; k < 4; k++) d.d1[k] = qpd[e * nq + q].d1[k];
                d.d1[0] += m.d1[0];
                d.d1[1] += m.d1[1];
            } else {
                law_plain(L, inv, d);
            }
            const float s = tab.w[q] * det;
            const float4 rs = make_float4(-2.0f * s * d.d1[0], -s * d.d1[1], -2.0f * s * d.d1[2], -2.0f * s * d.d1[3]);
#pragma unroll
            for (int a = 0; a < 10; a++) {
                const float g0 = tab.dphi[q][a][0], g1 = tab.dphi[q][a][1], g2 = tab.dphi[q][a][2];
                float G[3], x[3];
#pragma unroll
                for (int k = 0; k < 3; k++) G[k] = Bi[k] * g0 + Bi[3 + k] * g1 + Bi[6 + k] * g2;
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const float c = C[3 * i] * G[0] + C[3 * i + 1] * G[1] + C[3 * i + 2] * G[2];
                    const float f = F[3 * i] * G[0] + F[3 * i + 1] * G[1] + F[3 * i + 2] * G[2];
                    x[i] = __fmaf_rn(rs.x, f, __fmul_rn(rs.y, c));  // rounded as in the element kernel
                }
                if (kFibre) {
                    const float ag1 = L.a1[0] * G[0] + L.a1[1] * G[1] + L.a1[2] * G[2];
                    const float ag2 = L.a2[0] * G[0] + L.a2[1] * G[1] + L.a2[2] * G[2];
                    const float h1 = rs.z * ag1, h2 = rs.w * ag2;
#pragma unroll
                    for (int i = 0; i < 3; i++) x[i] += h1 * Fa1[i] + h2 * Fa2[i];
                }
#pragma unroll
                for (int i = 0; i < 3; i++) r[3 * a + i] = __fadd_rn(r[3 * a + i], x[i]);  // not contracted
            }
        }
    }
    float4 *S = reinterpret_cast<float4 *>(stage + e * kHyperRes);
#pragma unroll
    for (int a = 0; a < 10; a++) S[a] = make_float4(r[3 * a], r[3 * a + 1], r[3 * a + 2], 0.0f);
}

// one thread per node: its element entries summed in incidence order
__global__ void __launch_bounds__(128) k_hyper_residual_rows(const int64_t *__restrict__ inc_ptr,
                                                             const uint32_t *__restrict__ inc,
                                                             const float *__restrict__ stage, int64_t nnodes,
                                                             double *__restrict__ res) {
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nnodes) return;
    const int64_t i0 = inc_ptr[n];
    const int m = (int)(inc_ptr[n + 1] - i0);
    const float4 *S = reinterpret_cast<const float4 *>(stage);
    float x = 0.0f, y = 0.0f, z = 0.0f;
    // eight entries in flight
    for (int t0 = 0; t0 < m; t0 += 8) {
        float4 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (t0 + k < m) {
                const uint32_t ea = __ldg(inc + i0 + t0 + k);
                v[k] = __ldg(S + (int64_t)(ea >> 4) * 10 + (ea & 15u));
            }
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (t0 + k < m) {
                x += v[k].x;
                y += v[k].y;
                z += v[k].z;
            }
    }
    res[3 * n] = f2d_exact(x);
    res[3 * n + 1] = f2d_exact(y);
    res[3 * n + 2] = f2d_exact(z);
}

__global__ void k_hyper_dense(const float *__restrict__ stage, int64_t first, int64_t count, double *Ke, double *re) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= count * 930) return;
    int64_t e = t / 930;
    int k = (int)(t - e * 930);
    const float *S = stage + (first + e) * kElemStride;
    if (k < 900) {
        int p = k / 30, q = k % 30;
        Ke[e * 900 + k] = (double)S[32 * p + elem_col(p / 3, q)];
    } else {
        re[e * 30 + (k - 900)] = (double)S[32 * (k - 900) + elem_col((k - 900) / 3, kElemResCol)];
    }
}

}  // namespace

// ---- law evaluation for judging (FP32 math, one thread per F) -----------
__global__ void k_law_eval(LawParams L, MLPDev m, int use_mlp, int64_t n, const double *__restrict__ Fin,
                           double *psi_out, double *P, double *A) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n) return;
    float F[9], C[9];
#pragma unroll
    for (int k = 0; k < 9; k++) F[k] = (float)Fin[9 * t + k];
    cof3(F, C);
    float J = F[0] * C[0] + F[1] * C[1] + F[2] * C[2];
    float Fa[2][3], inv[4];
    inv[0] = 0.0f;
    for (int k = 0; k < 9; k++) inv[0] += F[k] * F[k];
    inv[1] = J;
    const float *af[2] = {L.a1, L.a2};
    for (int f = 0; f < 2; f++) {
        for (int i = 0; i < 3; i++) Fa[f][i] = F[3 * i] * af[f][0] + F[3 * i + 1] * af[f][1] + F[3 * i + 2] * af[f][2];
        inv[2 + f] = Fa[f][0] * Fa[f][0] + Fa[f][1] * Fa[f][1] + Fa[f][2] * Fa[f][2];
    }
    QPDerivs d;
    float psi = 0.0f;
    bool inside = true;
    if (use_mlp)
        for (int k = 0; k < 4; k++) inside = inside && inv[k] >= m.inv_lo[k] && inv[k] <= m.inv_hi[k];
    if (use_mlp && inside) {
        float x[4], y, g[4], h[16];
        float dk[4], d2k[4];
        for (int k = 0; k < 4; k++) x[k] = mlp_input(m, k, inv[k], dk[k], d2k[k]);
        mlp_eval_scalar(m, x, y, g, h);
        for (int k = 0; k < 10; k++) d.d2[k] = 0.0f;
        int kl = 0;
        for (int k = 0; k < 4; k++) {
            d.d1[k] = m.out_scale * g[k] * dk[k];
            for (int l = k; l < 4; l++, kl++)
                d.d2[kl] = m.out_scale * (h[4 * k + l] * dk[k] * dk[l] + (k == l ? g[k] * d2k[k] : 0.0f));
        }
        QPDerivs mm;
        for (int k = 0; k < 10; k++) mm.d2[k] = 0.0f;
        nh_matrix(kLawSKR1, L.mu, L.lam, J, mm);
        d.d1[0] += mm.d1[0];
        d.d1[1] += mm.d1[1];
        d.d2[4] += mm.d2[4];
        float lnJ = logf(J);
        psi = 0.5f * L.mu * (inv[0] - 3.0f) - L.mu * lnJ + 0.25f * L.lam * (J * J - 1.0f - 2.0f * lnJ) + m.out_scale * y;
    } else {
        law_plain(L, inv, d);
        float lnJ = logf(J);
        if (L.kind == kLawSKR2)
            psi = 0.5f * L.mu * (inv[0] - 3.0f) - L.mu * lnJ + 0.5f * L.lam * lnJ * lnJ;
        else if (L.kind == kLawSKR3)
            psi = 0.5f * L.mu * (inv[0] / (cbrtf(J) * cbrtf(J)) - 3.0f) + 0.5f * L.lam * (J - 1.0f) * (J - 1.0f);
        else
            psi = 0.5f * L.mu * (inv[0] - 3.0f) - L.mu * lnJ + 0.25f * L.lam * (J * J - 1.0f - 2.0f * lnJ);
        if (L.kind == kLawAniso || L.kind == kLawMLP)
            for (int f = 0; f < 2; f++) {
                float e = inv[2 + f] - 1.0f;
                if (e > 0.0f) psi += L.k1 / (2.0f * L.k2) * (expf(L.k2 * e * e) - 1.0f);
            }
    }
    psi_out[t] = psi;
    // P and A from the invariant form
    float D[4][9];
    for (int i = 0; i < 3; i++)
        for (int k = 0; k < 3; k++) {
            D[0][3 * i + k] = 2.0f * F[3 * i + k];
            D[1][3 * i + k] = C[3 * i + k];
            D[2][3 * i + k] = 2.0f * Fa[0][i] * L.a1[k];
            D[3][3 * i + k] = 2.0f * Fa[1][i] * L.a2[k];
        }
    float H[4][4];
    {
        int kl = 0;
        for (int k = 0; k < 4; k++)
            for (int l = k; l < 4; l++, kl++) H[k][l] = H[l][k] = d.d2[kl];
    }
    for (int mm = 0; mm < 9; mm++) {
        float s = 0.0f;
        for (int k = 0; k < 4; k++) s += d.d1[k] * D[k][mm];
        P[9 * t + mm] = s;
    }
    for (int i = 0; i < 3; i++)
        for (int k = 0; k < 3; k++)
            for (int j = 0; j < 3; j++)
                for (int l = 0; l < 3; l++) {
                    float s = 0.0f;
                    for (int a = 0; a < 4; a++)
                        for (int b = 0; b < 4; b++) s += H[a][b] * D[a][3 * i + k] * D[b][3 * j + l];
                    if (i == j) s += 2.0f * d.d1[0] * (k == l) + 2.0f * d.d1[2] * L.a1[k] * L.a1[l] +
                                     2.0f * d.d1[3] * L.a2[k] * L.a2[l];
                    s += d.d1[1] * (C[3 * i + k] * C[3 * j + l] - C[3 * i + l] * C[3 * j + k]) / J;
                    A[81 * t + ((i * 3 + k) * 3 + j) * 3 + l] = s;
                }
}

// ---- launchers --------------------------------------------------------------
static int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

void launch_hyper_elem(const float *geo, const int32_t *conn, int64_t ne, const double *u, const LawParams &law,
                       const HyperTables &tab, const QPDerivs *qpd, const uint8_t *qp_fallback, float *stage,
                       int want_res, int *d_err, cudaStream_t s, LaunchCounter &lc, int64_t e_begin,
                       int64_t e_end) {
    if (e_end < 0) e_end = ne;
    const int64_t count = e_end - e_begin;
    if (count <= 0) return;
    // batches of at most 32 elements, even, that give the chip's warps equal
    // shares in as few rounds as there have to be
    const int64_t chip = (int64_t)sm_count() * kElemCtas * kWarps, rounds = ceil_div(count, 32 * chip);
    const int batch = 2 * (int)ceil_div(count, 2 * rounds * chip);
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(count, (int64_t)batch * kWarps), (int64_t)sm_count() * 16);
    const bool hu = u != nullptr;
#define FEDD_HYPER(LAWK)                                                                                 \
    do {                                                                                                 \
        if (hu)                                                                                          \
            k_hyper_elem<LAWK, true><<<grid, 32 * kWarps, 0, s>>>(geo, conn, ne, u, law, qpd, qp_fallback, \
                                                                  stage, want_res, d_err, e_begin, e_end, batch, tab); \
        else                                                                                             \
            k_hyper_elem<LAWK, false><<<grid, 32 * kWarps, 0, s>>>(geo, conn, ne, u, law, qpd, qp_fallback, \
                                                                   stage, want_res, d_err, e_begin, e_end, batch, tab); \
    } while (0)
    switch (law.kind) {
    case kLawSKR2: FEDD_HYPER(kLawSKR2); break;
    case kLawSKR3: FEDD_HYPER(kLawSKR3); break;
    case kLawAniso: FEDD_HYPER(kLawAniso); break;
    case kLawMLP:
        if (law.mlp_fibre) FEDD_HYPER(kLawMLPF);
        else FEDD_HYPER(kLawMLP);
        break;
    default: FEDD_HYPER(kLawSKR1); break;
    }
#undef FEDD_HYPER
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_hyper_rows(const Graph &g, const float *stage, double *vals, double *res, int64_t nnodes, cudaStream_t s,
                       LaunchCounter &lc, int64_t n_begin) {
    constexpr int warps = 4;
    const int words = (9 * g.max_adj + kHPad + 3) & ~3;
    const size_t smem = (size_t)warps * (kHRing * kHStage + words) * sizeof(float);
    static_assert(warps * (kHRing * kHStage + 9 * kMaxAdjacency + kHPad + 3) * sizeof(float) <= 48 * 1024, "no opt-in needed");
    // about six nodes per warp (3.5 to 7 measured alike; one or fourteen cost
    // 5 %), or all the chip's warps on a small mesh
    const int64_t nodes = nnodes - n_begin, ctas = (nodes + warps - 1) / warps;
    const unsigned grid = (unsigned)std::min<int64_t>(ctas, std::max<int64_t>((ctas + 5) / 6, (int64_t)sm_count() * 16));
    if (grid == 0) return;
    k_hyper_rows<<<grid, 32 * warps, smem, s>>>(g.inc_ptr.p, g.inc.p, g.slots.p, g.adj_ptr.p, stage, vals, res, nnodes,
                                                words, n_begin);
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_hyper_residual(const Graph &g, const float *geo, const int32_t *conn, int64_t ne, const double *u,
                           const LawParams &law, const HyperTables &tab, const QPDerivs *qpd,
                           const uint8_t *qp_fallback, float *stage, double *res, int *d_err, cudaStream_t s,
                           LaunchCounter &lc) {
    if (ne > 0) {
        const unsigned grid = ceil_div(ne, 128);
#define FEDD_HYPER_RES(LAWK) \
    k_hyper_residual<LAWK><<<grid, 128, 0, s>>>(geo, conn, ne, u, law, qpd, qp_fallback, stage, d_err, tab)
        switch (law.kind) {
        case kLawSKR2: FEDD_HYPER_RES(kLawSKR2); break;
        case kLawSKR3: FEDD_HYPER_RES(kLawSKR3); break;
        case kLawAniso: FEDD_HYPER_RES(kLawAniso); break;
        case kLawMLP: FEDD_HYPER_RES(kLawMLP); break;
        default: FEDD_HYPER_RES(kLawSKR1); break;
        }
#undef FEDD_HYPER_RES
        FEDD_CUDA(cudaGetLastError());
        lc.n++;
    }
    if (g.nrow_nodes > 0) {
        k_hyper_residual_rows<<<ceil_div(g.nrow_nodes, 128), 128, 0, s>>>(g.inc_ptr.p, g.inc.p, stage, g.nrow_nodes,
                                                                          res);
        FEDD_CUDA(cudaGetLastError());
        lc.n++;
    }
}

void launch_hyper_invariants(const float *geo, const int32_t *conn, int64_t ne, const double *u,
                             const LawParams &law, const HyperTables &tab, float *inv, int *d_err, cudaStream_t s,
                             LaunchCounter &lc, int64_t e_begin, int64_t e_end) {
    if (e_end < 0) e_end = ne;
    if (e_end <= e_begin) return;
    k_hyper_invariants<<<ceil_div(e_end - e_begin, 128), 128, 0, s>>>(geo, conn, ne, u, law, inv, d_err, e_begin,
                                                                        e_end, tab);
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_law_eval(const LawParams &law, const MLPDev *m, int64_t n, const double *F, double *psi, double *P,
                     double *A, cudaStream_t s) {
    MLPDev mm{};
    if (m) mm = *m;
    if (n == 0) return;
    k_law_eval<<<ceil_div(n, 128), 128, 0, s>>>(law, mm, m != nullptr, n, F, psi, P, A);
    FEDD_CUDA(cudaGetLastError());
}

void launch_hyper_dense(const float *stage, int64_t first, int64_t count, double *Ke, double *re, cudaStream_t s) {
    if (count == 0) return;
    k_hyper_dense<<<ceil_div(count * 930, 256), 256, 0, s>>>(stage, first, count, Ke, re);
    FEDD_CUDA(cudaGetLastError());
}

}  // namespace fedd
