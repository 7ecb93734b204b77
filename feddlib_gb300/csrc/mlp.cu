// mlp.cu -- MLP strain-energy surrogate: tensor-core inference with input
// derivatives at every quadrature point, and the training kernels.
//
// The network (no FEDDLib counterpart) maps normalised invariants
// x = (inv - shift) * scale, inv = (I1, J, I4a, I4b), to
//     net(x) = w3 . sp(W2 sp(W1 x + b1) + b2) + b3,   sp = softplus.
// The assembly needs dPsi/dinv and d2Psi/dinv2.  Forward-mode through the
// first layer gives 15 "channels" per point (h1, dh1/dx_k, d2h1/dx_kdx_l)
// that all meet the same second-layer weights, so the second layer is one
// GEMM of [points x 15 channels, H] by W2^T: it runs on the tensor cores
// (mma.sync m16n8k16, bf16 weights, activations split into bf16 hi + lo,
// FP32 accumulation).  Training (FP32, deterministic) minimises the Sobolev
// loss  mean( wpsi (y - t)^2 + wgrad |grad y - g|^2 )  with Adam.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <new>

#include "kernels.cuh"
#include "mlp_dev.cuh"
#include "tcgen05.cuh"

namespace fedd {
namespace {

constexpr int kH = 64;        // tensor-core path width

// bf16 hi part of (x, y) and the bf16 rounding of the remainders: x ~ hi + lo
// to about 16 significant bits; x goes to the low half of each word (the
// lower K index of a K-major operand)
__device__ __forceinline__ void split_bf16(float x, float y, uint32_t &hi, uint32_t &lo) {
    uint32_t h, l;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(y), "f"(x));
    const float xh = __uint_as_float(h << 16), yh = __uint_as_float(h & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(y - yh), "f"(x - xh));
    hi = h;
    lo = l;
}

// ---- quadrature-point derivatives on the fifth-generation tensor cores ------
// Tiles of 128 quadrature points (M = 128: point r of the tile in TMEM lane
// r), two threads per point: thread (r, h) of the 256 works on hidden units
// [32 h, 32 h + 32) (warps h * 4 .. h * 4 + 3 reach TMEM lanes 0-127).  With
// s1 = sigmoid(z1), t1 = s1 (1 - s1), D_k = W2 (s1 * W1[:, k]),
// s2 = sigmoid(z2), t2 = s2 (1 - s2):
//   dnet/dx_k       = sum_j w3_j s2_j D_kj
//   d2net/dx_k dx_l = sum_j w3_j t2_j D_kj D_lj + sum_i beta_i t1_i W1_ik W1_il,
//   beta = W2^T (w3 * s2)   (the backward product replaces the forward
//                            second-derivative channels).
// Layer 1 runs on the CUDA cores, its weights read from the constant bank.
// Its NC = 1 + NA channels (h1 = sp(z1), and s1 * W1[:, k] for the NA active
// inputs), split into bf16 hi + lo parts, are the A operands (K-major,
// 128 x 64) of layer 2: tcgen05.mma kind::f16 with W2 (bf16) as B and FP32
// accumulators in TMEM, 64 columns per channel.  The layer-2 epilogue reads
// them back, forms G and the first Hessian term, and writes w3 * s2 (hi +
// lo) as the A operand of the backward product beta = W2^T (w3 s2), which
// accumulates in channel 0's columns; the second Hessian term follows from
// beta and the t1 kept in registers.  The two threads of a point add their
// partial sums through shared memory.  One thread issues the MMAs and
// commits them to an mbarrier; every wait is bounded.
constexpr int kQT = 128;                      // points per tile
constexpr int kQThreads = 2 * kQT;            // threads per CTA: two per point
constexpr int kMA = kQT * kH * 2;             // bytes of one 128 x 64 bf16 operand (4 K steps of 4,096)
constexpr int kMB = kH * kH * 2;              // bytes of one 64 x 64 bf16 operand (4 K steps of 2,048)
constexpr uint32_t kMlpWaitPolls = 1u << 20;  // bounded MMA waits (each poll sleeps ~32 ns)

// byte offset of the 8-element chunk kc (K = 8 kc .. 8 kc + 7) of row r in a
// K-major unswizzled bf16 operand: 8-row x 16-byte core matrices, the two of
// one K step (16) 128 B apart (LBO), row groups 256 B apart (SBO), K steps
// `step` bytes apart
__host__ __device__ constexpr int mlp_off(int r, int kc, int step) {
    return (kc >> 1) * step + (r >> 3) * 256 + (kc & 1) * 128 + (r & 7) * 16;
}
// shared memory: the channels' A operands (hi, lo), W2 and W2^T as B, mbarrier + TMEM address
template <int NA> __host__ __device__ constexpr size_t mlp_smem() {
    return (size_t)(1 + NA) * 2 * kMA + 2 * (size_t)kMB + 16;
}
template <int NA> __host__ __device__ constexpr uint32_t mlp_tmem_cols() {
    return (1 + NA) * 64 <= 128 ? 128u : ((1 + NA) * 64 <= 256 ? 256u : 512u);
}

template <int NA>
__global__ void __launch_bounds__(kQThreads) k_mlp_qp_tc(MLPDev m, const float *__restrict__ inv, int64_t nqp,
                                                         QPDerivs *out, uint8_t *fb, int *fb_count, int *err) {
    constexpr int NC = 1 + NA, NH = NA * (NA + 1) / 2;
    constexpr uint32_t kCols = mlp_tmem_cols<NA>();
    static_assert(NC >= 2 || NA == 1, "channels");
    extern __shared__ __align__(1024) uint8_t ms[];
    uint8_t *sA = ms;                  // [channel][hi, lo][kMA]; after layer 2 channel 0 holds w3 s2
    uint8_t *sB1 = ms + NC * 2 * kMA;  // W2 as B: row j, K = i
    uint8_t *sB2 = sB1 + kMB;          // W2^T as B: row i, K = j
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sB2 + kMB);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 1);
    // the upper threads' partial sums (channel 1's operand, free once layer 2 is done)
    float *sPart = reinterpret_cast<float *>(sA + 2 * kMA);
    const int tid = threadIdx.x, w = tid >> 5, r = tid & (kQT - 1), hh = tid >> 7;
    const MlpConst &c = m.c;
    const uint16_t *W2 = static_cast<const uint16_t *>(m.W2);
    for (int t = tid; t < kH * 8; t += kQThreads) {
        const int n = t >> 3, kc = t & 7;
        uint32_t b1w[4], b2w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k0 = 8 * kc + 2 * q;
            b1w[q] = (uint32_t)W2[n * kH + k0] | ((uint32_t)W2[n * kH + k0 + 1] << 16);
            b2w[q] = (uint32_t)W2[k0 * kH + n] | ((uint32_t)W2[(k0 + 1) * kH + n] << 16);
        }
        *reinterpret_cast<uint4 *>(sB1 + mlp_off(n, kc, 2048)) = make_uint4(b1w[0], b1w[1], b1w[2], b1w[3]);
        *reinterpret_cast<uint4 *>(sB2 + mlp_off(n, kc, 2048)) = make_uint4(b2w[0], b2w[1], b2w[2], b2w[3]);
    }
    if (w == 0) tc::tmem_alloc(tslot, kCols);
    if (tid == 0) tc::mbar_init(mbar, 1);
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;
    const uint32_t trow = tmem + ((uint32_t)(32 * (w & 3)) << 16);  // this warp's 32 TMEM lanes
    constexpr uint32_t idesc = tc::idesc_bf16(kQT, kH);
    const uint32_t aBase = tc::smem_u32(sA), b1Base = tc::smem_u32(sB1), b2Base = tc::smem_u32(sB2);
    const int64_t ntiles = (nqp + kQT - 1) / kQT;
    uint32_t phase = 0;
    bool ok = true;
    // this thread's invariants, loaded one tile ahead
    auto load_inv = [&](int64_t tile) {
        const int64_t qq = tile * kQT + r;
        return qq < nqp ? reinterpret_cast<const float4 *>(inv)[qq] : make_float4(3.f, 1.f, 1.f, 1.f);
    };
    float4 v_next = load_inv(blockIdx.x);
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t q = tile * kQT + r;
        bool inside = q < nqp;
        const float4 v4 = v_next;
        if (tile + gridDim.x < ntiles) v_next = load_inv(tile + gridDim.x);
        const float a4[4] = {v4.x, v4.y, v4.z, v4.w};
        // inputs, and the chain factors dx_k / dinv_k, d2x_k / dinv_k2 of the active ones
        float x[4], dk[NA], d2k[NA];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            inside = inside && a4[k] >= m.inv_lo[k] && a4[k] <= m.inv_hi[k];
            float d, h;
            x[k] = mlp_input(m, k, a4[k], d, h);
#pragma unroll
            for (int a = 0; a < NA; a++)
                if (c.act[a] == k) {
                    dk[a] = d;
                    d2k[a] = h;
                }
        }
        // layer 1 over this thread's 32 units, eight at a time: one 16-byte
        // chunk per channel and part
        float t1[kH / 2];
#pragma unroll
        for (int g = 0; g < 4; g++) {
            float v[NC][8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int i = 32 * hh + 8 * g + u;
                float z = c.b1[i];
#pragma unroll
                for (int k = 0; k < 4; k++) z = fmaf(c.W1[i][k], x[k], z);
                // softplus and sigmoid from one exponential, e = exp(-|z|) in
                // (0, 1]: sp = max(z, 0) + log(1 + e), s = 1 / (1 + e) or e / (1 + e);
                // fast-math log and reciprocal (a few ulp, below the bf16 hi + lo
                // rounding of the layer-2 operand)
                const float e1 = __expf(-fabsf(z)), r1 = __fdividef(1.0f, 1.0f + e1);
                const float s1 = z >= 0.0f ? r1 : e1 * r1;
                t1[8 * g + u] = s1 * (1.0f - s1);
                v[0][u] = fmaxf(z, 0.0f) + __logf(1.0f + e1);
#pragma unroll
                for (int a = 0; a < NA; a++) v[1 + a][u] = s1 * c.Wact[a][i];
            }
            const int o = mlp_off(r, 4 * hh + g, 4096);
#pragma unroll
            for (int ch = 0; ch < NC; ch++) {
                uint32_t hw[4], lw[4];
#pragma unroll
                for (int p = 0; p < 4; p++) split_bf16(v[ch][2 * p], v[ch][2 * p + 1], hw[p], lw[p]);
                *reinterpret_cast<uint4 *>(sA + (2 * ch) * kMA + o) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                *reinterpret_cast<uint4 *>(sA + (2 * ch + 1) * kMA + o) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            }
        }
        tc::fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int ch = 0; ch < NC; ch++)
#pragma unroll
                for (int part = 0; part < 2; part++)
#pragma unroll
                    for (int ks = 0; ks < 4; ks++)
                        tc::mma_bf16(tmem + 64 * ch, tc::smem_desc(aBase + (2 * ch + part) * kMA + ks * 4096, 128, 256),
                                     tc::smem_desc(b1Base + ks * 2048, 128, 256), idesc, (part | ks) != 0);
            tc::commit(mbar);
        }
        const bool done = tc::mbar_wait(mbar, phase, kMlpWaitPolls);
        phase ^= 1u;
        if (__syncthreads_or(!done)) {
            ok = false;
            break;
        }
        tc::fence_after_sync();
        // layer-2 epilogue over this thread's 32 units, 16 at a time; w3 s2
        // (hi + lo) becomes channel 0's operand (layer 2 has completed)
        float G[NA], Hh[NH];
#pragma unroll
        for (int a = 0; a < NA; a++) G[a] = 0.0f;
#pragma unroll
        for (int a = 0; a < NH; a++) Hh[a] = 0.0f;
#pragma unroll
        for (int jj = 0; jj < 2; jj++) {
            const int jc = 2 * hh + jj;
            float z2[16], dd[NA][16], vv[16];
            tc::tmem_ld16(trow + 16 * jc, z2);
#pragma unroll
            for (int a = 0; a < NA; a++) tc::tmem_ld16(trow + 64 * (1 + a) + 16 * jc, dd[a]);
#pragma unroll
            for (int u = 0; u < 16; u++) {
                const int j = 16 * jc + u;
                // sigmoid with a fast reciprocal (a few ulp, below the bf16
                // hi + lo rounding of the backward product's operand)
                const float zz = z2[u] + c.b2[j];
                const float e2 = __expf(-fabsf(zz)), r2 = __fdividef(1.0f, 1.0f + e2);
                const float s2 = zz >= 0.0f ? r2 : e2 * r2;
                const float cs = c.w3[j] * s2, ct = c.w3[j] * (s2 * (1.0f - s2));
                int ab = 0;
#pragma unroll
                for (int a = 0; a < NA; a++) {
                    G[a] = fmaf(cs, dd[a][u], G[a]);
                    const float cd = ct * dd[a][u];
#pragma unroll
                    for (int b = a; b < NA; b++, ab++) Hh[ab] = fmaf(cd, dd[b][u], Hh[ab]);
                }
                vv[u] = cs;
            }
#pragma unroll
            for (int hf = 0; hf < 2; hf++) {
                uint32_t hw[4], lw[4];
#pragma unroll
                for (int p = 0; p < 4; p++) split_bf16(vv[8 * hf + 2 * p], vv[8 * hf + 2 * p + 1], hw[p], lw[p]);
                const int o = mlp_off(r, 2 * jc + hf, 4096);
                *reinterpret_cast<uint4 *>(sA + o) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                *reinterpret_cast<uint4 *>(sA + kMA + o) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            }
        }
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int part = 0; part < 2; part++)
#pragma unroll
                for (int ks = 0; ks < 4; ks++)
                    tc::mma_bf16(tmem, tc::smem_desc(aBase + part * kMA + ks * 4096, 128, 256),
                                 tc::smem_desc(b2Base + ks * 2048, 128, 256), idesc, (part | ks) != 0);
            tc::commit(mbar);
        }
        const bool done2 = tc::mbar_wait(mbar, phase, kMlpWaitPolls);
        phase ^= 1u;
        if (__syncthreads_or(!done2)) {
            ok = false;
            break;
        }
        tc::fence_after_sync();
        // sum_i beta_i t1_i W1_ik W1_il over this thread's units
#pragma unroll
        for (int ii = 0; ii < 2; ii++) {
            const int ic = 2 * hh + ii;
            float bt[16];
            tc::tmem_ld16(trow + 16 * ic, bt);
#pragma unroll
            for (int u = 0; u < 16; u++) {
                const int i = 16 * ic + u;
                const float b = bt[u] * t1[16 * ii + u];
                int ab = 0;
#pragma unroll
                for (int a = 0; a < NA; a++) {
                    const float bw = b * c.Wact[a][i];
#pragma unroll
                    for (int b2 = a; b2 < NA; b2++, ab++) Hh[ab] = fmaf(bw, c.Wact[b2][i], Hh[ab]);
                }
            }
        }
        // the upper thread of each point hands its partial sums to the lower one
        if (hh == 1) {
#pragma unroll
            for (int a = 0; a < NA; a++) sPart[(NA + NH) * r + a] = G[a];
#pragma unroll
            for (int a = 0; a < NH; a++) sPart[(NA + NH) * r + NA + a] = Hh[a];
        }
        __syncthreads();
        if (hh == 0) {
#pragma unroll
            for (int a = 0; a < NA; a++) G[a] += sPart[(NA + NH) * r + a];
#pragma unroll
            for (int a = 0; a < NH; a++) Hh[a] += sPart[(NA + NH) * r + NA + a];
        }
        if (hh == 0 && q < nqp) {
            // scatter to the packed (I1, J, I4a, I4b) layout with static indices
            QPDerivs d;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float v = 0.0f;
#pragma unroll
                for (int a = 0; a < NA; a++)
                    if (c.act[a] == k) v = m.out_scale * G[a] * dk[a];
                d.d1[k] = v;
            }
            int kl = 0;
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int l = k; l < 4; l++, kl++) {
                    // packed symmetric index of (k, l), k <= l: 00,01,02,03,11,12,13,22,23,33
                    float v = 0.0f;
                    int ab = 0;
#pragma unroll
                    for (int a = 0; a < NA; a++)
#pragma unroll
                        for (int b = a; b < NA; b++, ab++)
                            if (c.act[a] == k && c.act[b] == l)
                                v = m.out_scale * (Hh[ab] * dk[a] * dk[b] + (a == b ? G[a] * d2k[a] : 0.0f));
                    d.d2[kl] = v;
                }
            out[q] = d;
            fb[q] = inside ? 0 : 1;
            if (!inside) atomicAdd(fb_count, 1);
        }
        tc::fence_before_sync();
        __syncthreads();
    }
    if (!ok) {
        // the MMAs did not complete in time: report it, give them a second
        // bounded wait, then free the tensor memory all the same
        if (tid == 0) set_dev_error(err, kDevTimeout);
        tc::mbar_wait(mbar, phase ^ 1u, kMlpWaitPolls);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (w == 0) tc::tmem_dealloc(tmem, kCols);
}

// general width: one thread per point (CUDA cores)
__global__ void k_mlp_qp_scalar(MLPDev m, const float *__restrict__ inv, int64_t nqp, QPDerivs *out, uint8_t *fb,
                                int *fb_count) {
    int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= nqp) return;
    float4 v = reinterpret_cast<const float4 *>(inv)[q];
    float a[4] = {v.x, v.y, v.z, v.w}, x[4], dk[4], d2k[4];
    bool inside = true;
    for (int k = 0; k < 4; k++) {
        inside = inside && a[k] >= m.inv_lo[k] && a[k] <= m.inv_hi[k];
        x[k] = mlp_input(m, k, a[k], dk[k], d2k[k]);
    }
    float y, g[4], h[16];
    mlp_eval_scalar(m, x, y, g, h);
    QPDerivs d;
    int kl = 0;
    for (int k = 0; k < 4; k++) {
        d.d1[k] = m.out_scale * g[k] * dk[k];
        for (int l = k; l < 4; l++, kl++)
            d.d2[kl] = m.out_scale * (h[4 * k + l] * dk[k] * dk[l] + (k == l ? g[k] * d2k[k] : 0.0f));
    }
    out[q] = d;
    fb[q] = inside ? 0 : 1;
    if (!inside) atomicAdd(fb_count, 1);
}

int sms() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}


template <int NA>
void launch_mlp_qp_tc(const MLPDev &m, const float *inv, int64_t nqp, QPDerivs *out, uint8_t *fallback, int *d_count,
                      int *d_err, cudaStream_t s) {
    constexpr size_t smem = mlp_smem<NA>();
    // CTAs per SM: shared memory (and, for two active inputs, the 512 TMEM columns) allow two up to NA = 2
    const int per_sm = NA <= 2 ? 2 : 1;
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(nqp, kQT), (int64_t)sms() * per_sm);
    FEDD_CUDA(cudaFuncSetAttribute(k_mlp_qp_tc<NA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_mlp_qp_tc<NA><<<grid, kQThreads, smem, s>>>(m, inv, nqp, out, fallback, d_count, d_err);
}

}  // namespace

void launch_mlp_qp(const MLPDev &m, const LawParams &law, const float *inv, int64_t nqp, QPDerivs *out,
                   uint8_t *fallback, int *d_count, int *d_err, cudaStream_t s, LaunchCounter &lc) {
    (void)law;
    if (nqp == 0) return;
    if (m.hidden == kH && m.c.nact > 0) {
        switch (m.c.nact) {
        case 1: launch_mlp_qp_tc<1>(m, inv, nqp, out, fallback, d_count, d_err, s); break;
        case 2: launch_mlp_qp_tc<2>(m, inv, nqp, out, fallback, d_count, d_err, s); break;
        case 3: launch_mlp_qp_tc<3>(m, inv, nqp, out, fallback, d_count, d_err, s); break;
        default: launch_mlp_qp_tc<4>(m, inv, nqp, out, fallback, d_count, d_err, s); break;
        }
    } else {
        k_mlp_qp_scalar<<<ceil_div(nqp, 128), 128, 0, s>>>(m, inv, nqp, out, fallback, d_count);
    }
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

// ============================ training =====================================
namespace {

// C[M x N] = sum_k A(m,k) B(k,n), FP32, 64x64 tiles, 256 threads (4x4 each).
// TA: A stored K x M (A(m,k) = A[k*lda + m]) else M x K.
// TB: B stored N x K (B(k,n) = B[n*ldb + k]) else K x N.
// Split-K: blockIdx.z handles K range [z*kc, (z+1)*kc), writes C + z*M*N.
template <bool TA, bool TB>
__global__ void k_sgemm(const float *__restrict__ A, const float *__restrict__ B, float *C, int M, int N, int64_t K,
                        int64_t kc) {
    __shared__ float As[16][65], Bs[16][65];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    const int64_t k_begin = (int64_t)blockIdx.z * kc, k_end = std::min<int64_t>(K, k_begin + kc);
    float acc[4][4] = {{0}};
    for (int64_t k0 = k_begin; k0 < k_end; k0 += 16) {
        for (int t = threadIdx.x; t < 16 * 64; t += 256) {
            const int kk = t / 64, mm = t % 64;
            const int64_t k = k0 + kk;
            float av = 0.0f, bv = 0.0f;
            if (k < k_end) {
                const int gm = m0 + mm, gn = n0 + mm;
                if (gm < M) av = TA ? A[k * M + gm] : A[(int64_t)gm * K + k];
                if (gn < N) bv = TB ? B[(int64_t)gn * K + k] : B[k * N + gn];
            }
            As[kk][mm] = av;
            Bs[kk][mm] = bv;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; kk++)
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(As[kk][ty * 4 + i], Bs[kk][tx * 4 + j], acc[i][j]);
        __syncthreads();
    }
    float *Cz = C + (int64_t)blockIdx.z * M * N;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gm = m0 + ty * 4 + i, gn = n0 + tx * 4 + j;
            if (gm < M && gn < N) Cz[(int64_t)gm * N + gn] = acc[i][j];
        }
}

// out[c] = sum over rows r (fixed order) of in[r * cols + c]
__global__ void k_colsum(const float *__restrict__ in, int64_t rows, int cols, float *out) {
    __shared__ float red[256];
    const int c = blockIdx.x;
    float s = 0.0f;
    for (int64_t r = threadIdx.x; r < rows; r += blockDim.x) s += in[r * cols + c];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = red[0];
}

struct TrainParams {
    const float *W1, *b1, *W2, *b2, *w3, *b3;
};

// forward layer 1: X1 = [H1; DH1_0..3] (5B x H), caches S1, T1
__global__ void k_tr_l1(TrainParams P, int H, const float *__restrict__ X, const int64_t *__restrict__ idx, int64_t B,
                        float *X1, float *S1, float *T1) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= B * H) return;
    const int64_t s = t / H;
    const int i = (int)(t - s * H);
    const float *x = X + 4 * (idx ? idx[s] : s);
    float z = P.b1[i];
    for (int k = 0; k < 4; k++) z = fmaf(P.W1[4 * i + k], x[k], z);
    const float sg = 1.0f / (1.0f + expf(-z)), tg = sg * (1.0f - sg);
    const float hv = z > 20.0f ? z : log1pf(expf(z));
    X1[s * H + i] = hv;
    for (int k = 0; k < 4; k++) X1[((1 + k) * B + s) * H + i] = sg * P.W1[4 * i + k];
    S1[s * H + i] = sg;
    T1[s * H + i] = tg;
}

// forward layer 2 + loss + start of the backward pass, one warp per sample
__global__ void k_tr_l2(TrainParams P, int H, const float *__restrict__ Z2, const float *__restrict__ ty,
                        const float *__restrict__ tgr, const int64_t *__restrict__ idx, int64_t B, float wpsi,
                        float wgrad, float *D, float *GW3, float *lossv, float *ey_out) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= B) return;
    float yp = 0.0f, gp[4] = {0, 0, 0, 0};
    for (int j = lane; j < H; j += 32) {
        const float z = Z2[s * H + j] + P.b2[j];
        const float sg = 1.0f / (1.0f + expf(-z));
        yp = fmaf(P.w3[j], z > 20.0f ? z : log1pf(expf(z)), yp);
        for (int k = 0; k < 4; k++) gp[k] = fmaf(P.w3[j] * sg, Z2[((1 + k) * B + s) * H + j], gp[k]);
    }
    const float y = warp_sum(yp) + *P.b3;
    float g[4];
    for (int k = 0; k < 4; k++) g[k] = warp_sum(gp[k]);
    const int64_t si = idx ? idx[s] : s;
    const float ey = 2.0f * wpsi * (y - ty[si]);
    float eg[4], l = wpsi * (y - ty[si]) * (y - ty[si]);
    for (int k = 0; k < 4; k++) {
        const float dk = g[k] - tgr[4 * si + k];
        eg[k] = 2.0f * wgrad * dk;
        l += wgrad * dk * dk;
    }
    for (int j = lane; j < H; j += 32) {
        const float z = Z2[s * H + j] + P.b2[j];
        const float sg = 1.0f / (1.0f + expf(-z)), tg = sg * (1.0f - sg);
        const float hv = z > 20.0f ? z : log1pf(expf(z));
        float dz2 = ey * P.w3[j] * sg, gw = ey * hv;
        for (int k = 0; k < 4; k++) {
            const float dzk = Z2[((1 + k) * B + s) * H + j];
            dz2 = fmaf(eg[k] * P.w3[j] * tg, dzk, dz2);
            gw = fmaf(eg[k] * sg, dzk, gw);
            D[((1 + k) * B + s) * H + j] = eg[k] * P.w3[j] * sg;
        }
        D[s * H + j] = dz2;
        GW3[s * H + j] = gw;
    }
    if (lane == 0) {
        lossv[s] = l;
        ey_out[s] = ey;
    }
}

// backward through layer 1: per-sample contributions to gW1 and gb1
__global__ void k_tr_l1b(TrainParams P, int H, const float *__restrict__ X, const int64_t *__restrict__ idx, int64_t B,
                         const float *__restrict__ DX1, const float *__restrict__ S1, const float *__restrict__ T1,
                         float *G1) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= B * H) return;
    const int64_t s = t / H;
    const int i = (int)(t - s * H);
    const float *x = X + 4 * (idx ? idx[s] : s);
    const float sg = S1[s * H + i], tg = T1[s * H + i];
    float dz = DX1[s * H + i] * sg;
    float dd[4];
    for (int k = 0; k < 4; k++) {
        dd[k] = DX1[((1 + k) * B + s) * H + i];
        dz = fmaf(dd[k] * tg, P.W1[4 * i + k], dz);
    }
    // layout per sample: [gW1 (H x 4) | gb1 (H)]
    float *o = G1 + s * (5 * H);
    for (int k = 0; k < 4; k++) o[4 * i + k] = dd[k] * sg + dz * x[k];
    o[4 * H + i] = dz;
}

// ---- width 64: one kernel for the forward and backward passes -------------
// The network's 5 channels (h and its four input derivatives) of a sample meet
// three 64 x 64 products: Z2 = X1 W2^T, DX1 = D W2 and gW2 = D^T X1.  As
// separate kernels they moved the five-channel matrices X1, Z2, D and DX1
// through memory nine times (84 MB each at a batch of 65,536), and the last
// one ran on 80 of the blocks the chip holds.  Here a CTA takes tiles of
// GROUPS x SPT samples and keeps them in shared memory: thread (s, c) owns
// hidden units 4 c .. 4 c + 3 of the samples s, s + GROUPS in all five
// channels, so the layer formulas between the products run on registers, and a
// block of gW2, which stays in registers over all tiles of the CTA, as do the
// thread's sums of the other gradients.  Each CTA writes one partial sum of
// every gradient; k_tr_update adds them in a fixed order and takes the Adam
// step.  FP32 throughout, two multiply-adds to an instruction in the products
// (3 x 20,480 per sample).  A 16-byte read that serves one sample's row and
// four weights is four of the shared-memory pipe's cycles to 20 multiply-adds:
// with one sample per thread that pipe is the bound (78 %), with two the FP32
// pipe.  For a batch of 65,536: 1,590 us of separate kernels; 213 us one
// sample per thread with scalar multiply-adds; 203 packed; 184 two samples and
// 384 threads (205 with 256: two warps per scheduler are too few); k_tr_update
// another 7 us.
constexpr int kTRows = 16;               // samples of a tile that one share of gW2 adds
constexpr int kTSample = 5 * kH + 4;     // floats per sample: five channels, and 4 so that two samples' rows differ in banks
constexpr int kTPar = 4 * kH + kH + kH * kH + kH + kH + 2;  // gradients in the parameters' order, then the loss
constexpr size_t tr_smem(int groups, int spt) {
    return (size_t)(2 * kH * kH + 2 * groups * spt * kTSample + 4 * kH + 3 * kH) * sizeof(float);
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, const float *v) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// acc[c] += x w for the four columns of w, two to an instruction
__device__ __forceinline__ void fma4(float *acc, float x, const float4 &w) {
    asm("{.reg .b64 x, w, a;\n\tmov.b64 x, {%2, %2};\n\tmov.b64 w, {%3, %4};\n\tmov.b64 a, {%0, %1};\n\t"
        "fma.rn.f32x2 a, x, w, a;\n\tmov.b64 {%0, %1}, a;}"
        : "+f"(acc[0]), "+f"(acc[1])
        : "f"(x), "f"(w.x), "f"(w.y));
    asm("{.reg .b64 x, w, a;\n\tmov.b64 x, {%2, %2};\n\tmov.b64 w, {%3, %4};\n\tmov.b64 a, {%0, %1};\n\t"
        "fma.rn.f32x2 a, x, w, a;\n\tmov.b64 {%0, %1}, a;}"
        : "+f"(acc[2]), "+f"(acc[3])
        : "f"(x), "f"(w.z), "f"(w.w));
}
// acc[m][ch][c] = sum_i rows[m][ch][i] W[i][u0 + c] over 64 i, samples `apart` floats apart
template <int SPT>
__device__ __forceinline__ void tile_product(float acc[SPT][5][4], const float *rows, int apart, const float *W, int u0) {
#pragma unroll
    for (int k = 0; k < SPT * 20; k++) (&acc[0][0][0])[k] = 0.0f;
#pragma unroll 2
    for (int i = 0; i < kH; i += 4) {
        const float4 w0 = ld4(W + i * kH + u0), w1 = ld4(W + (i + 1) * kH + u0), w2 = ld4(W + (i + 2) * kH + u0),
                     w3 = ld4(W + (i + 3) * kH + u0);
#pragma unroll
        for (int m = 0; m < SPT; m++) {
            float4 x[5];
#pragma unroll
            for (int ch = 0; ch < 5; ch++) x[ch] = ld4(rows + m * apart + kH * ch + i);
#pragma unroll
            for (int ch = 0; ch < 5; ch++) {
                fma4(acc[m][ch], x[ch].x, w0);
                fma4(acc[m][ch], x[ch].y, w1);
                fma4(acc[m][ch], x[ch].z, w2);
                fma4(acc[m][ch], x[ch].w, w3);
            }
        }
    }
}

// a sum with the rounding errors of its additions kept beside it (Knuth's
// two-sum), for the last levels of the gradients' sums and for b3's and the
// loss's, where many terms cancel: b3 after eight steps of 65,536 samples is
// 2.6e-7 off on average over 18 seeds, 2.9e-7 with plain sums over the tiles,
// 3.6e-7 with plain sums throughout (a trainer's creation on 200,000 samples and
// the eight steps take 2,207, 2,192 and 2,188 us); the loss, an evaluation at the
// updated parameters, is 5.6e-7 off in all three
struct TwoSum {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        const float t = __fadd_rn(s, x), xx = __fsub_rn(t, s);
        c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, xx)), __fsub_rn(x, xx)));
        s = t;
    }
    // an infinite sum's errors are not numbers: the sum itself
    __device__ __forceinline__ float value() const {
        const float v = __fadd_rn(s, c);
        return isfinite(v) ? v : s;
    }
};

// samples idx[0..B) (null: 0..B) in tiles of GROUPS SPT; part: gridDim.x x kTPar
template <int GROUPS, int SPT>
__global__ void __launch_bounds__(16 * GROUPS, SPT == 1 ? 2 : 1)
    k_tr_fused(TrainParams P, const float *__restrict__ X, const float *__restrict__ ty, const float *__restrict__ tgr,
               const int64_t *__restrict__ idx, int64_t B, float wpsi, float wgrad, float *__restrict__ part) {
    constexpr int TS = GROUPS * SPT, THREADS = 16 * GROUPS;
    // rows of the thread's gW2 block; SHARES threads own one, each adding kTRows samples of a tile
    constexpr int JB = 4 * SPT, SHARES = TS / kTRows;
    extern __shared__ __align__(16) float sm[];
    float *sW = sm, *sWT = sW + kH * kH;               // W2[j][i] and W2[j][i] at [i][j]
    float *sX = sWT + kH * kH, *sD = sX + TS * kTSample;
    float *sW1 = sD + TS * kTSample, *sb1 = sW1 + 4 * kH, *sb2 = sb1 + kH, *sw3 = sb2 + kH;
    const int tid = threadIdx.x, s = tid >> 4, u0 = 4 * (tid & 15);
    const int share = s / (kH / JB), j0 = JB * (s % (kH / JB));
    for (int t = tid; t < kH * kH; t += THREADS) {
        const float w = P.W2[t];
        sW[t] = w;
        sWT[(t & (kH - 1)) * kH + (t >> 6)] = w;
    }
    if (tid < 4 * kH) sW1[tid] = P.W1[tid];
    if (tid < kH) {
        sb1[tid] = P.b1[tid];
        sb2[tid] = P.b2[tid];
        sw3[tid] = P.w3[tid];
    }
    const float b3 = *P.b3;
    __syncthreads();
    float *xrow = sX + s * kTSample, *drow = sD + s * kTSample;
    float gW2[JB][4], gW1[4][4], gb1[4], gb2[4], gw3[4];
    TwoSum gb3, loss;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        gb1[a] = gb2[a] = gw3[a] = 0.0f;
#pragma unroll
        for (int b = 0; b < 4; b++) gW1[a][b] = 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 4 * JB; k++) (&gW2[0][0])[k] = 0.0f;
    const int64_t ntiles = (B + TS - 1) / TS;
    auto sample = [&](int64_t tile, int m) {
        const int64_t q = tile * TS + m * GROUPS + s;
        return q < B ? (idx ? idx[q] : q) : (int64_t)-1;
    };
    int64_t id[SPT];
#pragma unroll
    for (int m = 0; m < SPT; m++) id[m] = blockIdx.x < ntiles ? sample(blockIdx.x, m) : -1;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        bool valid[SPT];
        float x[SPT][4], tg[SPT][4], tyv[SPT], s1[SPT][4];
#pragma unroll
        for (int m = 0; m < SPT; m++) {
            valid[m] = id[m] >= 0;
            // the places behind the last sample hold zeros: their products with the
            // errors, which are zero, stay zero
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 x4 = valid[m] ? ld4(X + 4 * id[m]) : none, t4 = valid[m] ? ld4(tgr + 4 * id[m]) : none;
            x[m][0] = x4.x; x[m][1] = x4.y; x[m][2] = x4.z; x[m][3] = x4.w;
            tg[m][0] = t4.x; tg[m][1] = t4.y; tg[m][2] = t4.z; tg[m][3] = t4.w;
            tyv[m] = valid[m] ? ty[id[m]] : 0.0f;
            if (tile + gridDim.x < ntiles) id[m] = sample(tile + gridDim.x, m);
        }
#pragma unroll
        for (int m = 0; m < SPT; m++) {  // layer 1
            float v[5][4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float4 w = ld4(sW1 + 4 * (u0 + u));
                const float z = fmaf(w.w, x[m][3], fmaf(w.z, x[m][2], fmaf(w.y, x[m][1], fmaf(w.x, x[m][0], sb1[u0 + u]))));
                const float sg = 1.0f / (1.0f + expf(-z));
                s1[m][u] = sg;
                v[0][u] = z > 20.0f ? z : log1pf(expf(z));
                v[1][u] = sg * w.x;
                v[2][u] = sg * w.y;
                v[3][u] = sg * w.z;
                v[4][u] = sg * w.w;
            }
#pragma unroll
            for (int ch = 0; ch < 5; ch++) st4(xrow + m * GROUPS * kTSample + kH * ch + u0, v[ch]);
        }
        __syncwarp();  // a sample's rows are written and read by the same half warp
        float acc[SPT][5][4];
        tile_product<SPT>(acc, xrow, GROUPS * kTSample, sWT, u0);
#pragma unroll
        for (int m = 0; m < SPT; m++) {
            // layer 2, the sample's output, gradient and loss, and the backward rows D
            float sg[4], hv[4], yp = 0.0f, gp[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float z = acc[m][0][u] + sb2[u0 + u], w3 = sw3[u0 + u];
                sg[u] = 1.0f / (1.0f + expf(-z));
                hv[u] = z > 20.0f ? z : log1pf(expf(z));
                yp = fmaf(w3, hv[u], yp);
#pragma unroll
                for (int k = 0; k < 4; k++) gp[k] = fmaf(w3 * sg[u], acc[m][1 + k][u], gp[k]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                yp += __shfl_xor_sync(0xffffffffu, yp, o);
#pragma unroll
                for (int k = 0; k < 4; k++) gp[k] += __shfl_xor_sync(0xffffffffu, gp[k], o);
            }
            const float dy = yp + b3 - tyv[m], ey = valid[m] ? 2.0f * wpsi * dy : 0.0f;
            float eg[4], l = wpsi * dy * dy;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float dk = gp[k] - tg[m][k];
                eg[k] = valid[m] ? 2.0f * wgrad * dk : 0.0f;
                l += wgrad * dk * dk;
            }
            gb3.add(ey);
            loss.add(valid[m] ? l : 0.0f);
            float d[5][4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float w3 = sw3[u0 + u], tg2 = sg[u] * (1.0f - sg[u]);
                float dz2 = ey * w3 * sg[u], gw = ey * hv[u];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    dz2 = fmaf(eg[k] * w3 * tg2, acc[m][1 + k][u], dz2);
                    gw = fmaf(eg[k] * sg[u], acc[m][1 + k][u], gw);
                    d[1 + k][u] = eg[k] * w3 * sg[u];
                }
                d[0][u] = dz2;
                gb2[u] += dz2;
                gw3[u] += gw;
            }
#pragma unroll
            for (int ch = 0; ch < 5; ch++) st4(drow + m * GROUPS * kTSample + kH * ch + u0, d[ch]);
        }
        __syncthreads();
        // gW2 block of the share's samples, five rows each
        const float *gD = sD + share * kTRows * kTSample + j0, *gX = sX + share * kTRows * kTSample + u0;
#pragma unroll 2
        for (int q = 0; q < kTRows; q++)
#pragma unroll
            for (int ch = 0; ch < 5; ch++) {
                const float4 v = ld4(gX + q * kTSample + kH * ch);
#pragma unroll
                for (int a = 0; a < JB; a += 4) {
                    const float4 d = ld4(gD + q * kTSample + kH * ch + a);
                    fma4(gW2[a], d.x, v);
                    fma4(gW2[a + 1], d.y, v);
                    fma4(gW2[a + 2], d.z, v);
                    fma4(gW2[a + 3], d.w, v);
                }
            }
        // backward through layer 2's product and layer 1
        tile_product<SPT>(acc, drow, GROUPS * kTSample, sW, u0);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float4 w = ld4(sW1 + 4 * (u0 + u));
            const float wk[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int m = 0; m < SPT; m++) {
                const float sg = s1[m][u], t1 = sg * (1.0f - sg);
                float dz = acc[m][0][u] * sg;
#pragma unroll
                for (int k = 0; k < 4; k++) dz = fmaf(acc[m][1 + k][u] * t1, wk[k], dz);
#pragma unroll
                for (int k = 0; k < 4; k++) gW1[u][k] += fmaf(dz, x[m][k], acc[m][1 + k][u] * sg);
                gb1[u] += dz;
            }
        }
        __syncthreads();  // the next tile overwrites the rows
    }
    // the CTA's partial sums: the shares of gW2, and the others over the
    // sample groups, through shared memory
    float *out = part + (int64_t)blockIdx.x * kTPar;
    constexpr int kSmall = 7 * kH;  // gW1 (4 per unit), gb1, gb2, gw3
    float *red = sX;                // GROUPS x 448 floats in the rows' place, and behind them the other shares of gW2
    float *red2 = red + GROUPS * kSmall + 2 * GROUPS;
    static_assert(GROUPS * kSmall + 2 * GROUPS + (SHARES - 1) * kH * kH <= 2 * TS * kTSample, "the partial sums fit the rows");
    if (share > 0) {
#pragma unroll
        for (int a = 0; a < JB; a++) st4(red2 + (share - 1) * kH * kH + (j0 + a) * kH + u0, gW2[a]);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
#pragma unroll
        for (int k = 0; k < 4; k++) red[s * kSmall + 4 * (u0 + u) + k] = gW1[u][k];
        red[s * kSmall + 4 * kH + u0 + u] = gb1[u];
        red[s * kSmall + 5 * kH + u0 + u] = gb2[u];
        red[s * kSmall + 6 * kH + u0 + u] = gw3[u];
    }
    if (u0 == 0) {
        red[GROUPS * kSmall + s] = gb3.value();
        red[GROUPS * kSmall + GROUPS + s] = loss.value();
    }
    __syncthreads();
    if (share == 0) {
#pragma unroll
        for (int a = 0; a < JB; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int k = (j0 + a) * kH + u0 + b;
                float v = gW2[a][b];
#pragma unroll
                for (int c = 1; c < SHARES; c++) v += red2[(c - 1) * kH * kH + k];
                out[5 * kH + k] = v;
            }
    }
    for (int t = tid; t < kSmall + 2; t += THREADS) {
        TwoSum v;
        for (int q = 0; q < GROUPS; q++)
            v.add(t < kSmall ? red[q * kSmall + t] : red[GROUPS * kSmall + GROUPS * (t - kSmall) + q]);
        // gW1 | gb1 at the front, gb2 | gw3 | gb3 | loss behind gW2
        out[t < 5 * kH ? t : t + kH * kH] = v.value();
    }
}

// one gradient (or the loss) per lane, eight warps sharing its partial sums;
// with adam the parameter's Adam step, otherwise the sum into grad
__global__ void __launch_bounds__(256) k_tr_update(const float *__restrict__ part, int nparts, int adam, float *grad,
                                                   float *lsum, float *p, float *m1, float *m2, float lr, float b1,
                                                   float b2, float eps, float c1, float c2, float scale) {
    __shared__ float red[8][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    TwoSum sum;
    if (i < kTPar)
        for (int q = w; q < nparts; q += 8) sum.add(part[(int64_t)q * kTPar + i]);
    red[w][lane] = sum.value();
    __syncthreads();
    if (w != 0 || i >= kTPar) return;
#pragma unroll
    for (int q = 1; q < 8; q++) sum.add(red[q][lane]);
    const float v = sum.value();
    if (i == kTPar - 1) {
        *lsum = v;
    } else if (adam) {
        const float gi = v * scale;
        m1[i] = b1 * m1[i] + (1.0f - b1) * gi;
        m2[i] = b2 * m2[i] + (1.0f - b2) * gi * gi;
        p[i] -= lr * (m1[i] / c1) / (sqrtf(m2[i] / c2) + eps);
    } else {
        grad[i] = v;
    }
}

// ---- the seeded shuffle on the device ---------------------------------------
// The sequential shuffle  for i = n - 1 .. 1: swap(perm[i], perm[j_i]),  with
// j_i = draw(n - 1 - i) mod (i + 1), evaluated for all i at once.  Position p
// is written by the steps k > p with j_k = p, which run in descending order,
// so before step k the value at position k is that of position L_k[0] before
// its own step, where L_p lists the steps k > p with j_k = p in ascending
// order, or perm[k] if L_k is empty: V(k) = V(L_k[0]) or perm[k].  The result is
//     out[i] = V(i)                      if j_i = i (and for i = 0)
//            = V(k) or perm[j_i]         with k the successor of i in L_{j_i}.
// Lists and chains have about log n entries.  On the host a shuffle of 200,000
// samples took 1,140 us; these seven launches take 47 us.
__host__ __device__ inline uint64_t sm64_mix(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

__global__ void k_fy_targets(uint64_t seed, int64_t n, int64_t *target, int64_t *count) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t j = i == 0 ? 0 : (int64_t)(sm64_mix(seed + (uint64_t)(n - i) * 0x9E3779B97F4A7C15ULL) % (uint64_t)(i + 1));
    target[i] = j;
    if (j < i) atomicAdd(reinterpret_cast<unsigned long long *>(count + j), 1ull);
}

// counts the lists' cursors down
__global__ void k_fy_fill(const int64_t *__restrict__ target, int64_t n, const int64_t *__restrict__ off, int64_t *count,
                          int64_t *list) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t j = target[i];
    if (j < i) list[off[j] + (int64_t)atomicAdd(reinterpret_cast<unsigned long long *>(count + j), ~0ull) - 1] = i;
}

__global__ void k_fy_sort(int64_t n, const int64_t *__restrict__ off, int64_t *list) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int64_t a = off[p], b = off[p + 1];
    for (int64_t x = a + 1; x < b; x++) {
        const int64_t v = list[x];
        int64_t y = x;
        for (; y > a && list[y - 1] > v; y--) list[y] = list[y - 1];
        list[y] = v;
    }
}

__global__ void k_fy_resolve(int64_t n, const int64_t *__restrict__ target, const int64_t *__restrict__ off,
                             const int64_t *__restrict__ list, const int64_t *__restrict__ perm, int64_t *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t j = target[i];
    int64_t k = i;
    bool chain = true;
    if (j < i) {
        int64_t x = off[j];
        const int64_t b = off[j + 1];
        while (x < b && list[x] != i) x++;
        chain = x + 1 < b;
        k = chain ? list[x + 1] : j;
    }
    if (chain)
        for (;;) {  // strictly ascending
            const int64_t a = off[k];
            if (a == off[k + 1]) break;
            k = list[a];
        }
    out[i] = perm[k];
}

__global__ void k_iota(int64_t *p, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) p[i] = i;
}

__global__ void k_adam(float *p, const float *g, float *m1, float *m2, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2, float scale) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] * scale;
    m1[i] = b1 * m1[i] + (1.0f - b1) * gi;
    m2[i] = b2 * m2[i] + (1.0f - b2) * gi * gi;
    p[i] -= lr * (m1[i] / c1) / (sqrtf(m2[i] / c2) + eps);
}

}  // namespace
}  // namespace fedd

using namespace fedd;

struct fedd_trainer {
    int device = 0, H = 64;
    int64_t n = 0;
    Arena mem;  // the data set, the parameters and their Adam state, the loss
    DBuf<float> X, ty, tg;
    // parameters (flat): W1 (4H) | b1 (H) | W2 (HH) | b2 (H) | w3 (H) | b3 (1)
    DBuf<float> par, grad, m1, m2;
    int64_t step = 0;
    // partial gradients of the width-64 kernel, one set per CTA
    DBuf<float> partials;
    // the sample order (from the first run on) and the shuffle's workspace
    Arena order;
    int64_t *perm = nullptr, *perm_next = nullptr, *fy_target = nullptr, *fy_count = nullptr, *fy_off = nullptr,
            *fy_list = nullptr;
    // workspace for a batch of the general path
    int64_t B = 0;
    DBuf<float> X1, S1, T1, Z2, D, DX1, GW3, G1, lossv, ey, part;
    DBuf<float> lsum;  // the batch's summed loss
    uint64_t rng = 0;
    int64_t cursor = 0;
    std::string err;
    int nparams() const { return 4 * H + H + H * H + H + H + 1; }
    TrainParams tp() const {
        TrainParams t;
        t.W1 = par.p;
        t.b1 = par.p + 4 * H;
        t.W2 = par.p + 5 * H;
        t.b2 = par.p + 5 * H + H * H;
        t.w3 = par.p + 6 * H + H * H;
        t.b3 = par.p + 7 * H + H * H;
        return t;
    }
};

namespace {

void tr_workspace(fedd_trainer *t, int64_t B) {
    if (t->B == B) return;
    const int H = t->H;
    t->B = B;
    t->X1.alloc(5 * B * H);
    t->S1.alloc(B * H);
    t->T1.alloc(B * H);
    t->Z2.alloc(5 * B * H);
    t->D.alloc(5 * B * H);
    t->DX1.alloc(5 * B * H);
    t->GW3.alloc(B * H);
    t->G1.alloc(B * 5 * H);
    t->lossv.alloc(B);
    t->ey.alloc(B);
}

// general width: loss and gradient (sums over the batch, not yet divided by B)
// of the samples idx (null: 0..B) into t->lsum and t->grad
void tr_forward_backward(fedd_trainer *t, const int64_t *idx, int64_t B, float wpsi, float wgrad) {
    const int H = t->H;
    cudaStream_t s = 0;
    const TrainParams P = t->tp();
    k_tr_l1<<<ceil_div(B * H, 256), 256, 0, s>>>(P, H, t->X.p, idx, B, t->X1.p, t->S1.p, t->T1.p);
    {  // Z2 (5B x H) = X1 (5B x H) . W2^T
        dim3 grid(ceil_div(H, 64), ceil_div(5 * B, 64), 1);
        k_sgemm<false, true><<<grid, 256, 0, s>>>(t->X1.p, P.W2, t->Z2.p, (int)(5 * B), H, H, H);
    }
    k_tr_l2<<<ceil_div(B * 32, 256), 256, 0, s>>>(P, H, t->Z2.p, t->ty.p, t->tg.p, idx, B, wpsi, wgrad, t->D.p,
                                                  t->GW3.p, t->lossv.p, t->ey.p);
    float *g = t->grad.p;
    // gradient layout: W1 (4 H) | b1 (H) | W2 (H H) | b2 (H) | w3 (H) | b3; b1's
    // part is written together with W1's (one column sum over 5 H columns)
    float *gW1 = g, *gW2 = g + 5 * H, *gb2 = g + 5 * H + H * H, *gw3 = g + 6 * H + H * H,
          *gb3 = g + 7 * H + H * H;
    {  // gW2 (H x H) = D^T (H x 5B) . X1 (5B x H), split-K then fixed-order sum
        const int64_t K = 5 * B;
        const int64_t nz = std::min<int64_t>(256, (K + 4095) / 4096);
        const int64_t kc = ((K + nz - 1) / nz + 15) / 16 * 16;
        const int64_t zc = (K + kc - 1) / kc;
        if (t->part.n < (size_t)(zc * H * H)) t->part.alloc(zc * H * H);
        dim3 grid(ceil_div(H, 64), ceil_div(H, 64), (unsigned)zc);
        k_sgemm<true, false><<<grid, 256, 0, s>>>(t->D.p, t->X1.p, t->part.p, H, H, K, kc);
        k_colsum<<<H * H, 256, 0, s>>>(t->part.p, zc, H * H, gW2);
    }
    {  // DX1 (5B x H) = D (5B x H) . W2 (H x H)
        dim3 grid(ceil_div(H, 64), ceil_div(5 * B, 64), 1);
        k_sgemm<false, false><<<grid, 256, 0, s>>>(t->D.p, P.W2, t->DX1.p, (int)(5 * B), H, H, H);
    }
    k_tr_l1b<<<ceil_div(B * H, 256), 256, 0, s>>>(P, H, t->X.p, idx, B, t->DX1.p, t->S1.p, t->T1.p, t->G1.p);
    k_colsum<<<5 * H, 256, 0, s>>>(t->G1.p, B, 5 * H, gW1);  // gW1 | gb1 contiguous
    k_colsum<<<H, 256, 0, s>>>(t->D.p, B, H, gb2);
    k_colsum<<<H, 256, 0, s>>>(t->GW3.p, B, H, gw3);
    k_colsum<<<1, 256, 0, s>>>(t->ey.p, B, 1, gb3);
    FEDD_CUDA(cudaGetLastError());
    k_colsum<<<1, 256, 0, s>>>(t->lossv.p, B, 1, t->lsum.p);
    FEDD_CUDA(cudaGetLastError());
}

// width 64: the same, then the Adam step when adam is set (idx null: samples 0..B)
struct AdamStep {
    float lr, b1, b2, eps, c1, c2, scale;
};
void tr_fused(fedd_trainer *t, const int64_t *idx, int64_t B, float wpsi, float wgrad, const AdamStep *adam) {
    cudaStream_t s = 0;
    // tiles of 48 samples, one CTA per SM, or of 16, two per SM: whichever takes
    // less time over its rounds of tiles (20.4 and 14.6 us a round; wall time
    // of a step with its share of the shuffles: 65,536 samples 205 against 226 us, 20,000 77 and
    // 84, 15,000 76 and 69, 30,000 118 and 114)
    const int64_t rounds1 = ceil_div(B, 32 * (int64_t)sms()), rounds2 = ceil_div(B, 48 * (int64_t)sms());
    const int spt = 7 * rounds2 < 5 * rounds1 ? 2 : 1;
    const int groups = spt == 2 ? 24 : 16;
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(B, groups * spt), (int64_t)sms() * (2 / spt));
    const size_t smem = tr_smem(groups, spt);
    if (t->partials.n < (size_t)grid * kTPar) t->partials.alloc((size_t)grid * kTPar);
    auto kern = spt == 2 ? k_tr_fused<24, 2> : k_tr_fused<16, 1>;
    FEDD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, 16 * groups, smem, s>>>(t->tp(), t->X.p, t->ty.p, t->tg.p, idx, B, wpsi, wgrad, t->partials.p);
    const AdamStep a = adam ? *adam : AdamStep{};
    k_tr_update<<<ceil_div(kTPar, 32), 256, 0, s>>>(t->partials.p, (int)grid, adam != nullptr, t->grad.p, t->lsum.p,
                                                    t->par.p, t->m1.p, t->m2.p, a.lr, a.b1, a.b2, a.eps, a.c1, a.c2,
                                                    a.scale);
    FEDD_CUDA(cudaGetLastError());
}

// the sample order and the shuffle's workspace
void tr_order(fedd_trainer *t) {
    if (t->perm) return;
    const int64_t n = t->n;
    t->order.reserve(6 * Arena::bytes<int64_t>(n + 1) + scan_scratch(n + 1));
    t->perm_next = t->order.take<int64_t>(n + 1);
    t->fy_target = t->order.take<int64_t>(n + 1);
    t->fy_count = t->order.take<int64_t>(n + 1);
    t->fy_off = t->order.take<int64_t>(n + 1);
    t->fy_list = t->order.take<int64_t>(n + 1);
    t->perm = t->order.take<int64_t>(n + 1);
    FEDD_CUDA(cudaMemsetAsync(t->fy_count, 0, (n + 1) * sizeof(int64_t), 0));  // k_fy_fill counts it back to zero
}

void tr_shuffle(fedd_trainer *t, uint64_t seed) {
    const int64_t n = t->n;
    const unsigned nb = ceil_div(n, 256);
    k_fy_targets<<<nb, 256>>>(seed, n, t->fy_target, t->fy_count);
    exclusive_scan_i64(t->fy_count, t->fy_off, n + 1, t->order, 0);
    k_fy_fill<<<nb, 256>>>(t->fy_target, n, t->fy_off, t->fy_count, t->fy_list);
    k_fy_sort<<<nb, 256>>>(n, t->fy_off, t->fy_list);
    k_fy_resolve<<<nb, 256>>>(n, t->fy_target, t->fy_off, t->fy_list, t->perm, t->perm_next);
    FEDD_CUDA(cudaGetLastError());
    std::swap(t->perm, t->perm_next);
}

template <class F> fedd_status tguard(fedd_trainer *t, F &&f) {
    try {
        f();
        return FEDD_OK;
    } catch (const Status &s) {
        if (t) t->err = s.msg;
        return s.code;
    } catch (const CudaError &e) {
        if (t) t->err = std::string(e.what) + ": " + cudaGetErrorString(e.code);
        return FEDD_ERR_CUDA;
    } catch (...) {
        return FEDD_ERR_CUDA;
    }
}

}  // namespace

extern "C" {

fedd_status fedd_trainer_create(int32_t hidden, int64_t n, const float *x, const float *tpsi, const float *tgrad,
                                int device, fedd_trainer **out) {
    if (!out || hidden < 4 || hidden > 512 || n <= 0 || !x || !tpsi || !tgrad) return FEDD_ERR_ARG;
    fedd_trainer *t = new (std::nothrow) fedd_trainer;
    if (!t) return FEDD_ERR_NOMEM;
    fedd_status st = tguard(t, [&] {
        FEDD_CUDA(cudaSetDevice(device));
        t->device = device;
        t->H = hidden;
        t->n = n;
        const int np = t->nparams();
        t->mem.reserve(2 * Arena::bytes<float>(n * 4) + Arena::bytes<float>(n) + 4 * Arena::bytes<float>(np) +
                       Arena::bytes<float>(1));
        auto put = [&](DBuf<float> &b, int64_t count) { b.view(t->mem.take<float>((size_t)count), (size_t)count); };
        put(t->X, n * 4);
        put(t->ty, n);
        put(t->tg, n * 4);
        for (DBuf<float> *b : {&t->par, &t->grad, &t->m1, &t->m2}) put(*b, np);
        put(t->lsum, 1);
        FEDD_CUDA(cudaMemcpyAsync(t->X.p, x, n * 4 * sizeof(float), cudaMemcpyHostToDevice, 0));
        FEDD_CUDA(cudaMemcpyAsync(t->ty.p, tpsi, n * sizeof(float), cudaMemcpyHostToDevice, 0));
        FEDD_CUDA(cudaMemcpyAsync(t->tg.p, tgrad, n * 4 * sizeof(float), cudaMemcpyHostToDevice, 0));
        t->par.zero();
        t->m1.zero();
        t->m2.zero();
        FEDD_CUDA(cudaDeviceSynchronize());
    });
    if (st != FEDD_OK) {
        delete t;
        return st;
    }
    *out = t;
    return FEDD_OK;
}

fedd_status fedd_trainer_set_params(fedd_trainer *t, const float *W1, const float *b1, const float *W2,
                                    const float *b2, const float *w3, float b3) {
    if (!t || !W1 || !b1 || !W2 || !b2 || !w3) return FEDD_ERR_ARG;
    return tguard(t, [&] {
        FEDD_CUDA(cudaSetDevice(t->device));
        const int H = t->H;
        std::vector<float> h(t->nparams());
        std::memcpy(h.data(), W1, 4 * H * sizeof(float));
        std::memcpy(h.data() + 4 * H, b1, H * sizeof(float));
        std::memcpy(h.data() + 5 * H, W2, (size_t)H * H * sizeof(float));
        std::memcpy(h.data() + 5 * H + H * H, b2, H * sizeof(float));
        std::memcpy(h.data() + 6 * H + H * H, w3, H * sizeof(float));
        h[7 * H + H * H] = b3;
        FEDD_CUDA(cudaMemcpy(t->par.p, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
        t->m1.zero();
        t->m2.zero();
        t->step = 0;
        FEDD_CUDA(cudaDeviceSynchronize());
    });
}

fedd_status fedd_trainer_get_params(fedd_trainer *t, float *W1, float *b1, float *W2, float *b2, float *w3, float *b3) {
    if (!t || !W1 || !b1 || !W2 || !b2 || !w3 || !b3) return FEDD_ERR_ARG;
    return tguard(t, [&] {
        FEDD_CUDA(cudaSetDevice(t->device));
        const int H = t->H;
        std::vector<float> h(t->nparams());
        FEDD_CUDA(cudaMemcpy(h.data(), t->par.p, h.size() * sizeof(float), cudaMemcpyDeviceToHost));
        std::memcpy(W1, h.data(), 4 * H * sizeof(float));
        std::memcpy(b1, h.data() + 4 * H, H * sizeof(float));
        std::memcpy(W2, h.data() + 5 * H, (size_t)H * H * sizeof(float));
        std::memcpy(b2, h.data() + 5 * H + H * H, H * sizeof(float));
        std::memcpy(w3, h.data() + 6 * H + H * H, H * sizeof(float));
        *b3 = h[7 * H + H * H];
    });
}

fedd_status fedd_trainer_grad(fedd_trainer *t, float wpsi, float wgrad, float *loss, float *gW1, float *gb1,
                              float *gW2, float *gb2, float *gw3, float *gb3) {
    if (!t || !loss) return FEDD_ERR_ARG;
    return tguard(t, [&] {
        FEDD_CUDA(cudaSetDevice(t->device));
        const int H = t->H;
        if (H == kH) {
            tr_fused(t, nullptr, t->n, wpsi, wgrad, nullptr);
        } else {
            tr_workspace(t, t->n);
            tr_forward_backward(t, nullptr, t->n, wpsi, wgrad);
        }
        float L = 0;
        FEDD_CUDA(cudaMemcpy(&L, t->lsum.p, sizeof L, cudaMemcpyDeviceToHost));
        *loss = L / (float)t->n;
        std::vector<float> g(t->nparams());
        FEDD_CUDA(cudaMemcpy(g.data(), t->grad.p, g.size() * sizeof(float), cudaMemcpyDeviceToHost));
        const float r = 1.0f / (float)t->n;
        for (auto &v : g) v *= r;
        if (gW1) std::memcpy(gW1, g.data(), 4 * H * sizeof(float));
        if (gb1) std::memcpy(gb1, g.data() + 4 * H, H * sizeof(float));
        if (gW2) std::memcpy(gW2, g.data() + 5 * H, (size_t)H * H * sizeof(float));
        if (gb2) std::memcpy(gb2, g.data() + 5 * H + H * H, H * sizeof(float));
        if (gw3) std::memcpy(gw3, g.data() + 6 * H + H * H, H * sizeof(float));
        if (gb3) *gb3 = g[7 * H + H * H];
    });
}

fedd_status fedd_trainer_run(fedd_trainer *t, int32_t steps, int64_t batch, float lr, float wpsi, float wgrad,
                             uint64_t seed, float *last_loss) {
    if (!t || steps < 0 || batch <= 0 || batch > t->n) return FEDD_ERR_ARG;
    return tguard(t, [&] {
        FEDD_CUDA(cudaSetDevice(t->device));
        const int H = t->H;
        if (H != kH) tr_workspace(t, batch);
        if (!t->perm || t->rng != seed) {
            tr_order(t);
            k_iota<<<ceil_div(t->n, 256), 256>>>(t->perm, t->n);
            FEDD_CUDA(cudaGetLastError());
            t->rng = seed;
            t->cursor = t->n;
        }
        for (int it = 0; it < steps; it++) {
            if (t->cursor + batch > t->n) {  // reshuffle (Fisher-Yates, seeded)
                tr_shuffle(t, t->rng ^ (0x5851F42D4C957F2DULL * (uint64_t)(t->step + 1)));
                t->cursor = 0;
            }
            const int64_t *idx = t->perm + t->cursor;
            t->cursor += batch;
            t->step++;
            AdamStep a;
            a.lr = lr;
            a.b1 = 0.9f;
            a.b2 = 0.999f;
            a.eps = 1e-8f;
            // in double: 1 - beta^t in FP32 keeps beta^t's rounding, up to 1.5e-5 of
            // c2 in the early steps, which scales all parameters' moves alike (loss
            // of eight steps of 65,536 samples off by 2.6e-6 on average over 18
            // seeds, 5.6e-7 this way)
            a.c1 = (float)(1.0 - std::pow((double)a.b1, (double)t->step));
            a.c2 = (float)(1.0 - std::pow((double)a.b2, (double)t->step));
            a.scale = 1.0f / (float)batch;
            if (H == kH) {
                tr_fused(t, idx, batch, wpsi, wgrad, &a);
            } else {
                tr_forward_backward(t, idx, batch, wpsi, wgrad);
                const int np = t->nparams();
                k_adam<<<ceil_div(np, 256), 256>>>(t->par.p, t->grad.p, t->m1.p, t->m2.p, np, a.lr, a.b1, a.b2, a.eps,
                                                   a.c1, a.c2, a.scale);
                FEDD_CUDA(cudaGetLastError());
            }
        }
        float L = 0;
        if (steps > 0) FEDD_CUDA(cudaMemcpy(&L, t->lsum.p, sizeof L, cudaMemcpyDeviceToHost));
        L /= (float)batch;
        FEDD_CUDA(cudaDeviceSynchronize());
        if (last_loss) *last_loss = L;
    });
}

fedd_status fedd_trainer_destroy(fedd_trainer *t) {
    if (!t) return FEDD_ERR_ARG;
    cudaSetDevice(t->device);
    delete t;
    return FEDD_OK;
}

}  // extern "C"
