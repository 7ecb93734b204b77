// k_ns.cu -- P2-P1 Taylor-Hood Navier-Stokes Jacobian + residual.
//
// Element math of AssembleFENavierStokes
// (feddlib/core/AceFemAssembly/specific/AssembleFENavierStokes_def.hpp):
//   A  (Laplacian, :149-196), N (advection, :227-298),
//   W  (Newton term, :301-369), B / B^T (divergence, :373-461),
//   J = nu rho A - B - B^T + rho N (+ rho W for Newton)      :66-112
//   r = (nu rho A - B - B^T + rho N) x  (coeff = 1)          :199-224
// For affine elements each term is a contraction of a few per-element
// coefficients with reference integrals (tables.cpp):
//   A_ab  = sum_s Gs_s KS[a][b][s],           Gs = |det B| B^-1 B^-T
//   N_ab  = sum_{c,k} uT[c][k] T[c][a][b][k], uT = |det B| B^-1 u_k
//   W_(ai)(bj) = sum_m g[j][m][i] R[a][b][m],  g = |det B| grad u at vertex m
//   Bd_p(bd) = sum_c Bs[d][c] Y[b][p][c],     Bs = |det B| B^-1
// A record kernel (one thread per element) writes these
// coefficients; the row kernels (a warp per node or two) contract them for the
// node's row and accumulate in shared memory, then write each CSR value once.
#include <type_traits>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace fedd {
namespace {

// record layout (floats, 16-byte aligned groups)
// [0, kRecVel) holds everything the velocity rows read besides NA, so one
// 336-byte bulk copy stages it
constexpr int kRecG = 0;     // g[j][12] = (m*3 + i)
constexpr int kRecBS = 36;   // Bs[d][4] (c < 3)
constexpr int kRecU = 48;    // u[30] node-wise
constexpr int kRecP = 78;    // p[4]
constexpr int kRecVel = 84;
constexpr int kRecUT = 84;   // uT[c][12] = |det B| (B^-1 u_k)_c   (k < 10)
constexpr int kRecGS = 120;  // Gs[6]
constexpr int kRecNA = 128;  // NA[a][b] = nu rho A_ab + rho N_ab (100 floats)
static_assert(kNSRecord == kRecNA + 100, "record size");
// the residual alone reads Bs, p, u and NA, in 16-byte words: Bs[d][4] | p[4] |
// u[30], two unused | NA in rows of 12
constexpr int kResRecP = 12, kResRecU = 16, kResRecNA = 48;
static_assert(kNSResRecord == kResRecNA + 120, "residual record layout");

// device table layout (floats)
// T is stored per row node a and chunk of four k as [a][kc][lane][4] with
// lane = 3 b + c (30 of 32 used), so that the warp's 16-byte reads of one
// chunk cover 512 contiguous bytes (no bank conflicts).
constexpr int kTabT = 0;        // T[a][kc][lane][4]  3840
constexpr int kTabKS = 3840;    // KS[a][b][6]        600
constexpr int kTabR = 4440;     // R[a][b][4]         400
constexpr int kTabY = 4840;     // Y[b][p][4] (c < 3) 160
constexpr int kTabB = 5000;     // T and KS as the B operand of the NA product, in na_off's word order: 4480
static_assert(kTabY + 160 == kTabB && kTabB + 4480 == kNSTab, "table size");
constexpr int kVelTab = 560;    // floats of tables the velocity-row kernel keeps in shared memory (R, Y)

// reference P2 gradients at the vertices, d_c phi_k at vertex m: with the
// barycentric gradients L, (4 [k = m] - 1) L_k for the vertex functions and
// 4 ([a = m] L_b + [b = m] L_a) for the function of edge (a, b)
__constant__ float c_dv[4][10][3] = {
    {{-3, -3, -3}, {-1, 0, 0}, {0, -1, 0}, {0, 0, -1}, {4, 0, 0}, {0, 0, 0}, {0, 4, 0}, {0, 0, 4}, {0, 0, 0}, {0, 0, 0}},
    {{1, 1, 1}, {3, 0, 0}, {0, -1, 0}, {0, 0, -1}, {-4, -4, -4}, {0, 4, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 4}, {0, 0, 0}},
    {{1, 1, 1}, {-1, 0, 0}, {0, 3, 0}, {0, 0, -1}, {0, 0, 0}, {4, 0, 0}, {-4, -4, -4}, {0, 0, 0}, {0, 0, 0}, {0, 0, 4}},
    {{1, 1, 1}, {-1, 0, 0}, {0, -1, 0}, {0, 0, 3}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {-4, -4, -4}, {4, 0, 0}, {0, 4, 0}}};


// ---- the record stage: coefficients, and NA on the fifth-generation tensor cores
// NA_e[n] = sum_kk X_e[kk] Y[kk][n], n = 10 a + b, with
//   X_e = (uT[c][k] at kk = 10 c + k for c < 3, k < 10; Gs[s] at kk = 30 + s)
//   Y   = (rho T[c][a][b][k]; nu rho KS[a][b][s])
// is a GEMM of (elements x 36) by (36 x 100), K padded to 40 and N to 112.
// One kernel computes each element's record (one thread per element) and, for every tile of 128 elements (M = 128, element i of the
// tile in TMEM lane i), that tile's NA: the threads split X into TF32 hi +
// lo parts and write them to shared memory as K-major operands, one thread
// issues tcgen05.mma kind::tf32 for hi hi + hi lo + lo hi (5 K steps of 8,
// FP32 accumulation in TMEM: about FP32 accuracy) and commits to an
// mbarrier, and each warp reads its 32 rows of NA back from TMEM.  A CTA
// (one per SM, persistent) runs four independent groups of 128 threads,
// each with its own tiles, A region, mbarrier, named barrier and 128 TMEM
// columns; the groups share one copy of Y's hi and lo parts, built once.
constexpr int kNAK = 40;                     // K: 36 coefficients padded to 5 steps of 8
constexpr int kNAN = 112;                    // N: 100 (a, b) pairs padded to a multiple of 16
constexpr int kRecTile = 128;                // M: elements per tile = threads per group
constexpr int kRecGroups = 4;                // groups per CTA
constexpr int kRecThreads = kRecGroups * kRecTile;
constexpr int kNAStepA = kRecTile * 32;      // bytes of one K step (8 TF32) of the A operand
constexpr int kNAStepB = kNAN * 32;          // ... of the B operand
constexpr int kNABytesA = 5 * kNAStepA;      // 20,480 per part
constexpr int kNABytesB = 5 * kNAStepB;      // 17,920 per part
constexpr int kRecWarpBytes = 2 * kNABytesA / 4;  // each warp's share of its group's A region between the MMAs
// Shared memory: B (hi, lo), then each group's A region (hi, lo), which
// between the MMAs holds its warps' record and NA staging, then the groups'
// mbarriers and the TMEM address: 199,728 bytes, one CTA (16 warps) per SM.
constexpr int kRecAOff = 2 * kNABytesB;
constexpr int kRecBarOff = kRecAOff + kRecGroups * 2 * kNABytesA;
constexpr size_t kRecSmem = (size_t)kRecBarOff + 8 * kRecGroups + 16;
constexpr uint32_t kNAWaitPolls = 1u << 20;  // bounded wait for the MMAs (each poll sleeps ~32 ns)
static_assert(kRecGS == kRecUT + 36 && kRecNA == kRecGS + 8, "uT, Gs and NA are laid out back to back");
static_assert(kRecWarpBytes >= 32 * 17 * 16 && kRecWarpBytes >= 32 * 68 * 4 && kRecWarpBytes >= 32 * 65 * 4,
              "per-warp staging fits");
static_assert(kRecSmem <= 227 * 1024 && kRecGroups * 128 <= 512, "one CTA per SM: shared memory and TMEM");

// byte offset of (row, k) in a K-major, unswizzled operand: 8-row x 16-byte
// core matrices, the two of one K step 128 B apart (LBO), row groups 256 B
// apart (SBO), K steps `step` bytes apart
__host__ __device__ __forceinline__ int na_off(int row, int k, int step) {
    return (k >> 3) * step + (row >> 3) * 256 + ((k >> 2) & 1) * 128 + (row & 7) * 16 + (k & 3) * 4;
}

// barrier over the 128 threads of group g (named barrier 1 + g)
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory"); }
// ... which also returns whether any of them passed v != 0
__device__ __forceinline__ bool group_sync_or(int g, bool v) {
    uint32_t r;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, %2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r)
                 : "r"((uint32_t)v), "r"(1 + g)
                 : "memory");
    return r != 0;
}

// The warp's 32 rows of NA (100 columns from TMEM) into the residual records:
// row a of 10 values at 12 a.  Two halves of 50 columns (five rows a) through
// the warp's staging in padded form (rows of 64 floats, 60 used, as 15 words),
// then contiguous runs of 240 bytes.
__device__ __forceinline__ void na_rows_padded(float *sN, uint32_t trow, int lane, float *dst, int64_t ew0, int64_t e_end) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
            // columns 48 h + 16 ch ...: of these [50 h, 50 h + 50) are wanted
            float v[16];
            tc::tmem_ld16(trow + 48 * h + 16 * ch, v);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int c = 48 * h + 16 * ch + i - 50 * h;  // column within the half
                if (c >= 0 && c < 50) sN[lane * 65 + 12 * (c / 10) + c % 10] = v[i];
            }
        }
#pragma unroll
        for (int a = 0; a < 5; a++) sN[lane * 65 + 12 * a + 10] = sN[lane * 65 + 12 * a + 11] = 0.0f;
        __syncwarp();
#pragma unroll 4
        for (int k = lane; k < 32 * 15; k += 32) {
            const int rr = k / 15, c = k - 15 * rr;
            const float *s = sN + rr * 65 + 4 * c;
            if (ew0 + rr < e_end)
                reinterpret_cast<float4 *>(dst + (ew0 + rr) * kNSResRecord + 60 * h)[c] = make_float4(s[0], s[1], s[2], s[3]);
        }
        __syncwarp();
    }
}

// elements [e_begin, e_end); RES: the residual's record
template <bool RES>
__global__ void __launch_bounds__(kRecThreads, 1) k_ns_record(const float *__restrict__ geo, const int32_t *__restrict__ conn2,
                                                             const int32_t *__restrict__ conn1, int64_t ne,
                                                             const double *__restrict__ u, const double *__restrict__ p,
                                                             float *rec, int *err, int64_t e_begin, int64_t e_end,
                                                             const float *__restrict__ gtab, float visc_dens, float dens) {
    extern __shared__ __align__(1024) uint8_t rs[];
    const int tid = threadIdx.x, gi = tid >> 7, gt = tid & (kRecTile - 1), wl = (tid >> 5) & 3, lane = tid & 31;
    uint8_t *sBh = rs, *sBl = rs + kNABytesB;
    uint8_t *sAh = rs + kRecAOff + gi * 2 * kNABytesA, *sAl = sAh + kNABytesA;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(rs + kRecBarOff) + gi;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(rs + kRecBarOff + 8 * kRecGroups);
    uint8_t *sW = sAh + wl * kRecWarpBytes;  // this warp's staging, between the MMAs
    // B = Y^T: row n, column kk; the table holds T and KS in the operand's word
    // order (na_off), zero padded
#pragma unroll 3
    for (int t = tid; t < kNAN * kNAK; t += kRecThreads) {
        const int r = t % (kNAN * 8), kk = t / (kNAN * 8) * 8 + ((r >> 5) & 1) * 4 + (r & 3);
        const float y = (kk < 30 ? dens : visc_dens) * gtab[kTabB + t];
        const uint32_t h = to_tf32(y);
        reinterpret_cast<uint32_t *>(sBh)[t] = h;
        reinterpret_cast<uint32_t *>(sBl)[t] = to_tf32(y - __uint_as_float(h));
    }
    if (tid < 32) tc::tmem_alloc(tslot, 128 * kRecGroups);
    if (gt == 0) tc::mbar_init(mbar, 1);
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot + 128u * gi;                  // this group's 128 columns
    const uint32_t trow = tmem + ((uint32_t)(32 * wl) << 16);  // this warp's 32 TMEM lanes
    constexpr uint32_t idesc = tc::idesc_tf32(kRecTile, kNAN);
    const int64_t ntiles = (e_end - e_begin + kRecTile - 1) / kRecTile;
    uint32_t phase = 0;
    bool ok = true;
    // tiles go to the CTAs first and to their groups then, so that few tiles
    // spread over as many SMs
    for (int64_t tile = blockIdx.x + (int64_t)gridDim.x * gi; tile < ntiles; tile += (int64_t)gridDim.x * kRecGroups) {
        // every thread stays for the collective steps; threads past the range
        // recompute the last element and store nothing
        const int64_t e_lane = e_begin + tile * kRecTile + gt;
        const int64_t e = e_lane < e_end ? e_lane : e_end - 1;
        float Bi[9];
        const float det = load_geometry(geo, ne, e, Bi);
        if (!(det > 0.0f) && !(det < 0.0f)) set_dev_error(err, kDevBadDet);
        const float ad = fabsf(det);
        float ue[30];
#pragma unroll
        for (int k = 0; k < 10; k++) {
            const int32_t node = conn2[(int64_t)k * ne + e];
            const double *up = u + 3 * (int64_t)node;
            ue[3 * k] = d2f_rn(up[0]);
            ue[3 * k + 1] = d2f_rn(up[1]);
            ue[3 * k + 2] = d2f_rn(up[2]);
        }
        float R[kRecNA];
#pragma unroll
        for (int k = 0; k < kRecNA; k++) R[k] = 0.0f;
        // uT[c][k] = |det| sum_d Binv[c][d] u_{k,d}
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int k = 0; k < 10; k++)
                R[kRecUT + 12 * c + k] = ad * (Bi[3 * c] * ue[3 * k] + Bi[3 * c + 1] * ue[3 * k + 1] + Bi[3 * c + 2] * ue[3 * k + 2]);
        // g[j][m][i] = |det| sum_c Binv[c][j] sum_k u_{k,i} dphi_ref_c(phi_k)(v_m)
#pragma unroll
        for (int m = 0; m < 4; m++) {
            float Hm[3][3];
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    float h = 0.0f;
#pragma unroll
                    for (int k = 0; k < 10; k++) h = fmaf(ue[3 * k + i], c_dv[m][k][c], h);
                    Hm[i][c] = h;
                }
#pragma unroll
            for (int j = 0; j < 3; j++)
#pragma unroll
                for (int i = 0; i < 3; i++)
                    R[kRecG + 12 * j + 3 * m + i] = ad * (Bi[j] * Hm[i][0] + Bi[3 + j] * Hm[i][1] + Bi[6 + j] * Hm[i][2]);
        }
        // Gs = |det| B^-1 B^-T (00,11,22,01,02,12)
        const int SC[6] = {0, 1, 2, 0, 0, 1}, SD[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
        for (int s = 0; s < 6; s++)
            R[kRecGS + s] = ad * (Bi[3 * SC[s]] * Bi[3 * SD[s]] + Bi[3 * SC[s] + 1] * Bi[3 * SD[s] + 1] +
                                  Bi[3 * SC[s] + 2] * Bi[3 * SD[s] + 2]);
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
            for (int c = 0; c < 3; c++) R[kRecBS + 4 * d + c] = ad * Bi[3 * c + d];
#pragma unroll
        for (int k = 0; k < 30; k++) R[kRecU + k] = ue[k];
#pragma unroll
        for (int k = 0; k < 4; k++) R[kRecP + k] = p ? d2f_rn(p[conn1[(int64_t)k * ne + e]]) : 0.0f;
        // the warp's 32 records (floats [0, kRecNA)) go out through shared
        // memory in two halves of 64 floats, so that each store instruction
        // writes two records' halves as contiguous 256-byte runs; rows of 17
        // chunks keep the 16-byte shared stores conflict-free
        float4 *sRec = reinterpret_cast<float4 *>(sW);
        const int64_t ew0 = e_lane - lane;
        if (RES) {  // twelve chunks per record, rows of 13
            float4 *mine = sRec + lane * 13;
#pragma unroll
            for (int k = 0; k < 3; k++)
                mine[k] = make_float4(R[kRecBS + 4 * k], R[kRecBS + 4 * k + 1], R[kRecBS + 4 * k + 2], 0.0f);
            mine[3] = make_float4(R[kRecP], R[kRecP + 1], R[kRecP + 2], R[kRecP + 3]);
#pragma unroll
            for (int k = 0; k < 8; k++)
                mine[4 + k] = make_float4(R[kRecU + 4 * k], R[kRecU + 4 * k + 1], k < 7 ? R[kRecU + 4 * k + 2] : 0.0f,
                                          k < 7 ? R[kRecU + 4 * k + 3] : 0.0f);
            __syncwarp();
#pragma unroll 4
            for (int k = lane; k < 32 * 12; k += 32) {
                const int rr = k / 12, c = k - 12 * rr;
                if (ew0 + rr < e_end) reinterpret_cast<float4 *>(rec + (ew0 + rr) * kNSResRecord)[c] = sRec[rr * 13 + c];
            }
            __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < (RES ? 0 : 2); h++) {
#pragma unroll
            for (int k = 0; k < 16; k++)
                sRec[lane * 17 + k] = make_float4(R[64 * h + 4 * k], R[64 * h + 4 * k + 1], R[64 * h + 4 * k + 2],
                                                  R[64 * h + 4 * k + 3]);
            __syncwarp();
#pragma unroll 4
            for (int r = 0; r < 32; r += 2) {
                const int rr = r + (lane >> 4);
                const int64_t er = ew0 + rr;
                if (er < e_end) reinterpret_cast<float4 *>(rec + er * kNSRecord)[16 * h + (lane & 15)] = sRec[rr * 17 + (lane & 15)];
            }
            __syncwarp();
        }
        group_sync(gi);  // every warp's staging is done before the A operand overwrites it
#pragma unroll
        for (int q = 0; q < kNAK / 4; q++) {
            uint32_t hv[4], lv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int kk = 4 * q + i;
                const float v = kk < 30 ? R[kRecUT + 12 * (kk / 10) + kk % 10] : (kk < 36 ? R[kRecGS + kk - 30] : 0.0f);
                hv[i] = to_tf32(v);
                lv[i] = to_tf32(v - __uint_as_float(hv[i]));
            }
            const int o = na_off(gt, 4 * q, kNAStepA);
            *reinterpret_cast<uint4 *>(sAh + o) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
            *reinterpret_cast<uint4 *>(sAl + o) = make_uint4(lv[0], lv[1], lv[2], lv[3]);
        }
        tc::fence_proxy_async();
        group_sync(gi);
        if (gt == 0) {
            tc::fence_after_sync();
            const uint32_t aH = tc::smem_u32(sAh), aL = tc::smem_u32(sAl), bH = tc::smem_u32(sBh), bL = tc::smem_u32(sBl);
#pragma unroll
            for (int ks = 0; ks < 5; ks++) {
                const uint64_t ah = tc::smem_desc(aH + ks * kNAStepA, 128, 256), al = tc::smem_desc(aL + ks * kNAStepA, 128, 256);
                const uint64_t bh = tc::smem_desc(bH + ks * kNAStepB, 128, 256), bl = tc::smem_desc(bL + ks * kNAStepB, 128, 256);
                tc::mma_tf32(tmem, ah, bh, idesc, ks > 0);
                tc::mma_tf32(tmem, ah, bl, idesc, 1);
                tc::mma_tf32(tmem, al, bh, idesc, 1);
            }
            tc::commit(mbar);
        }
        const bool done = tc::mbar_wait(mbar, phase, kNAWaitPolls);
        phase ^= 1u;
        if (group_sync_or(gi, !done)) {
            ok = false;
            break;
        }
        tc::fence_after_sync();
        if (RES) {
            // NA rows padded to 12 floats: two halves of 50 columns, staging
            // rows of 65 floats
            na_rows_padded(reinterpret_cast<float *>(sW), trow, lane, rec + kResRecNA, ew0, e_end);
        } else {
            // NA rows out through the warp's staging: columns 0-63 (rows of 68
            // floats), then 64-99 (rows of 36); each store instruction writes
            // whole 256-byte (two rows) or 144-byte (three rows) runs of records
            float *sN = reinterpret_cast<float *>(sW);
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {
                float v[16];
                tc::tmem_ld16(trow + 16 * ch, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    *reinterpret_cast<float4 *>(sN + lane * 68 + 16 * ch + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            }
            __syncwarp();
#pragma unroll 4
            for (int r = 0; r < 32; r += 2) {
                const int rr = r + (lane >> 4);
                const int64_t er = ew0 + rr;
                if (er < e_end)
                    reinterpret_cast<float4 *>(rec + er * kNSRecord + kRecNA)[lane & 15] =
                        *reinterpret_cast<const float4 *>(sN + rr * 68 + 4 * (lane & 15));
            }
            __syncwarp();
#pragma unroll
            for (int ch = 4; ch < 7; ch++) {
                float v[16];
                tc::tmem_ld16(trow + 16 * ch, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    if (16 * ch + i < 100)
                        *reinterpret_cast<float4 *>(sN + lane * 36 + 16 * (ch - 4) + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            }
            __syncwarp();
            for (int r = 0; r < 32; r += 3) {
                const int rr = r + lane / 9, c4 = lane % 9;
                const int64_t er = ew0 + rr;
                if (lane < 27 && rr < 32 && er < e_end)
                    reinterpret_cast<float4 *>(rec + er * kNSRecord + kRecNA + 64)[c4] =
                        *reinterpret_cast<const float4 *>(sN + rr * 36 + 4 * c4);
            }
        }
        tc::fence_before_sync();
        group_sync(gi);
    }
    if (!ok) {
        // the MMAs did not complete in time: report it, give them a second
        // bounded wait, then free the tensor memory all the same
        if (gt == 0) set_dev_error(err, kDevTimeout);
        tc::mbar_wait(mbar, phase ^ 1u, kNAWaitPolls);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid < 32) tc::tmem_dealloc(*tslot, 128 * kRecGroups);
}

__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Lane (b, j) of one incidence with row node a: returns its share of
// (nu rho A_ab + rho N_ab) (the three lanes of b hold the c = j parts) and
// fills w[i] = W_(ai)(bj).
__device__ __forceinline__ float ns_lane_terms(const float *rec, const float *tab, int a, int b, int j,
                                               float visc_dens, float dens, float w[3]) {
    const float *T = tab + kTabT + (a * 96 + 3 * b + j) * 4;
    const float *U = rec + kRecUT + 12 * j;
    const float4 t0 = lds4(T), t1 = lds4(T + 128), t2 = lds4(T + 256);
    const float4 u0 = lds4(U), u1 = lds4(U + 4), u2 = lds4(U + 8);
    const float n = (u0.x * t0.x + u0.y * t0.y + u0.z * t0.z + u0.w * t0.w) +
                    (u1.x * t1.x + u1.y * t1.y + u1.z * t1.z + u1.w * t1.w) + (u2.x * t2.x + u2.y * t2.y);
    const float2 ks = *reinterpret_cast<const float2 *>(tab + kTabKS + (a * 10 + b) * 6 + 2 * j);
    const float2 gs = *reinterpret_cast<const float2 *>(rec + kRecGS + 2 * j);
    const float av = gs.x * ks.x + gs.y * ks.y;
    const float4 r = lds4(tab + kTabR + (a * 10 + b) * 4);
    const float *G = rec + kRecG + 12 * j;
    const float4 g0 = lds4(G), g1 = lds4(G + 4), g2 = lds4(G + 8);
    // g[j][m*3+i]: m0 = (g0.x,g0.y,g0.z) m1 = (g0.w,g1.x,g1.y) m2 = (g1.z,g1.w,g2.x) m3 = (g2.y,g2.z,g2.w)
    w[0] = g0.x * r.x + g0.w * r.y + g1.z * r.z + g2.y * r.w;
    w[1] = g0.y * r.x + g1.x * r.y + g1.w * r.z + g2.z * r.w;
    w[2] = g0.z * r.x + g1.y * r.y + g2.x * r.z + g2.w * r.w;
    return visc_dens * av + dens * n;
}

// -Bd_p(a,i) for B^T lane (i, p): the (0,1) entry of velocity row (a, i)
__device__ __forceinline__ float ns_bt(const float *rec, const float *tab, int a, int i, int p) {
    const float4 bs = lds4(rec + kRecBS + 4 * i);
    const float4 y = lds4(tab + kTabY + (a * 4 + p) * 4);
    return -(bs.x * y.x + bs.y * y.y + bs.z * y.z);
}

__device__ __forceinline__ float sum3_lanes(float part, int lane) {
    const int b = lane / 3, j = lane - 3 * b;
    int s1 = 3 * b + (j + 1) % 3, s2 = 3 * b + (j + 2) % 3;
    if (lane >= 30) { s1 = lane; s2 = lane; }
    float x1 = __shfl_sync(0xffffffffu, part, s1);
    float x2 = __shfl_sync(0xffffffffu, part, s2);
    return part + x1 + x2;
}

// Per velocity-row node, one 16-byte word: the first incidence (int64, x | y),
// the P1 node at the vertex (z, -1 for edge nodes or without a verified
// vertex map) and w = K | Kp << 8 | m << 16 (velocity and pressure
// neighbours, at most kMaxAdjacency = 255 each; incidences, at most 64).
__device__ __forceinline__ int64_t node_i0(int4 v) {
    return (int64_t)(((uint64_t)(uint32_t)v.y << 32) | (uint32_t)v.x);
}
__device__ __forceinline__ int node_k(int4 v) { return v.w & 255; }
__device__ __forceinline__ int node_kp(int4 v) { return (v.w >> 8) & 255; }
__device__ __forceinline__ int node_m(int4 v) { return (v.w >> 16) & 255; }

__global__ void k_ns_node_info(const int64_t *__restrict__ inc_ptr, const int64_t *__restrict__ adj_ptr,
                               const int64_t *__restrict__ padj_ptr, const int32_t *__restrict__ vmap, int64_t nn,
                               int4 *info) {
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int64_t i0 = inc_ptr[n];
    const int m = (int)(inc_ptr[n + 1] - i0);
    const int K = (int)(adj_ptr[n + 1] - adj_ptr[n]), Kp = (int)(padj_ptr[n + 1] - padj_ptr[n]);
    info[n] = make_int4((int)(uint32_t)(uint64_t)i0, (int)(uint32_t)((uint64_t)i0 >> 32), vmap ? vmap[n] : -1,
                        K | (Kp << 8) | (m << 16));
}

// velocity rows: block (0,0) and (0,1) values and the velocity residual, and
// at the vertices of a mesh with a verified vertex map the pressure row too.
// A warp works on two row nodes at a time (NPW = 2), one per half warp, an
// incidence of each per step: with lanes (p, j) of 15 the half's lane owns the columns
// (b, j) of the two nodes b = 2 p and 2 p + 1, so every value that the ten
// nodes share (the gradient rows g[j], Bs, the wait, the staging) is read or
// done once for two incidences.  Warps claim four or eight consecutive nodes and pair
// them by their number of incidences, so that the halves end together (on a
// lattice vertices, 24 incidences, and edge nodes, 4 or 6, alternate).
// Each incidence's record head (g, Bs, u, p), the 48-byte window holding
// NA[a][:] and its slot map (25 chunks of 16 bytes) are copied by cp.async
// into the half's ring of kVRing shared-memory slots, kVRing - 1 incidences
// ahead.  Each half accumulates in three runs in the order of the CSR
// values: the 9 K velocity values, the 3 Kp of block (0,1) and the 3 K of the
// pressure row, so the write-out is a linear copy, pairs of values as 16-byte
// stores; each run is shifted by one word when its values start at an odd
// multiple of 8 bytes.  Lanes without work update a scratch word.
// With a generalized-Newtonian viscous stage (the dense element matrix with
// rows padded to 32 floats, kGNStride floats per element) each slot also
// holds the element's three rows 3 a + i and an 8-float window holding its
// residual entries 3 a .. 3 a + 2 (26 more chunks), which the lanes fold into
// the same accumulation: no separate pass re-reads and re-writes the rows.
// Bound by the shared-memory pipe (about 53 wavefronts per incidence, most of
// them the accumulators' scattered updates and the broadcast 16-byte reads).
// At 48^3 x 6 tets 1,299 us, against 1,480 us with one node per warp, three
// planes of accumulators and 8-byte stores; without the Newton term, whose
// reads and products the Picard form leaves out, 197 us against 240 at
// 27 x 19 x 33 x 6 tets in file order, 189 without staging the gradients and 183
// without the residual (RES), its sums and the chunks of u and p; the Newton
// form without the residual at 51 x 37 x 39 x 6 886 us for the call against 977; with the viscous rows 494 us against 522
// at 32^3 x 6.  Groups of four nodes 1,319 us, rings of three or six slots
// 1,389 and 1,423, eleven warps per CTA (80 registers, spills) 1,461.
constexpr int kVRing = 4;
constexpr int kVStage = 100;  // floats per ring slot: record head 84 | NA window 12 | slot map 16 B
constexpr int kVNA = kRecVel, kVSlots = kRecVel + 12;
constexpr int kVGn = kVStage, kVGnRes = kVStage + 96, kVStageGn = kVStage + 104;
static_assert(kVSlots + 4 == kVStage && kRecVel % 4 == 0, "ring slot layout: chunk c holds floats [4 c, 4 c + 4)");
static_assert(kRecG == 0 && kRecBS == 36 && kRecBS < kRecU && kRecBS < kRecP && kRecVel == 84,
              "without the gradients at its front the head has twelve chunks");
// the ring and the accumulators of a half are 16 mod 32 words, so the halves'
// accesses to the same place of theirs differ in banks
static_assert(kVRing * kVStage % 32 == 16 && kVRing * kVStageGn % 32 == 16, "half-warp bank offset");
// Small meshes take one node per warp (NPW = 1: lane (b, j) of 30 owns one
// column): a warp then has a node or a few, the time is that of the longest
// chain of steps, and a step of 30 lanes with a column each is shorter than one
// of 15 with two (2,197 nodes 20.4 us against 22.9, 9,261 nodes 34 against
// 38 us; from 24,000 nodes on the pairs are faster, 57 us against 61).
// warps per CTA at most, two CTAs per SM (shared memory: about 10.3 KB per pair
// of nodes on the structured meshes, 13.6 with the viscous rows)
__host__ __device__ constexpr int vel_warps(bool gn, int npw) { return npw == 1 ? 12 : gn ? 8 : 10; }

// words of one node's accumulators: the three runs, each with its shift and
// padding to 16 bytes, 32 words of the pressure residual's sum, the scratch word
__host__ __device__ __forceinline__ int vel_run_words(int len) { return (len + 1 + 3) & ~3; }
__host__ __device__ __forceinline__ int vel_acc_words(int max_adj, int max_padj, bool pres) {
    const int w = vel_run_words(9 * max_adj) + vel_run_words(3 * max_padj) + (pres ? vel_run_words(3 * max_adj) : 0) + 36;
    return (w + 31) & ~31;
}

// len values of a run (mem + shift) out as FP64 by W lanes
template <int W>
__device__ __forceinline__ void vel_write(const float *mem, int shift, int len, double *out, int hl) {
    if (shift && len > 0 && hl == W - 1) st_cs(out, f2d_exact(mem[1]));
    const int pairs = len > 0 ? (len - shift) >> 1 : 0;
    for (int c = hl; c < pairs; c += W) {
        const float2 x = *reinterpret_cast<const float2 *>(mem + 2 * shift + 2 * c);
        __stcs(reinterpret_cast<double2 *>(out + shift) + c, make_double2(f2d_exact(x.x), f2d_exact(x.y)));
    }
    if (len > 0 && ((len - shift) & 1) && hl == W - 2) st_cs(out + len - 1, f2d_exact(mem[shift + len - 1]));
}
__device__ __forceinline__ int odd8(const void *p) { return (int)((reinterpret_cast<uintptr_t>(p) >> 3) & 1); }

// velocity residual of the node n of W lanes: row (a, i) sums rj over the lanes
// (p, i), the nodes b = 2 p and 2 p + 1 with 16 lanes, b = p with 32, and rb
// over the lanes 4 i + q by strided trees
// (in b: (((0+1)+(2+3))+((4+5)+(6+7)))+(8+9)); rg, in lane i, is the viscous
// residual of a generalized-Newtonian fluid.
// uu (N(u) u + viscous) + up (-B^T p), with the residual's block factors
template <bool GN, int W>
__device__ __forceinline__ void vel_residual_out(float rj0, float rj1, float rb, float rg, int64_t n, int hl, bool node,
                                                 const NSCoeff &co, double *res_u) {
    float x = W == 16 ? rj0 + rj1 : rj0 + __shfl_down_sync(0xffffffffu, rj0, 3);
    constexpr int D = W == 16 ? 3 : 6;  // lanes from one pair of nodes b to the next
    if (hl >= 30 * W / 32) x = 0.0f;
    float z = hl < 12 ? rb : 0.0f;
    const float x2 = x + __shfl_down_sync(0xffffffffu, x, D, W);
    const float x4 = x2 + __shfl_down_sync(0xffffffffu, x2, 2 * D, W);
    const float xs = x4 + __shfl_down_sync(0xffffffffu, x, 4 * D, W);
    z += __shfl_down_sync(0xffffffffu, z, 1, W);
    z += __shfl_down_sync(0xffffffffu, z, 2, W);
    z = __shfl_sync(0xffffffffu, z, hl < 3 ? 4 * hl : 0, W);
    const float cuu = (float)co.uu, s = fmaf(cuu, xs, (float)co.up * z);
    if (node && hl < 3) res_u[3 * n + hl] = f2d_exact(GN ? fmaf(cuu, rg, s) : s);
}

template <bool GN, bool NEWTON, int NPW, bool RES>
__global__ void __launch_bounds__(32 * vel_warps(GN, NPW), 2)
    k_ns_vel_rows(const int4 *__restrict__ ninfo, const uint32_t *__restrict__ inc, const uint8_t *__restrict__ slots,
                  const float *__restrict__ rec, const float *__restrict__ gtab, const int64_t *__restrict__ rowptr00,
                  const int64_t *__restrict__ rowptr01, double *vals00, double *vals01, double *res_u, int64_t nnodes,
                  float dens, int group, int acc_words, int64_t n_begin, const int64_t *__restrict__ rowptr10,
                  double *vals10, double *res_p, const float *__restrict__ gstage, unsigned long long *work, NSCoeff co) {
    constexpr int kStg = GN ? kVStageGn : kVStage;
    constexpr int W = 32 / NPW;  // lanes per node, each with the columns of NPW nodes b
    extern __shared__ __align__(16) float smem[];
    // the W table scaled by the Newton weight rho and the B^T table negated:
    // sR = rho R[a][b][4], sY = -Y[a][p][4]; the diagonal part NA comes with
    // each record (and is all of the Picard form)
    float *sR = smem, *sY = smem + 400;
    static_assert(kTabY == kTabR + 400 && kVelTab == 560, "R and Y are adjacent");
    for (int t = threadIdx.x; t < kVelTab; t += blockDim.x) smem[t] = t < 400 ? dens * gtab[kTabR + t] : -gtab[kTabR + t];
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = lane / W, hl = lane % W, nw = blockDim.x >> 5;
    float *ring = smem + kVelTab + (size_t)(NPW * w + h) * (kVRing * kStg + acc_words);
    float *mem = ring + kVRing * kStg;
    float *sum32 = mem + acc_words - 36, *scratch = mem + acc_words - 4;
    // lane roles: (p, j) of the NA / W part for hl < 30 / NPW, (i, q) = (bi, bq) of the B^T part for hl < 12
    const bool lw = hl < 30 / NPW, lb = hl < 12;
    const int p = lw ? hl / 3 : 0, j = lw ? hl - 3 * (hl / 3) : 0;
    const int bi = hl >> 2, bq = hl & 3;
    const float e0 = j == 0 ? 1.0f : 0.0f, e1 = j == 1 ? 1.0f : 0.0f, e2 = j == 2 ? 1.0f : 0.0f;
    // lane-constant addresses in ring slot 0 and in the tables
    const float *pG = ring + kRecG + 12 * j;
    const float *pU = ring + kRecU + 3 * NPW * p + j;
    const float *pNA = ring + kVNA + NPW * p;
    const float *pBS = ring + kRecBS + 4 * (lb ? bi : 0);
    const float *pBSj = ring + kRecBS + 4 * j;
    const float *pP = ring + kRecP + bq;
    const uint8_t *pS = reinterpret_cast<const uint8_t *>(ring + kVSlots);
    const float *pR = sR + 4 * NPW * p, *pY = sY + 4 * bq, *pYb = sY + 16 * NPW * p;
    // chunks of 16 bytes: record head (to 20), NA window (21-23), slot map (24).  Two nodes per warp: chunk hl,
    // and c2 = 16 + hl for hl < 9; one: c2 = hl < 25 alone.  Without the Newton term the head's nine chunks of
    // velocity gradients stay behind, without the residual its nine of u and p, and c2 for hl < 16 is all
    const int cg = NPW == 2 ? 16 + hl : hl;
    const int c2 = NEWTON && RES ? cg
                   : RES         ? kRecBS / 4 + hl
                   : NEWTON      ? (hl < 12 ? hl : 9 + hl)
                                 : (hl < 3 ? kRecBS / 4 + hl : hl < 7 ? 18 + hl : 25);
    const char *src1 = reinterpret_cast<const char *>(rec + 4 * hl);
    const char *src2 = reinterpret_cast<const char *>(c2 < 21 ? rec + 4 * c2 : rec + kRecNA + 4 * (c2 - 21));
    float *dst_lane = ring + 4 * hl, *dst2 = ring + 4 * c2, *dstg = ring + kVGn + 4 * cg;
    // with `work`, nodes come from a global counter, a group per warp step, so
    // all warps stay on one sharp front of the sweep and the ten readers of
    // an element's record come close in time
    for (int64_t it = n_begin + group * ((int64_t)blockIdx.x * nw + w);; it += group * (int64_t)gridDim.x * nw) {
        if (work) {
            unsigned long long k = 0;
            if (lane == 0) k = atomicAdd(work, (unsigned long long)group);
            it = n_begin + (int64_t)__shfl_sync(0xffffffffu, k, 0);
        }
        if (it >= nnodes) break;
        // lane k < group: node it + k; rank 0 has the most incidences
        const bool member = NPW == 1 || ((lane & 7) < group && it + (lane & 7) < nnodes);
        const int4 inf4 = member ? ninfo[it + (NPW == 1 ? 0 : lane & 7)] : make_int4(0, 0, -1, 0);
        int rank = 0;
        if (NPW == 2) {
            const int m4 = node_m(inf4);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int mk = __shfl_sync(0xffffffffu, m4, k);
                rank += mk > m4 || (mk == m4 && k < (lane & 7));
            }
        }
#pragma unroll 1
        for (int pair = 0; NPW * pair < group; pair++) {
            int k = 0;
            int4 inf = inf4;
            if (NPW == 2) {
                const unsigned f0 = __ballot_sync(0xffffffffu, lane < 8 && rank == 2 * pair);
                const unsigned f1 = __ballot_sync(0xffffffffu, lane < 8 && rank == 2 * pair + 1);
                k = __ffs(h ? f1 : f0) - 1;
                inf.x = __shfl_sync(0xffffffffu, inf4.x, k);
                inf.y = __shfl_sync(0xffffffffu, inf4.y, k);
                inf.z = __shfl_sync(0xffffffffu, inf4.z, k);
                inf.w = __shfl_sync(0xffffffffu, inf4.w, k);
            }
            const int64_t n = it + k;
            const bool node = k < group && n < nnodes;
            const int m = node_m(inf), K = node_k(inf), Kp = node_kp(inf);
            const int qp = inf.z;  // the P1 node at this vertex, whose pressure row this half assembles too
            const int mm = NPW == 2 ? max(m, __shfl_xor_sync(0xffffffffu, m, 16)) : m;
            const int64_t i0 = node_i0(inf);
            const uint32_t *il = inc + i0;
            if (c2 == 24) src2 = reinterpret_cast<const char *>(slots + i0 * kSlotStride);
            // the node's list, a window of W entries at a time
            uint32_t lst = hl < m ? __ldg(il + hl) : 0u, lst_next = W + hl < m ? __ldg(il + W + hl) : 0u;
            // incidence t of the node into its ring slot; every call
            // commits one group, empty past the end, so the wait counts hold
            auto stage = [&](int slot, int t) {
                if (t > 0 && t % W == 0) {  // warp-uniform
                    lst = lst_next;
                    lst_next = t + W + hl < m ? __ldg(il + t + W + hl) : 0u;
                }
                const uint32_t ea = __shfl_sync(0xffffffffu, lst, t % W, W);
                if (t < m) {
                    const uint32_t a = ea & 15u;
                    const size_t eo = (size_t)(ea >> 4) * (kNSRecord * sizeof(float));
                    if (NPW == 2 && NEWTON && RES) cp_async16(dst_lane + slot * kStg, src1 + eo);
                    // NA[a][0..9] starts 8 bytes into a 16-byte boundary when a is odd
                    const size_t o2 = c2 == 24 ? (size_t)(t * kSlotStride) : eo + (c2 < 21 ? 0u : 40u * a - 8u * (a & 1u));
                    if (c2 < 25) cp_async16(dst2 + slot * kStg, src2 + o2);
                    if (GN) {
                        const float *Ke = gstage + (size_t)(ea >> 4) * kGNStride;
                        if (NPW == 2) cp_async16(dst_lane + slot * kStg + kVGn, Ke + 96 * a + 4 * hl);
                        if (cg < (RES ? 26 : 24))
                            cp_async16(dstg + slot * kStg,
                                       cg < 24 ? Ke + 96 * a + 4 * cg : Ke + kGNRes + 4 * ((3 * a) >> 2) + 4 * (cg - 24));
                    }
                }
                cp_async_commit();
            };
#pragma unroll 1
            for (int t = 0; t < kVRing - 1; t++) stage(t, t);
            double *out00 = node ? vals00 + rowptr00[3 * n] : nullptr, *out01 = node ? vals01 + rowptr01[3 * n] : nullptr;
            double *out10 = qp >= 0 ? vals10 + rowptr10[qp] : nullptr;
            const int s00 = odd8(out00), s01 = odd8(out01), s10 = odd8(out10);
            const int o01 = vel_run_words(9 * K), o10 = o01 + vel_run_words(3 * Kp);
            const int used = o10 + (qp >= 0 ? vel_run_words(3 * K) : 0);
            for (int c = 4 * hl; c < used; c += 4 * W) *reinterpret_cast<float4 *>(mem + c) = make_float4(0.f, 0.f, 0.f, 0.f);
            float *acc = mem + s00, *acc1 = mem + o01 + s01, *acc2 = mem + o10 + s10;
            const int st = 3 * K;
            float rj0 = 0.0f, rj1 = 0.0f, rb = 0.0f, rq0 = 0.0f, rq1 = 0.0f, rg = 0.0f;
            // the table rows of the current local index a; incidences come sorted
            // by a, so they reload only when a run of equal a ends
            int a_cur = -1;
            float4 ra = make_float4(0.f, 0.f, 0.f, 0.f), rc = ra, y = ra, ya = ra, yc = ra;
#pragma unroll 1
            for (int t = 0; t < mm; t++) {
                const int r = t & (kVRing - 1);
                cp_async_wait<kVRing - 2>();
                // the slot's copies are visible to the warp, and every lane is
                // done with the slot consumed in the previous step, which is
                // refilled next
                __syncwarp();
                stage((r + kVRing - 1) & (kVRing - 1), t + kVRing - 1);
                if (NPW == 2 && t >= m) continue;  // this half's node is done
                const int off = r * kStg;
                const int a = pS[4 * off + kSlotLocal];  // the staged slot map's local-index byte (broadcast)
                if (a != a_cur) {
                    a_cur = a;
                    if (NEWTON) {
                        ra = lds4(pR + 40 * a);
                        if (NPW == 2) rc = lds4(pR + 40 * a + 4);
                    }
                    y = lds4(pY + 16 * a);
                    if (qp >= 0 && a < 4) {
                        ya = lds4(pYb + 4 * a);
                        if (NPW == 2) yc = lds4(pYb + 16 + 4 * a);
                    }
                }
                // NA_ab on the diagonal (i = j) plus wn W_(ai)(bj), i = 0..2
                float4 g0, g1, g2;
                if (NEWTON) {
                    g0 = lds4(pG + off);
                    g1 = lds4(pG + off + 4);
                    g2 = lds4(pG + off + 8);
                }
                float2 an;
                uint32_t ss;
                if (NPW == 2) {
                    an = *reinterpret_cast<const float2 *>(pNA + off + 2 * (a & 1));
                    ss = *reinterpret_cast<const uint16_t *>(pS + 4 * off + 2 * p);
                } else {
                    an = make_float2(pNA[off + 2 * (a & 1)], 0.0f);
                    ss = pS[4 * off + p];
                }
                float *dA = lw ? acc + 3 * (ss & 255u) + j : scratch, *dB = lw ? acc + 3 * (ss >> 8) + j : scratch;
                const int sl = lw ? st : 0;
                // g[j][m*3+i]: m0 = (g0.x,g0.y,g0.z) m1 = (g0.w,g1.x,g1.y) m2 = (g1.z,g1.w,g2.x) m3 = (g2.y,g2.z,g2.w)
                {
                    float v0 = dA[0], v1 = dA[sl], v2 = dA[2 * sl];
                    // the viscous rows (a, i), columns (b, j), and the viscous residual of row (a, hl)
                    const float *V = ring + off + kVGn + 3 * NPW * p + j;
                    if (GN) {
                        v0 += V[0];
                        v1 += V[32];
                        v2 += V[64];
                        if (RES) rg += ring[off + kVGnRes + ((3 * a) & 3) + (hl & 3)];
                    }
                    v0 = fmaf(e0, an.x, v0);
                    v1 = fmaf(e1, an.x, v1);
                    v2 = fmaf(e2, an.x, v2);
                    if (NEWTON) {
                        v0 = fmaf(g2.y, ra.w, fmaf(g1.z, ra.z, fmaf(g0.w, ra.y, fmaf(g0.x, ra.x, v0))));
                        v1 = fmaf(g2.z, ra.w, fmaf(g1.w, ra.z, fmaf(g1.x, ra.y, fmaf(g0.y, ra.x, v1))));
                        v2 = fmaf(g2.w, ra.w, fmaf(g2.x, ra.z, fmaf(g1.y, ra.y, fmaf(g0.z, ra.x, v2))));
                    }
                    if (NPW == 2) {
                        float w0 = dB[0], w1 = dB[sl], w2 = dB[2 * sl];
                        if (GN) {
                            w0 += V[3];
                            w1 += V[35];
                            w2 += V[67];
                        }
                        w0 = fmaf(e0, an.y, w0);
                        w1 = fmaf(e1, an.y, w1);
                        w2 = fmaf(e2, an.y, w2);
                        if (NEWTON) {
                            w0 = fmaf(g2.y, rc.w, fmaf(g1.z, rc.z, fmaf(g0.w, rc.y, fmaf(g0.x, rc.x, w0))));
                            w1 = fmaf(g2.z, rc.w, fmaf(g1.w, rc.z, fmaf(g1.x, rc.y, fmaf(g0.y, rc.x, w1))));
                            w2 = fmaf(g2.w, rc.w, fmaf(g2.x, rc.z, fmaf(g1.y, rc.y, fmaf(g0.z, rc.x, w2))));
                        }
                        dB[0] = w0;
                        dB[sl] = w1;
                        dB[2 * sl] = w2;
                    }
                    dA[0] = v0;
                    dA[sl] = v1;
                    dA[2 * sl] = v2;
                }
                const float ua = RES ? pU[off] : 0.0f, ub = RES && NPW == 2 ? pU[off + 3] : 0.0f;
                if (RES) {
                    rj0 = fmaf(an.x, ua, rj0);
                    if (NPW == 2) rj1 = fmaf(an.y, ub, rj1);
                }
                // -Bd_q(a, i): the (0,1) entry of velocity row (a, i), pressure column q
                const float4 bs = lds4(pBS + off);
                const float bt = fmaf(bs.z, y.z, fmaf(bs.y, y.y, bs.x * y.x));
                float *dp = lb ? acc1 + bi * Kp + pS[4 * off + 10 + bq] : scratch;
                *dp += bt;
                if (RES) rb = fmaf(bt, pP[off], rb);
                if (qp >= 0 && a < 4) {
                    // -Bd_q(b j): the (1,0) entries of pressure row q = this vertex, columns (b, j)
                    const float4 bj = lds4(pBSj + off);
                    const float pa = fmaf(bj.z, ya.z, fmaf(bj.y, ya.y, bj.x * ya.x));
                    float *qa = lw ? acc2 + 3 * (ss & 255u) + j : scratch;
                    *qa += pa;
                    if (RES) rq0 = fmaf(pa, ua, rq0);
                    if (NPW == 2) {
                        const float pc = fmaf(bj.z, yc.z, fmaf(bj.y, yc.y, bj.x * yc.x));
                        float *qc = lw ? acc2 + 3 * (ss >> 8) + j : scratch;
                        *qc += pc;
                        if (RES) rq1 = fmaf(pc, ub, rq1);
                    }
                }
            }
            cp_async_wait<0>();
            __syncwarp();
            vel_write<W>(mem, s00, 9 * K, out00, hl);
            vel_write<W>(mem + o01, s01, 3 * Kp, out01, hl);
            if (RES && res_u) vel_residual_out<GN, W>(rj0, rj1, rb, rg, n, hl, node, co, res_u);
            if (qp >= 0) vel_write<W>(mem + o10, s10, 3 * K, out10, hl);
            if (RES && res_p && __any_sync(0xffffffffu, qp >= 0)) {
                // the pressure residual: the pairwise (xor) tree over 32 words, (b, j) at 3 b + j
                float v;
                if (NPW == 2) {
                    if (lw) {
                        sum32[6 * p + j] = rq0;
                        sum32[6 * p + 3 + j] = rq1;
                    } else {
                        sum32[30] = sum32[31] = 0.0f;
                    }
                    __syncwarp();
                    v = sum32[hl] + sum32[hl + 16];
                } else {
                    v = lw ? rq0 : 0.0f;
                    v += __shfl_xor_sync(0xffffffffu, v, 16);
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (qp >= 0 && hl == 0) res_p[qp] = f2d_exact((float)co.pu * v);
            }
            __syncwarp();
        }
    }
}

// pressure rows: block (1,0) values and the pressure residual.  One warp per
// pressure node q; per incidence lanes 0-10 copy the record's Bs and u
// (floats [kRecBS, kRecBS + 44)) and lane 11 the slot map into a ring slot
// with one 16-byte cp.async each; lane (b, d) < 30 adds -Bd_q(b d).
constexpr int kPRing = 4;
constexpr int kPStage = 48;  // floats per ring slot: Bs 12 | u 30 | pad 2 | slot map 16 B
constexpr int kPU = kRecU - kRecBS, kPSlots = 44;
static_assert(kRecU == kRecBS + 12 && kRecP <= kRecBS + kPSlots, "Bs and u are adjacent in the record");

__device__ __forceinline__ void stage_pres(float *dst_lane, int slot, int t, int m, const IncList &il,
                                           const float *__restrict__ rec_lane, int lane,
                                           const uint8_t *__restrict__ slots_node) {
    if (t < m) {
        const uint32_t ea = incidence_at(il, t);
        const void *src = lane == kPSlots / 4 ? static_cast<const void *>(slots_node + t * kSlotStride)
                                              : static_cast<const void *>(rec_lane + (size_t)(ea >> 4) * kNSRecord);
        if (lane <= kPSlots / 4) cp_async16(dst_lane + slot * kPStage, src);
    }
    cp_async_commit();
}

__global__ void __launch_bounds__(256) k_ns_pres_rows(const int64_t *__restrict__ inc_ptr, const uint32_t *__restrict__ inc,
                                                      const uint8_t *__restrict__ slots, const int64_t *__restrict__ adj_ptr,
                                                      const float *__restrict__ rec, const float *__restrict__ gtab,
                                                      const int64_t *__restrict__ rowptr10, double *vals10, double *res_p,
                                                      int64_t nnodes, int max_adj, float cpu) {
    extern __shared__ __align__(16) float smem[];
    float *sY = smem;  // -Y[b][q][4]
    for (int t = threadIdx.x; t < 160; t += blockDim.x) sY[t] = -gtab[kTabY + t];
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int acc_words = (3 * max_adj + 1 + 3) & ~3;  // + one scratch word that idle lanes write
    float *ring = smem + 160 + (size_t)w * (kPRing * kPStage + acc_words);
    float *acc = ring + kPRing * kPStage;
    const bool lw = lane < 30;
    const int b = lw ? lane / 3 : 0, d = lw ? lane - 3 * (lane / 3) : 0;
    const float *pBS = ring + 4 * d;
    const float *pU = ring + kPU + 3 * b + d;
    const uint8_t *pS = reinterpret_cast<const uint8_t *>(ring + kPSlots) + b;
    const float *pY = sY + 16 * b;
    float *dst_lane = ring + 4 * lane;
    const float *rec_lane = rec + kRecBS + 4 * lane;
    for (int64_t n = (int64_t)blockIdx.x * nw + w; n < nnodes; n += (int64_t)gridDim.x * nw) {
        const int64_t i0 = inc_ptr[n], i1 = inc_ptr[n + 1];
        const int m = (int)(i1 - i0);
        const IncList il = load_incidences(inc, i0, m, lane);
        const uint8_t *slots_node = slots + i0 * kSlotStride;
#pragma unroll
        for (int t = 0; t < kPRing - 1; t++) stage_pres(dst_lane, t, t, m, il, rec_lane, lane, slots_node);
        const int K = (int)(adj_ptr[n + 1] - adj_ptr[n]);
        for (int c = lane; c < 3 * K; c += 32) acc[c] = 0.0f;
        float r = 0.0f;
        for (int t0 = 0; t0 < m; t0 += kPRing) {
#pragma unroll
            for (int rs = 0; rs < kPRing; rs++) {
                const int t = t0 + rs;
                if (t >= m) break;
                cp_async_wait<kPRing - 2>();
                __syncwarp();
                stage_pres(dst_lane, (rs + kPRing - 1) % kPRing, t + kPRing - 1, m, il, rec_lane, lane, slots_node);
                const int off = rs * kPStage;
                const int q = (int)(incidence_at(il, t) & 15u);
                const float4 bs = lds4(pBS + off);
                const float4 y = lds4(pY + 4 * q);
                const float v = fmaf(bs.z, y.z, fmaf(bs.y, y.y, bs.x * y.x));
                float *dst = acc + (lw ? 3 * pS[4 * off] + d : 3 * max_adj);
                *dst += v;
                r = fmaf(v, pU[off], r);
            }
        }
        cp_async_wait<0>();
        __syncwarp();
        double *out = vals10 + rowptr10[n];
        for (int c = lane; c < 3 * K; c += 32) st_cs(out + c, f2d_exact(acc[c]));
        if (res_p) {
            float v = warp_sum(lw ? r : 0.0f);
            if (lane == 0) res_p[n] = f2d_exact(cpu * v);
        }
        __syncwarp();
    }
}

// ---- the residual alone -------------------------------------------------
// One thread per node with the sums of k_ns_vel_rows' lanes in registers, each
// in that kernel's order, and the lanes' tree sums at the end: the values are
// those of the call that assembles both.  Per incidence a thread reads 240
// bytes of the element's record as 16-byte words, and these scattered reads
// bound it (l1tex 89 % of its peak).  At 40^3 x 6 tets it takes 220 us and the
// smaller records 102, against 741 and 122 us of the matrix stages.  One warp
// per node with a lane per sum, as in the row kernels, spends about fifty warp
// instructions on each incidence for some thirty products: 353 us.
constexpr int kResY = 20;  // row stride of -Y[a][p][4]: the lanes' rows a start in different bank groups

template <bool GN>
__device__ __forceinline__ void vel_residual_node(const float *sY, int64_t n, const int4 *__restrict__ ninfo,
                                                  const uint32_t *__restrict__ inc, const float *__restrict__ rec,
                                                  const float *__restrict__ gn_res, double *__restrict__ res_u,
                                                  const NSCoeff &co) {
    const int4 inf = ninfo[n];
    const int m = node_m(inf);
    const uint32_t *il = inc + node_i0(inf);
    float rj[30], rb[12], rg[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 30; k++) rj[k] = 0.0f;
#pragma unroll
    for (int k = 0; k < 12; k++) rb[k] = 0.0f;
    uint32_t next = m > 0 ? __ldg(il) : 0u;
#pragma unroll 1
    for (int t = 0; t < m; t++) {
        const uint32_t ea = next;
        if (t + 1 < m) next = __ldg(il + t + 1);
        const int a = (int)(ea & 15u);
        const float4 *r = reinterpret_cast<const float4 *>(rec + (size_t)(ea >> 4) * kNSResRecord);
        float u[32], na[12];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float4 v = __ldg(r + kResRecNA / 4 + 3 * a + k);
            na[4 * k] = v.x; na[4 * k + 1] = v.y; na[4 * k + 2] = v.z; na[4 * k + 3] = v.w;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float4 v = __ldg(r + kResRecU / 4 + k);
            u[4 * k] = v.x; u[4 * k + 1] = v.y; u[4 * k + 2] = v.z; u[4 * k + 3] = v.w;
        }
        const float4 pv = __ldg(r + kResRecP / 4);
        const float pp[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float4 bs = __ldg(r + i);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                const float4 y = lds4(sY + kResY * a + 4 * p);
                const float bt = fmaf(bs.z, y.z, fmaf(bs.y, y.y, bs.x * y.x));
                rb[4 * i + p] = fmaf(bt, pp[p], rb[4 * i + p]);
            }
            if (GN) rg[i] += __ldg(gn_res + (size_t)(ea >> 4) * 32 + 3 * a + i);
        }
#pragma unroll
        for (int b = 0; b < 10; b++)
#pragma unroll
            for (int j = 0; j < 3; j++) rj[3 * b + j] = fmaf(na[b], u[3 * b + j], rj[3 * b + j]);
    }
    const float cuu = (float)co.uu;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        // vel_residual_out's trees
        const float x = (((rj[i] + rj[3 + i]) + (rj[6 + i] + rj[9 + i])) + ((rj[12 + i] + rj[15 + i]) + (rj[18 + i] + rj[21 + i]))) +
                        (rj[24 + i] + rj[27 + i]);
        const float z = (rb[4 * i] + rb[4 * i + 1]) + (rb[4 * i + 2] + rb[4 * i + 3]);
        const float s = fmaf(cuu, x, (float)co.up * z);
        res_u[3 * n + i] = f2d_exact(GN ? fmaf(cuu, rg[i], s) : s);
    }
}

// the pressure residual: one thread per pressure node, the sums of the lanes
// (b, j) in registers and their pairwise (xor) tree at the end
__device__ __forceinline__ void pres_residual_node(const float *sY, int64_t n, const int64_t *__restrict__ inc_ptr,
                                                   const uint32_t *__restrict__ inc, const float *__restrict__ rec,
                                                   double *__restrict__ res_p, float cpu) {
    const int64_t i0 = inc_ptr[n];
    const int m = (int)(inc_ptr[n + 1] - i0);
    float s[32];
#pragma unroll
    for (int k = 0; k < 32; k++) s[k] = 0.0f;
#pragma unroll 1
    for (int t = 0; t < m; t++) {
        const uint32_t ea = __ldg(inc + i0 + t);
        const int q = (int)(ea & 15u);
        const float4 *r = reinterpret_cast<const float4 *>(rec + (size_t)(ea >> 4) * kNSResRecord);
        float u[32];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float4 v = __ldg(r + kResRecU / 4 + k);
            u[4 * k] = v.x; u[4 * k + 1] = v.y; u[4 * k + 2] = v.z; u[4 * k + 3] = v.w;
        }
        const float4 b0 = __ldg(r), b1 = __ldg(r + 1), b2 = __ldg(r + 2);
#pragma unroll
        for (int b = 0; b < 10; b++) {
            const float4 y = lds4(sY + kResY * b + 4 * q);
            s[3 * b] = fmaf(fmaf(b0.z, y.z, fmaf(b0.y, y.y, b0.x * y.x)), u[3 * b], s[3 * b]);
            s[3 * b + 1] = fmaf(fmaf(b1.z, y.z, fmaf(b1.y, y.y, b1.x * y.x)), u[3 * b + 1], s[3 * b + 1]);
            s[3 * b + 2] = fmaf(fmaf(b2.z, y.z, fmaf(b2.y, y.y, b2.x * y.x)), u[3 * b + 2], s[3 * b + 2]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (k < o) s[k] += s[k + o];
    res_p[n] = f2d_exact(cpu * s[0]);
}

// blocks [0, pblocks) take the pressure nodes (24 incidences each on the
// structured meshes: the long threads start first), the rest the velocity nodes
template <bool GN>
__global__ void __launch_bounds__(128) k_ns_residual(const int4 *__restrict__ ninfo, const uint32_t *__restrict__ inc,
                                                     const int64_t *__restrict__ pinc_ptr,
                                                     const uint32_t *__restrict__ pinc, const float *__restrict__ rec,
                                                     const float *__restrict__ gtab, const float *__restrict__ gn_res,
                                                     int64_t nnodes, int64_t pnodes, unsigned pblocks,
                                                     double *__restrict__ res_u, double *__restrict__ res_p, NSCoeff co) {
    __shared__ __align__(16) float sY[10 * kResY];  // -Y[a][p][4]
    for (int t = threadIdx.x; t < 160; t += blockDim.x) sY[kResY * (t >> 4) + (t & 15)] = -gtab[kTabY + t];
    __syncthreads();
    if (blockIdx.x < pblocks) {
        const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
        if (n < pnodes) pres_residual_node(sY, n, pinc_ptr, pinc, rec, res_p, (float)co.pu);
    } else {
        const int64_t n = (blockIdx.x - pblocks) * (int64_t)blockDim.x + threadIdx.x;
        if (n < nnodes) vel_residual_node<GN>(sY, n, ninfo, inc, rec, gn_res, res_u, co);
    }
}

// dense 34x34 element matrices and element residuals (AssembleFE view)
__global__ void k_ns_dense(const float *__restrict__ rec, const float *__restrict__ gtab, int64_t first, int64_t count,
                           float visc_dens, float dens, int newton, double *Ke, double *re, NSCoeff co) {
    const int64_t e = blockIdx.x;
    if (e >= count) return;
    const int lane = threadIdx.x;
    const float *R = rec + (first + e) * kNSRecord;
    double *J = Ke + e * 34 * 34;
    double *r = re + e * 34;
    for (int t = lane; t < 34 * 34; t += 32) J[t] = 0.0;
    __syncwarp();
    const int b = lane < 30 ? lane / 3 : 0, j = lane < 30 ? lane % 3 : 0;
    float rr[3] = {0, 0, 0};
    for (int a = 0; a < 10; a++) {
        float wv[3] = {0, 0, 0}, part = 0.0f;
        if (lane < 30) part = ns_lane_terms(R, gtab, a, b, j, visc_dens, dens, wv);
        float an = sum3_lanes(part, lane);
        float racc = 0.0f;
        if (lane < 30) {
            for (int i = 0; i < 3; i++) {
                float v = (i == j ? an : 0.0f);
                if (newton) v = fmaf(dens, wv[i], v);
                J[(3 * a + i) * 34 + 3 * b + j] = (double)v;
            }
            racc = an * R[kRecU + 3 * b + j];
        }
        for (int i = 0; i < 3; i++) {
            float s = warp_sum((lane < 30 && j == i) ? racc : 0.0f);
            if (lane == 0) rr[i] = s;
        }
        if (lane < 12) {
            int bi = lane >> 2, bp = lane & 3;
            float v = ns_bt(R, gtab, a, bi, bp);
            J[(3 * a + bi) * 34 + 30 + bp] = (double)v;
            J[(30 + bp) * 34 + 3 * a + bi] = (double)v;
        }
        __syncwarp();
        if (lane == 0) {
            for (int i = 0; i < 3; i++) {
                double s = co.uu * (double)rr[i];
                for (int pp = 0; pp < 4; pp++) s = fma(co.up * J[(3 * a + i) * 34 + 30 + pp], (double)R[kRecP + pp], s);
                r[3 * a + i] = s;
            }
        }
        __syncwarp();
    }
    if (lane < 4) {
        double s = 0.0;
        for (int k = 0; k < 30; k++) s += J[(30 + lane) * 34 + k] * (double)R[kRecU + k];
        r[30 + lane] = co.pu * s;
    }
}

int sm_count_ns() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

}  // namespace

void ns_upload_tables(float *d_tables, cudaStream_t s) {
    // constants of the element, the same for every handle
    static const std::vector<float> tab = [] {
        NSTables t;
        make_ns_tables(&t);
        std::vector<float> h(kNSTab, 0.0f);
        for (int c = 0; c < 3; c++)
            for (int a = 0; a < 10; a++)
                for (int b = 0; b < 10; b++)
                    for (int k = 0; k < 10; k++) h[kTabT + ((a * 3 + k / 4) * 32 + 3 * b + c) * 4 + k % 4] = t.T[c][a][b][k];
        for (int a = 0; a < 10; a++)
            for (int b = 0; b < 10; b++) {
                for (int s = 0; s < 6; s++) h[kTabKS + (a * 10 + b) * 6 + s] = t.KS[a][b][s];
                for (int m = 0; m < 4; m++) h[kTabR + (a * 10 + b) * 4 + m] = t.R[a][b][m];
            }
        for (int b = 0; b < 10; b++)
            for (int p = 0; p < 4; p++)
                for (int c = 0; c < 3; c++) h[kTabY + (b * 4 + p) * 4 + c] = t.Y[c][p][b];
        for (int ab = 0; ab < 100; ab++)
            for (int kk = 0; kk < 36; kk++)
                h[kTabB + na_off(ab, kk, kNAStepB) / 4] =
                    kk < 30 ? t.T[kk / 10][ab / 10][ab % 10][kk % 10] : t.KS[ab / 10][ab % 10][kk - 30];
        return h;
    }();
    FEDD_CUDA(cudaMemcpyAsync(d_tables, tab.data(), tab.size() * sizeof(float), cudaMemcpyHostToDevice, s));
}

void launch_ns_record(const float *geo, const int32_t *conn2, const int32_t *conn1, int64_t ne, const double *u,
                      const double *p, const float *d_tables, float visc_dens, float dens, float *rec, int *d_err,
                      cudaStream_t s, LaunchCounter &lc, int64_t e_begin, int64_t e_end, bool residual_only) {
    if (e_end < 0) e_end = ne;
    const int64_t count = e_end - e_begin;
    if (count <= 0) return;
    // persistent CTAs, one per SM (shared memory, all 512 TMEM columns)
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(count, (int64_t)kRecTile), (int64_t)sm_count_ns());
    auto kern = residual_only ? k_ns_record<true> : k_ns_record<false>;
    FEDD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRecSmem));
    kern<<<grid, kRecThreads, kRecSmem, s>>>(geo, conn2, conn1, ne, u, p, rec, d_err, e_begin, e_end, d_tables, visc_dens,
                                             dens);
    FEDD_CUDA(cudaGetLastError());
    lc.n += 1;
}

void launch_ns_node_info(const Graph &g, const int64_t *padj_ptr, const int32_t *vmap, int4 *info, cudaStream_t s) {
    const int64_t nn = g.nrow_nodes;
    if (nn == 0) return;
    k_ns_node_info<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(g.inc_ptr.p, g.adj_ptr.p, padj_ptr, vmap, nn, info);
    FEDD_CUDA(cudaGetLastError());
}

void launch_ns_vel_rows(const Graph &g, const int4 *ninfo, const float *rec, const float *d_tables,
                        const int64_t *rowptr00, const int64_t *rowptr01, double *vals00, double *vals01, double *res_u,
                        float dens, int newton, int max_adj, int max_padj, bool vmap, const int64_t *rowptr10,
                        double *vals10, double *res_p, const float *gstage, cudaStream_t s, LaunchCounter &lc,
                        int64_t n_begin, int64_t n_end, unsigned long long *work, const NSCoeff &co) {
    const bool gn = gstage != nullptr;
    const int acc_words = vel_acc_words(max_adj, max_padj, vmap);
    const size_t tables = kVelTab * sizeof(float);
    const size_t per_node = (size_t)(kVRing * (gn ? kVStageGn : kVStage) + acc_words) * sizeof(float);
    const int64_t nn = n_end < 0 ? g.nrow_nodes : n_end, count = nn - n_begin, sms = sm_count_ns();
    // one node per warp below six nodes for each of the chip's warps (24,389
    // nodes: pairs 57 us, 66 with the viscous rows, one per warp 61 and 73;
    // 9,261 nodes 38 and 38 against 34 and 39)
    const int npw = count < 6 * 2 * sms * vel_warps(gn, 1) ? 1 : 2;
    // two CTAs per SM share its shared memory; one where the rows are so long
    // that two would leave few warps
    const size_t per_warp = npw * per_node;
    const int most = vel_warps(gn, npw);
    int warps = (int)std::min<size_t>(most, (113 * 1024 - tables) / per_warp);
    if (warps < 4) warps = (int)std::max<size_t>(1, std::min<size_t>(most, (227 * 1024 - tables) / per_warp));
    // pairs come from groups of eight nodes, of four below 40 nodes per warp,
    // where the last groups would leave warps idle (Newton form, lattice and
    // shuffled: 50,653 nodes 92 and 92 us against 107 and 119; 91,125 nodes 150
    // and 157 against 161 and 155; 185,193 nodes 281 and 303 against 291 and 298)
    const int group = npw == 1 ? 1 : count < 40 * 2 * sms * warps ? 4 : 8;
    if (npw == 1 && count <= 2 * sms * warps) {
        work = nullptr;  // a node per warp at most, spread over all SMs
        warps = (int)std::min<int64_t>(warps, std::max<int64_t>(2, ceil_div(count, 2 * sms)));
    }
    const size_t smem = tables + (size_t)warps * per_warp;
    const bool res = res_u || res_p;
    using Kern = decltype(&k_ns_vel_rows<true, true, 1, true>);
    auto pick = [&](auto GN, auto NEWTON) -> Kern {
        constexpr bool g = decltype(GN)::value, n = decltype(NEWTON)::value;
        if (npw == 1) return res ? k_ns_vel_rows<g, n, 1, true> : k_ns_vel_rows<g, n, 1, false>;
        return res ? k_ns_vel_rows<g, n, 2, true> : k_ns_vel_rows<g, n, 2, false>;
    };
    const std::true_type yes;
    const std::false_type no;
    const Kern kern = gn ? (newton ? pick(yes, yes) : pick(yes, no)) : (newton ? pick(no, yes) : pick(no, no));
    allow_dynamic_smem(kern);
    unsigned grid = (unsigned)std::min<int64_t>((count + group * warps - 1) / (group * warps), sms * 4);
    if (work) {  // dynamic positions: exactly the CTAs that fit
        int per_sm = 0;
        FEDD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, smem));
        grid = (unsigned)std::min<int64_t>(grid, sms * std::max(per_sm, 1));
    }
    if (grid == 0) return;
    kern<<<grid, 32 * warps, smem, s>>>(ninfo, g.inc.p, g.slots.p, rec, d_tables, rowptr00, rowptr01, vals00, vals01,
                                        res_u, nn, dens, group, acc_words, n_begin, rowptr10, vals10, res_p, gstage,
                                        work, co);
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_ns_pres_rows(const Graph &gp, const float *rec, const float *d_tables, const int64_t *rowptr10,
                         double *vals10, double *res_p, int max_adj, cudaStream_t s, LaunchCounter &lc, const NSCoeff &co) {
    const int warps = 8;
    const int acc_words = (3 * max_adj + 1 + 3) & ~3;
    size_t smem = (160 + (size_t)warps * (kPRing * kPStage + acc_words)) * sizeof(float);
    allow_dynamic_smem(k_ns_pres_rows);
    const int64_t nn = gp.nrow_nodes;
    unsigned grid = (unsigned)std::min<int64_t>((nn + warps - 1) / warps, (int64_t)sm_count_ns() * 8);
    if (grid == 0) return;
    k_ns_pres_rows<<<grid, 32 * warps, smem, s>>>(gp.inc_ptr.p, gp.inc.p, gp.slots.p, gp.adj_ptr.p, rec, d_tables,
                                                  rowptr10, vals10, res_p, nn, max_adj, (float)co.pu);
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_ns_residual(const Graph &g, const Graph &gp, const int4 *ninfo, const float *rec, const float *d_tables,
                        const float *gn_res, double *res_u, double *res_p, cudaStream_t s, LaunchCounter &lc,
                        const NSCoeff &co) {
    const int64_t nn = g.nrow_nodes, np = gp.nrow_nodes;
    const unsigned pb = ceil_div(np, 128), vb = ceil_div(nn, 128);
    if (pb + vb == 0) return;
    auto kern = gn_res ? k_ns_residual<true> : k_ns_residual<false>;
    kern<<<pb + vb, 128, 0, s>>>(ninfo, g.inc.p, gp.inc_ptr.p, gp.inc.p, rec, d_tables, gn_res, nn, np, pb, res_u, res_p,
                                 co);
    FEDD_CUDA(cudaGetLastError());
    lc.n++;
}

void launch_ns_dense(const float *rec, const float *d_tables, int64_t first, int64_t count, float visc_dens,
                     float dens, int newton, double *Ke, double *re, cudaStream_t s, const NSCoeff &co) {
    if (count == 0) return;
    k_ns_dense<<<(unsigned)count, 32, 0, s>>>(rec, d_tables, first, count, visc_dens, dens, newton, Ke, re, co);
    FEDD_CUDA(cudaGetLastError());
}

}  // namespace fedd
