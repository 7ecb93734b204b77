// graph.cu -- device construction of incidences, node adjacency and CSR
// patterns (built once per mesh).
//
// Replaces the pattern FEDDLib obtains from Tpetra: FE::addFeBlock /
// addFeBlockMatrix insert every dof pair of every node pair of an element
// (feddlib/core/FE/FE_def.hpp:1419-1442, 982-1062) and fillComplete sorts the
// columns and merges duplicates (Matrix_decl.hpp:133-138).  Here: per row
// node, the union of the column nodes of its incident elements, made unique
// by one warp in a shared-memory hash table and put in order by counting
// ranks; the scalar CSR follows as node pattern x (dofs_r x dofs_c) blocks.
//
// The element arrays are read as the caller lays them out (num_elements x
// npe): the ten column nodes of an incidence are then one or two 32-byte
// sectors, where the transposed layout touches ten.  Against a bitonic sort
// of all candidates (240 of a P2 vertex for 65 distinct nodes), run once to
// count and once to fill, adjacency counting (with the sort of the incidences) went from 210 to 75 us
// and filling from 267 to 99 us on a 24^3 x 6 mesh in file order (P2
// rows, P2 columns).
#include "engine.hpp"

namespace fedd {

namespace {

constexpr int kMaxCand = kMaxIncidence * 10;  // candidates of one row node at most
constexpr int kHash = 512;                    // hash table entries per warp (at most 255 + 32 are ever inserted)
constexpr int kGraphWarps = 8;

__global__ void k_count_inc(const int32_t *__restrict__ conn, int npe, int64_t ne, int64_t nnodes,
                            int32_t *cnt, int *err) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= ne * npe) return;
    int32_t n = conn[t];
    if (n < 0 || n >= nnodes) {
        set_dev_error(err, kDevMesh);
        return;
    }
    atomicAdd(&cnt[n], 1);
}

// counts each node's cursor down to zero: entry ptr[n] + cursor
__global__ void k_fill_inc(const int32_t *__restrict__ conn, int npe, int64_t ne, int64_t nnodes,
                           const int64_t *__restrict__ ptr, int32_t *cursor, uint32_t *inc) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= ne * npe) return;
    int32_t n = conn[t];
    if (n < 0 || n >= nnodes) return;
    const int64_t e = t / npe;
    const int a = (int)(t - e * npe);
    int pos = atomicSub(&cursor[n], 1) - 1;
    inc[ptr[n] + pos] = ((uint32_t)e << 4) | (uint32_t)a;
}

// the fill order above depends on atomic timing: each list is sorted so that
// the incidence order (and with it the summation order) is fixed: by the
// node's local index in the element, then by element, so that a row kernel
// meets the incidences sharing a local index (and its rows of the reference
// tables) in one run
__device__ __forceinline__ uint32_t inc_key(uint32_t v) { return ((v & 15u) << 28) | (v >> 4); }

// one warp sorts its node's m <= 64 incidences (lane k holds entries k and
// k + 32): every entry's rank is the number of smaller keys (keys differ)
__device__ __forceinline__ void warp_sort_incidences(uint32_t *inc, int m, int lane) {
    const uint32_t lo = lane < m ? inc[lane] : 0xffffffffu, hi = lane + 32 < m ? inc[lane + 32] : 0xffffffffu;
    const uint32_t klo = inc_key(lo), khi = inc_key(hi);
    int rlo = 0, rhi = 0;
    for (int t = 0; t < m; t++) {
        const uint32_t k = __shfl_sync(0xffffffffu, t < 32 ? klo : khi, t & 31);
        rlo += k < klo;
        rhi += k < khi;
    }
    __syncwarp();
    if (lane < m) inc[rlo] = lo;
    if (lane + 32 < m) inc[rhi] = hi;
    __syncwarp();
}

// per-warp shared memory of the node union
struct __align__(16) UnionSmem {
    int32_t key[kHash];       // hash table: node ids, -1 empty
    int32_t list[256];        // distinct nodes in order of first occurrence (padded to a multiple of 4)
    uint16_t at[256];         // their places in the table
    uint8_t rank[kHash];      // place -> position in the sorted adjacency row
    uint16_t cand[kMaxCand];  // place of every candidate
};

// Enters the column nodes of a node's m incidences into the hash table key;
// with LIST also the list of distinct ones and every candidate's place into
// S (key is S->key then).  Returns
// the number of distinct nodes, or -1 when they exceed kMaxAdjacency.
// Negative node ids do not occur: the caller has counted, and so checked,
// every element array (an array with bad ids is reported before the result
// is used; its entries are only compared here).
template <bool LIST>
__device__ __forceinline__ int node_union(int32_t *key, UnionSmem *S, const uint32_t *__restrict__ inc, int m,
                                          const int32_t *__restrict__ col_conn, int npe, int lane) {
    const int cnt = m * npe;
    int bits = 6;
    while (bits < 9 && (1 << bits) < 2 * cnt) bits++;
    const int mask = (1 << bits) - 1;
    for (int i = lane; i <= mask; i += 32) key[i] = -1;
    __syncwarp();
    int K = 0;
    for (int base = 0; base < cnt; base += 32) {
        const int i = base + lane;
        bool fresh = false;
        int32_t v = 0;
        int h = 0;
        if (i < cnt) {
            const int k = i / npe, j = i - k * npe;
            v = __ldg(col_conn + (int64_t)(inc[k] >> 4) * npe + j);
            h = (int)(((uint32_t)v * 2654435769u) >> (32 - bits));
            // at most 255 + 32 of the 512 places are taken, or cnt of 2 cnt
            for (;;) {
                const int32_t old = atomicCAS(&key[h], -1, v);
                fresh = old == -1;
                if (fresh || old == v) break;
                h = (h + 1) & mask;
            }
            if (LIST) S->cand[i] = (uint16_t)h;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, fresh);
        if (LIST && fresh) {
            const int pos = K + __popc(bal & ((1u << lane) - 1u));
            if (pos < 256) {
                S->list[pos] = v;
                S->at[pos] = (uint16_t)h;
            }
        }
        K += __popc(bal);
        if (K > kMaxAdjacency) return -1;
    }
    __syncwarp();
    return K;
}

// SORT: the first adjacency of a graph also puts its incidences in order
template <bool SORT>
__global__ void __launch_bounds__(32 * kGraphWarps) k_adj_count(const int64_t *__restrict__ ptr, uint32_t *inc,
                                                                const int32_t *__restrict__ col_conn, int npe_col,
                                                                int64_t nnodes, int64_t *cnt, int *err, int *maxinc,
                                                                int *maxadj) {
    __shared__ int32_t key[kGraphWarps][kHash];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n = blockIdx.x * (int64_t)kGraphWarps + w;
    if (n > nnodes) return;
    if (n == nnodes) {  // the scan's last entry
        if (lane == 0) cnt[n] = 0;
        return;
    }
    const int64_t b = ptr[n];
    const int64_t m = ptr[n + 1] - b;
    int K = -1;
    if (m <= kMaxIncidence) {
        if (SORT) warp_sort_incidences(inc + b, (int)m, lane);
        K = node_union<false>(key[w], nullptr, inc + b, (int)m, col_conn, npe_col, lane);
    }
    if (lane == 0) {
        if (K < 0) set_dev_error(err, kDevCapacity);
        cnt[n] = K < 0 ? 0 : K;
        // the maxima settle after a few nodes: most warps only read them
        if (SORT && m <= kMaxIncidence && (int)m > *(volatile int *)maxinc) atomicMax(maxinc, (int)m);
        if (K > *(volatile int *)maxadj) atomicMax(maxadj, K);
    }
}

__global__ void __launch_bounds__(32 * kGraphWarps) k_adj_fill(const int64_t *__restrict__ ptr,
                                                               const uint32_t *__restrict__ inc,
                                                               const int32_t *__restrict__ col_conn, int npe_col,
                                                               int64_t nnodes, const int64_t *__restrict__ adj_ptr,
                                                               int32_t *adj, uint8_t *slots, int slot_off) {
    __shared__ UnionSmem smem[kGraphWarps];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n = blockIdx.x * (int64_t)kGraphWarps + w;
    if (n >= nnodes) return;
    UnionSmem &S = smem[w];
    const int64_t b = ptr[n];
    const int m = (int)(ptr[n + 1] - b);
    const int K = node_union<true>(S.key, &S, inc + b, m, col_conn, npe_col, lane);
    if (K <= 0) return;
    // pad the list to whole 16-byte reads with ids above every node's
    if (lane < 4 && K + lane < 256) S.list[K + lane] = 0x7fffffff;
    __syncwarp();
    // every node's position is the number of smaller ids in the list
    const int64_t a0 = adj_ptr[n];
    for (int i = lane; i < K; i += 32) {
        const int32_t v = S.list[i];
        int r = 0;
        for (int t = 0; t < K; t += 4) {
            const int4 x = *reinterpret_cast<const int4 *>(S.list + t);
            r += (x.x < v) + (x.y < v) + (x.z < v) + (x.w < v);
        }
        adj[a0 + r] = v;
        S.rank[S.at[i]] = (uint8_t)r;
    }
    __syncwarp();
    for (int i = lane; i < m * npe_col; i += 32) {
        const int k = i / npe_col, j = i - k * npe_col;
        slots[(b + k) * kSlotStride + slot_off + j] = S.rank[S.cand[i]];
    }
    if (slot_off == 0)  // the row node's local index, for the row kernels' staged slot maps
        for (int k = lane; k < m; k += 32) slots[(b + k) * kSlotStride + kSlotLocal] = (uint8_t)(inc[b + k] & 15u);
}

// the totals of up to three adjacencies next to the maxima, so that one copy
// to the host brings everything the build needs
__global__ void k_collect(GraphStats *st, const int64_t *a0, const int64_t *a1, const int64_t *a2) {
    if (a0) st->n_adj[0] = *a0;
    if (a1) st->n_adj[1] = *a1;
    if (a2) st->n_adj[2] = *a2;
}

__global__ void k_csr(const int64_t *__restrict__ adj_ptr, const int32_t *__restrict__ adj, int64_t nnodes,
                      int dr_n, int dc_n, int64_t *rowptr, int32_t *colind, int64_t nnz) {
    int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t n = blockIdx.x * (int64_t)(blockDim.x >> 5) + w;
    if (n >= nnodes) return;
    int64_t a0 = adj_ptr[n];
    int K = (int)(adj_ptr[n + 1] - a0);
    int64_t base = (int64_t)dr_n * dc_n * a0;
    if (lane < dr_n) rowptr[n * dr_n + lane] = base + (int64_t)lane * dc_n * K;
    if (n == nnodes - 1 && lane == 0) rowptr[nnodes * dr_n] = nnz;
    for (int i = lane; i < K * dc_n; i += 32) {
        int s = i / dc_n, dc = i - s * dc_n;
        int32_t c = adj[a0 + s] * dc_n + dc;
        for (int dr = 0; dr < dr_n; dr++) colind[base + (int64_t)dr * dc_n * K + i] = c;
    }
}

// ---- scans ------------------------------------------------------------
template <class TIn>
__global__ void k_scan_block(const TIn *in, int64_t *out, int64_t *bsum, int64_t n) {
    __shared__ int64_t ws[32];
    int64_t i = blockIdx.x * 1024LL + threadIdx.x;
    int64_t v = i < n ? (int64_t)in[i] : 0;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t s = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int64_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        ws[lane] = s;
    }
    __syncthreads();
    int64_t incl = x + (w > 0 ? ws[w - 1] : 0);
    if (i < n) out[i] = incl - v;
    if (threadIdx.x == 1023 && bsum) bsum[blockIdx.x] = incl;
}

__global__ void k_scan_add(int64_t *out, const int64_t *boff, int64_t n) {
    int64_t i = blockIdx.x * 1024LL + threadIdx.x;
    if (i < n) out[i] += boff[blockIdx.x];
}

template <class TIn>
void scan_impl(const TIn *in, int64_t *out, int64_t n, Arena &tmp, cudaStream_t s) {
    if (n <= 0) return;
    int64_t nb = (n + 1023) / 1024;
    if (nb == 1) {
        k_scan_block<TIn><<<1, 1024, 0, s>>>(in, out, nullptr, n);
        return;
    }
    const size_t mark = tmp.used;
    int64_t *bsum = tmp.take<int64_t>(nb), *boff = tmp.take<int64_t>(nb);
    k_scan_block<TIn><<<(unsigned)nb, 1024, 0, s>>>(in, out, bsum, n);
    scan_impl<int64_t>(bsum, boff, nb, tmp, s);
    k_scan_add<<<(unsigned)nb, 1024, 0, s>>>(out, boff, n);
    tmp.used = mark;  // whoever takes this memory next uses it behind these kernels on s
}

}  // namespace

size_t scan_scratch(int64_t n) {
    size_t bytes = 0;
    for (int64_t nb = (n + 1023) / 1024; nb > 1; nb = (nb + 1023) / 1024) bytes += 2 * Arena::bytes<int64_t>(nb);
    return bytes;
}

void exclusive_scan_i64(const int64_t *in, int64_t *out, int64_t n, Arena &tmp, cudaStream_t s) {
    scan_impl<int64_t>(in, out, n, tmp, s);
}

size_t graph_scratch(int64_t nnodes) {
    // incidence counts, then adjacency counts (never at the same time), and the scans over them
    return Arena::bytes<int64_t>(nnodes + 1) + scan_scratch(nnodes + 1);
}

void build_incidences(Graph &g, int64_t ne, const int32_t *row_conn, int npe_row, GraphStats *st, Arena &tmp,
                      cudaStream_t s) {
    const int64_t nn = g.nrow_nodes, nt = ne * npe_row;
    const size_t mark = tmp.used;
    int32_t *cnt = tmp.take<int32_t>(nn + 1);
    FEDD_CUDA(cudaMemsetAsync(cnt, 0, (nn + 1) * sizeof(int32_t), s));
    k_count_inc<<<ceil_div(nt, 256), 256, 0, s>>>(row_conn, npe_row, ne, nn, cnt, &st->err);
    scan_impl<int32_t>(cnt, g.inc_ptr.p, nn + 1, tmp, s);
    k_fill_inc<<<ceil_div(nt, 256), 256, 0, s>>>(row_conn, npe_row, ne, nn, g.inc_ptr.p, cnt, g.inc.p);
    FEDD_CUDA(cudaGetLastError());
    g.n_inc = nt;
    tmp.used = mark;
}

void count_adjacency(const Graph &g, bool sort, const int32_t *col_conn, int npe_col, int64_t *adj_ptr, int *maxinc,
                     int *maxadj, GraphStats *st, Arena &tmp, cudaStream_t s) {
    const int64_t nn = g.nrow_nodes;
    const size_t mark = tmp.used;
    int64_t *cnt = tmp.take<int64_t>(nn + 1);
    const unsigned nb = ceil_div(nn + 1, kGraphWarps);
    if (sort)
        k_adj_count<true><<<nb, 32 * kGraphWarps, 0, s>>>(g.inc_ptr.p, g.inc.p, col_conn, npe_col, nn, cnt, &st->err,
                                                          maxinc, maxadj);
    else
        k_adj_count<false><<<nb, 32 * kGraphWarps, 0, s>>>(g.inc_ptr.p, g.inc.p, col_conn, npe_col, nn, cnt, &st->err,
                                                           maxinc, maxadj);
    FEDD_CUDA(cudaGetLastError());
    scan_impl<int64_t>(cnt, adj_ptr, nn + 1, tmp, s);
    tmp.used = mark;
}

GraphStats read_graph_stats(GraphStats *st, const int64_t *end0, const int64_t *end1, const int64_t *end2,
                            cudaStream_t s) {
    k_collect<<<1, 1, 0, s>>>(st, end0, end1, end2);
    FEDD_CUDA(cudaGetLastError());
    GraphStats h{};
    FEDD_CUDA(cudaMemcpyAsync(&h, st, sizeof h, cudaMemcpyDeviceToHost, s));
    FEDD_CUDA(cudaStreamSynchronize(s));
    if (h.err == kDevMesh) FEDD_FAIL(FEDD_ERR_MESH, "incidence count: element node index out of range");
    if (h.err == kDevCapacity)
        FEDD_FAIL(FEDD_ERR_CAPACITY, "adjacency: a node exceeds " + std::to_string(kMaxIncidence) +
                                         " incident elements or " + std::to_string(kMaxAdjacency) + " neighbours");
    if (h.err) FEDD_FAIL(FEDD_ERR_CUDA, "graph build: device error " + std::to_string(h.err));
    return h;
}

void fill_adjacency(const Graph &g, const int32_t *col_conn, int npe_col, int slot_off, const int64_t *adj_ptr,
                    int32_t *adj, cudaStream_t s) {
    k_adj_fill<<<ceil_div(g.nrow_nodes, kGraphWarps), 32 * kGraphWarps, 0, s>>>(
        g.inc_ptr.p, g.inc.p, col_conn, npe_col, g.nrow_nodes, adj_ptr, adj, g.slots.p, slot_off);
    FEDD_CUDA(cudaGetLastError());
}

// ---- Taylor-Hood vertex map ------------------------------------------------
__global__ void k_vmap_fill(const int32_t *__restrict__ conn2, const int32_t *__restrict__ conn1, int64_t ne,
                            int32_t *vmap) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    for (int k = 0; k < 4; k++) vmap[conn2[k * ne + e]] = conn1[k * ne + e];
}

__global__ void k_vmap_check_elems(const int32_t *__restrict__ conn2, const int32_t *__restrict__ conn1, int64_t ne,
                                   const int32_t *__restrict__ vmap, int *bad) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    for (int k = 0; k < 4; k++)
        if (vmap[conn2[k * ne + e]] != conn1[k * ne + e]) atomicOr(bad, 1);
    for (int k = 4; k < 10; k++)
        if (vmap[conn2[k * ne + e]] >= 0) atomicOr(bad, 2);
}

__global__ void k_vmap_count(const int32_t *__restrict__ vmap, int64_t nn2, int64_t nn1, int *cnt, int *bad) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= nn2) return;
    const int32_t q = vmap[v];
    if (q >= nn1) atomicOr(bad, 4);
    else if (q >= 0) atomicAdd(cnt + q, 1);
}

// one warp per P2 node: a mapped vertex has exactly one preimage of its P1
// node and the same adjacency row in both graphs
__global__ void k_vmap_rows(const int32_t *__restrict__ vmap, int64_t nn2, const int *__restrict__ cnt,
                            const int64_t *__restrict__ ap2, const int32_t *__restrict__ adj2,
                            const int64_t *__restrict__ ap1, const int32_t *__restrict__ adj1, int *bad) {
    const int64_t v = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (v >= nn2) return;
    const int32_t q = vmap[v];
    if (q < 0) return;
    const int64_t a2 = ap2[v], k2 = ap2[v + 1] - a2, a1 = ap1[q], k1 = ap1[q + 1] - a1;
    if (lane == 0 && (cnt[q] != 1 || k1 != k2)) atomicOr(bad, 8);
    if (k1 != k2) return;
    for (int64_t i = lane; i < k2; i += 32)
        if (adj2[a2 + i] != adj1[a1 + i]) atomicOr(bad, 16);
}

__global__ void k_vmap_cover(const int *__restrict__ cnt, int64_t nn1, int *bad) {
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q < nn1 && cnt[q] != 1) atomicOr(bad, 32);
}

void launch_vertex_map(const int32_t *conn2, const int32_t *conn1, int64_t ne, int64_t nn2, int64_t nn1,
                       const Graph &g2, const Graph &g1, int32_t *vmap, int *bad, Arena &tmp, cudaStream_t s) {
    const size_t mark = tmp.used;
    int *cnt = tmp.take<int>(nn1);
    FEDD_CUDA(cudaMemsetAsync(vmap, 0xff, nn2 * sizeof(int32_t), s));  // -1
    FEDD_CUDA(cudaMemsetAsync(cnt, 0, nn1 * sizeof(int), s));
    k_vmap_fill<<<ceil_div(ne, 256), 256, 0, s>>>(conn2, conn1, ne, vmap);
    k_vmap_check_elems<<<ceil_div(ne, 256), 256, 0, s>>>(conn2, conn1, ne, vmap, bad);
    k_vmap_count<<<ceil_div(nn2, 256), 256, 0, s>>>(vmap, nn2, nn1, cnt, bad);
    k_vmap_rows<<<ceil_div(nn2, 8), 256, 0, s>>>(vmap, nn2, cnt, g2.adj_ptr.p, g2.adj.p, g1.adj_ptr.p, g1.adj.p, bad);
    k_vmap_cover<<<ceil_div(nn1, 256), 256, 0, s>>>(cnt, nn1, bad);
    FEDD_CUDA(cudaGetLastError());
    tmp.used = mark;
}

// largest element index among the incidences of each node range
// [bounds[k], bounds[k + 1]); one warp per node, its range found by a scan
// of the K + 1 bounds
__global__ void k_range_max_elem(const int64_t *__restrict__ inc_ptr, const uint32_t *__restrict__ inc,
                                 const int64_t *__restrict__ bounds, int K, int *out) {
    const int64_t n = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (n >= bounds[K]) return;  // uniform per warp
    int m = -1;
    for (int64_t i = inc_ptr[n] + lane; i < inc_ptr[n + 1]; i += 32) m = max(m, (int)(inc[i] >> 4));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) {
        int k = 0;
        while (k + 1 < K && n >= bounds[k + 1]) k++;
        atomicMax(out + k, m);
    }
}

void node_range_max_elem(const Graph &g, const int64_t *bounds, int K, int64_t *out, cudaStream_t s) {
    DBuf<int64_t> db;
    DBuf<int> dm;
    db.upload(bounds, (size_t)K + 1, s);
    dm.alloc((size_t)K);
    FEDD_CUDA(cudaMemsetAsync(dm.p, 0xff, (size_t)K * sizeof(int), s));  // -1
    if (bounds[K] > 0) {
        k_range_max_elem<<<(unsigned)ceil_div(bounds[K] * 32, 256), 256, 0, s>>>(g.inc_ptr.p, g.inc.p, db.p, K, dm.p);
        FEDD_CUDA(cudaGetLastError());
    }
    std::vector<int> m((size_t)K);
    FEDD_CUDA(cudaMemcpyAsync(m.data(), dm.p, (size_t)K * sizeof(int), cudaMemcpyDeviceToHost, s));
    FEDD_CUDA(cudaStreamSynchronize(s));
    for (int k = 0; k < K; k++) out[k] = m[(size_t)k];
}

void fill_csr(const Csr &c, const int64_t *adj_ptr, const int32_t *adj, int64_t nrow_nodes, int dofs_r, int dofs_c,
              cudaStream_t s) {
    if (nrow_nodes <= 0) return;
    k_csr<<<ceil_div(nrow_nodes, 8), 256, 0, s>>>(adj_ptr, adj, nrow_nodes, dofs_r, dofs_c, c.rowptr.p, c.colind.p,
                                                   c.nnz);
    FEDD_CUDA(cudaGetLastError());
}

}  // namespace fedd
