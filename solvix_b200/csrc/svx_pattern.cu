// svx_pattern.cu - K3: the CSR pattern of the global stiffness, built on the
// device from the mesh connectivity.
//
// The reference builds its pattern implicitly: every element pushes all
// N x N (row, col) triplets of its node pairs, zeros included, and every
// dof gets a diagonal seed (crates/solvix-core/src/assembly.rs:120-133,
// :299-302); csr_from_triplets then sorts each row by column
// (assembly.rs:87-116).  The resulting pattern is exactly
//   row (i, a): columns (j, b) for every node j sharing an element with i
//               (i itself included) and every dof b, ascending;
//   a node used by no element keeps only its diagonal.
// This file computes that pattern without materialising triplets:
//   1. node -> incident (element, local position) slots, sorted ascending
//      (counting pass, scan, atomic fill, per-node insertion sort);
//   2. node adjacency = sorted union of the slots' element nodes;
//   3. row_ptr / col_idx / diagonal positions from the node blocks;
//   4. the element-to-nonzero map: for each slot and each node of the slot's
//      element, its position in the owner node's adjacency.
// All integer work; the result is bit-exact against the oracle's CSR.

#include "svx_internal.h"

#include <climits>

namespace svx {

namespace {

constexpr int SCAN_T = 512;
constexpr int SCAN_I = 8;
constexpr int64_t SCAN_TILE = int64_t(SCAN_T) * SCAN_I;

__global__ void scan_tile_kernel(const int64_t* __restrict__ in, int64_t* __restrict__ out,
                                 int64_t n, int64_t* __restrict__ tile_sums) {
    __shared__ int64_t s[SCAN_T];
    const int64_t base = int64_t(blockIdx.x) * SCAN_TILE + int64_t(threadIdx.x) * SCAN_I;
    int64_t v[SCAN_I];
    int64_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
        int64_t idx = base + k;
        v[k] = idx < n ? in[idx] : 0;
        sum += v[k];
    }
    s[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < SCAN_T; off <<= 1) {
        int64_t t = threadIdx.x >= off ? s[threadIdx.x - off] : 0;
        __syncthreads();
        s[threadIdx.x] += t;
        __syncthreads();
    }
    int64_t run = s[threadIdx.x] - sum;
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
        int64_t idx = base + k;
        if (idx < n) out[idx] = run;
        run += v[k];
    }
    if (threadIdx.x == SCAN_T - 1) tile_sums[blockIdx.x] = s[SCAN_T - 1];
}

__global__ void scan_add_kernel(int64_t* __restrict__ out, int64_t n,
                                const int64_t* __restrict__ tile_offsets) {
    int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx < n) out[idx] += tile_offsets[idx / SCAN_TILE];
}

__global__ void scan_total_kernel(const int64_t* in, int64_t* out, int64_t n) {
    out[n] = n > 0 ? out[n - 1] + in[n - 1] : 0;
}

void scan_rec(svx_ctx* ctx, const int64_t* in, int64_t* out, int64_t n) {
    if (n <= 0) return;
    int64_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    DBuf<int64_t> sums, offs;
    sums.alloc(ctx->pool, tiles + 1);
    scan_tile_kernel<<<unsigned(tiles), SCAN_T, 0, ctx->stream>>>(in, out, n, sums.p);
    SVX_LAUNCH_CHECK();
    if (tiles > 1) {
        offs.alloc(ctx->pool, tiles + 1);
        scan_rec(ctx, sums.p, offs.p, tiles);
        scan_add_kernel<<<unsigned((n + 255) / 256), 256, 0, ctx->stream>>>(out, n, offs.p);
        SVX_LAUNCH_CHECK();
    }
    // the temporaries go back to the context's pool, whose later users are
    // ordered behind this stream
}

// ---- 1. incidence ---------------------------------------------------------
__global__ void count_incidence_kernel(const int64_t* __restrict__ conn_ptr,
                                       const int32_t* __restrict__ conn, int64_t n_elem,
                                       unsigned long long* __restrict__ cnt) {
    int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= n_elem) return;
    for (int64_t q = conn_ptr[e]; q < conn_ptr[e + 1]; ++q)
        atomicAdd(&cnt[conn[q]], 1ull);
}

__global__ void fill_incidence_kernel(const int64_t* __restrict__ conn_ptr,
                                      const int32_t* __restrict__ conn, int64_t n_elem,
                                      const int64_t* __restrict__ slot_ptr,
                                      unsigned long long* __restrict__ cursor,
                                      int64_t* __restrict__ keys) {
    int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= n_elem) return;
    int64_t q0 = conn_ptr[e];
    for (int64_t q = q0; q < conn_ptr[e + 1]; ++q) {
        int32_t node = conn[q];
        unsigned long long pos = atomicAdd(&cursor[node], 1ull);
        keys[slot_ptr[node] + int64_t(pos)] = (e << 8) | int64_t(q - q0);
    }
}

// Per-node insertion sort of the (element, local) keys, then split.
__global__ void sort_slots_kernel(int64_t n_nodes, const int64_t* __restrict__ slot_ptr,
                                  int64_t* __restrict__ keys, int32_t* __restrict__ slot_elem,
                                  uint8_t* __restrict__ slot_local, int* max_slots) {
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_nodes) return;
    int64_t a = slot_ptr[i], b = slot_ptr[i + 1];
    for (int64_t x = a + 1; x < b; ++x) {
        int64_t key = keys[x];
        int64_t y = x;
        while (y > a && keys[y - 1] > key) {
            keys[y] = keys[y - 1];
            --y;
        }
        keys[y] = key;
    }
    for (int64_t x = a; x < b; ++x) {
        slot_elem[x] = int32_t(keys[x] >> 8);
        slot_local[x] = uint8_t(keys[x] & 0xff);
    }
    atomicMax(max_slots, int(b - a));
}

// ---- 2. adjacency ------------------------------------------------------------
// G lanes a node: a warp where elements have up to 8 nodes, 8 lanes where they
// have up to 4 (a plate's 16 element nodes leave most of a warp idle).  The
// nodes of up to 16 or 8 elements are held in registers, four a lane, and
// every round takes the smallest above the last by a minimum over the group.
// (A thread a node read all its elements' nodes again each round: 27 rounds of
// 64 dependent loads, 65 us for 325 nodes and 305 us for 150,625, twice a
// pattern; now 6 and 101.)
template <int G>
struct Neighbours {
    static constexpr int HELD = 4, L = G == 32 ? 8 : 4, STEP = G / L;
    int32_t v[HELD];
    int64_t s0, s1;
    int slot, at;  // the lane's slot of a step and its node there
    bool held;

    __device__ __forceinline__ void open(int64_t a, int64_t b, int max_nn,
                                         const int32_t* __restrict__ slot_elem,
                                         const int64_t* __restrict__ conn_ptr,
                                         const int32_t* __restrict__ conn) {
        s0 = a;
        s1 = b;
        slot = int(threadIdx.x & (G - 1)) / L;
        at = int(threadIdx.x & (L - 1));
        held = b - a <= STEP * HELD && max_nn <= L;
#pragma unroll
        for (int t = 0; t < HELD; ++t) {
            const int64_t s = a + STEP * t + slot;
            v[t] = INT_MAX;
            if (held && s < b) {
                const int64_t e = slot_elem[s], q = conn_ptr[e] + at;
                if (q < conn_ptr[e + 1]) v[t] = conn[q];
            }
        }
    }
    // Smallest element node > last (INT_MAX if none), the same in the group.
    // All lanes of the warp call it.
    __device__ __forceinline__ int32_t next(int32_t last, const int32_t* __restrict__ slot_elem,
                                            const int64_t* __restrict__ conn_ptr,
                                            const int32_t* __restrict__ conn) const {
        int32_t best = INT_MAX;
        if (held) {
#pragma unroll
            for (int t = 0; t < HELD; ++t)
                if (v[t] > last && v[t] < best) best = v[t];
        } else {
            for (int64_t s = s0 + slot; s < s1; s += STEP) {
                const int64_t e = slot_elem[s], q1 = conn_ptr[e + 1];
                for (int64_t q = conn_ptr[e] + at; q < q1; q += L)
                    if (conn[q] > last && conn[q] < best) best = conn[q];
            }
        }
        __syncwarp();
        if (G == 32) return __reduce_min_sync(0xffffffffu, best);
#pragma unroll
        for (int m = G / 2; m; m >>= 1)
            best = min(best, __shfl_xor_sync(0xffffffffu, best, m));
        return best;
    }
};

template <int G>
__global__ void degree_kernel(int64_t n_nodes, int max_nn, const int64_t* __restrict__ slot_ptr,
                              const int32_t* __restrict__ slot_elem,
                              const int64_t* __restrict__ conn_ptr,
                              const int32_t* __restrict__ conn, int64_t* __restrict__ deg,
                              int* max_deg) {
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / G;
    const bool node = i < n_nodes;
    Neighbours<G> nb;
    nb.open(node ? slot_ptr[i] : 0, node ? slot_ptr[i + 1] : 0, max_nn, slot_elem, conn_ptr, conn);
    int d = 0;
    for (int32_t last = -1;;) {
        const int32_t nx = nb.next(last, slot_elem, conn_ptr, conn);
        if (nx != INT_MAX) ++d;
        last = nx;
        if (!__any_sync(0xffffffffu, nx != INT_MAX)) break;
    }
    if (node && (threadIdx.x & (G - 1)) == 0) {
        deg[i] = d;
        if (d > *static_cast<volatile int*>(max_deg)) atomicMax(max_deg, d);
    }
}

// ---- 3. CSR rows --------------------------------------------------------------
__global__ void node_nnz_kernel(int64_t n_nodes, int ndof, const int64_t* __restrict__ adj_ptr,
                                int64_t* __restrict__ node_nnz) {
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_nodes) return;
    int64_t d = adj_ptr[i + 1] - adj_ptr[i];
    node_nnz[i] = d > 0 ? int64_t(ndof) * ndof * d : int64_t(ndof);
}

// G lanes a node list its neighbours, map its elements' nodes to their
// positions in that list and write its ND rows: all three in the rounds the
// list takes (as three kernels they searched the list for each element node
// and each diagonal, 39 us beside the list's 70 for 1,025 solid nodes, 728
// beside 690 for the 40 solids of a batch; now 9 and 649).
template <int ND, int G>
__global__ void rows_kernel(int64_t n_nodes, int max_nn, const int64_t* __restrict__ slot_ptr,
                            const int32_t* __restrict__ slot_elem,
                            const int64_t* __restrict__ conn_ptr,
                            const int32_t* __restrict__ conn,
                            const int64_t* __restrict__ adj_ptr, int32_t* adj,
                            const int64_t* __restrict__ node_base, uint16_t* slot_map,
                            int32_t* __restrict__ row_ptr, int32_t* __restrict__ col_idx,
                            int32_t* __restrict__ diag_pos) {
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / G;
    const bool node = i < n_nodes;
    const int lane = threadIdx.x & (G - 1);
    const int64_t a0 = node ? adj_ptr[i] : 0, base = node ? node_base[i] : 0;
    const int d = node ? int(adj_ptr[i + 1] - a0) : 0;
    if (i == n_nodes - 1 && lane == 0) row_ptr[n_nodes * ND] = int32_t(node_base[n_nodes]);
    if (node && d == 0 && lane < ND) {
        const int64_t row = i * ND + lane;
        row_ptr[row] = int32_t(base + lane);
        col_idx[base + lane] = int32_t(row);
        diag_pos[row] = int32_t(base + lane);
    }
    Neighbours<G> nb;
    nb.open(d > 0 ? slot_ptr[i] : 0, d > 0 ? slot_ptr[i + 1] : 0, max_nn, slot_elem, conn_ptr,
            conn);
    const int most = __reduce_max_sync(0xffffffffu, d);
    int self = 0;
    int32_t nx = -1;
    for (int k = 0; k < most; ++k) {
        nx = nb.next(nx, slot_elem, conn_ptr, conn);
        if (k >= d) continue;  // a neighbour in the warp has more
        if (nx == int32_t(i)) self = k;
        if (lane == 0) adj[a0 + k] = nx;
        if (nb.held) {
#pragma unroll
            for (int t = 0; t < nb.HELD; ++t)
                if (nb.v[t] == nx)
                    slot_map[(nb.s0 + nb.STEP * t + nb.slot) * max_nn + nb.at] = uint16_t(k);
        } else {
            for (int64_t s = nb.s0 + nb.slot; s < nb.s1; s += nb.STEP) {
                const int64_t e = slot_elem[s], q0 = conn_ptr[e];
                const int nn = int(conn_ptr[e + 1] - q0);
                for (int c = nb.at; c < nn; c += nb.L)
                    if (conn[q0 + c] == nx) slot_map[s * max_nn + c] = uint16_t(k);
            }
        }
    }
    __syncwarp();
    const unsigned rowlen = unsigned(ND * d);
    if (d > 0 && lane < ND) {
        const int64_t row = i * ND + lane, first = base + lane * int64_t(rowlen);
        row_ptr[row] = int32_t(first);
        diag_pos[row] = int32_t(first + self * ND + lane);
    }
    for (unsigned r = lane; r < rowlen; r += G) {
        const int32_t col = adj[a0 + r / ND] * ND + int32_t(r % ND);
#pragma unroll
        for (int a = 0; a < ND; ++a) col_idx[base + int64_t(a) * rowlen + r] = col;
    }
}

inline unsigned blocks_for(int64_t n, int t) { return unsigned((n + t - 1) / t); }

}  // namespace

// out[0..n]: exclusive sums of in and their total, all on the device.
void exclusive_scan_i64(svx_ctx* ctx, const int64_t* in, int64_t* out, int64_t n) {
    scan_rec(ctx, in, out, n);
    scan_total_kernel<<<1, 1, 0, ctx->stream>>>(in, out, n);
    SVX_LAUNCH_CHECK();
}

void build_pattern(svx_ctx* ctx, svx_op* op) {
    Pattern& P = op->pat;
    cudaStream_t st = ctx->stream;
    const int64_t nn = op->n_nodes, ne = op->n_elem;
    P.n_nodes = nn;
    P.n_elem = ne;
    P.ndof = op->ndof;
    P.n = nn * op->ndof;

    DBuf<int> flags;  // [0] max_slots, [1] max_deg
    flags.alloc(ctx->pool, 2);
    SVX_CUDA(cudaMemsetAsync(flags.p, 0, 2 * sizeof(int), st));

    // 1. incidence
    DBuf<int64_t> cnt, cursor, keys;
    cnt.alloc(ctx->pool, nn + 1);
    cursor.alloc(ctx->pool, nn + 1);
    SVX_CUDA(cudaMemsetAsync(cnt.p, 0, (nn + 1) * sizeof(int64_t), st));
    SVX_CUDA(cudaMemsetAsync(cursor.p, 0, (nn + 1) * sizeof(int64_t), st));
    if (ne > 0) {
        count_incidence_kernel<<<blocks_for(ne, 256), 256, 0, st>>>(
            op->conn_ptr.p, op->conn.p, ne, reinterpret_cast<unsigned long long*>(cnt.p));
        SVX_LAUNCH_CHECK();
    }
    P.slot_ptr.alloc(ctx->pool, nn + 1);
    exclusive_scan_i64(ctx, cnt.p, P.slot_ptr.p, nn);
    const int64_t n_slots = op->n_conn;
    P.n_slots = n_slots;
    keys.alloc(ctx->pool, n_slots + 1);
    P.slot_elem.alloc(ctx->pool, n_slots + 1);
    P.slot_local.alloc(ctx->pool, n_slots + 1);
    if (ne > 0) {
        fill_incidence_kernel<<<blocks_for(ne, 256), 256, 0, st>>>(
            op->conn_ptr.p, op->conn.p, ne, P.slot_ptr.p,
            reinterpret_cast<unsigned long long*>(cursor.p), keys.p);
        SVX_LAUNCH_CHECK();
    }
    if (nn > 0) {
        sort_slots_kernel<<<blocks_for(nn, 128), 128, 0, st>>>(nn, P.slot_ptr.p, keys.p,
                                                               P.slot_elem.p, P.slot_local.p,
                                                               flags.p);
        SVX_LAUNCH_CHECK();
    }
    keys.reset();
    cursor.reset();

    // 2. adjacency: count, scan, fill
    const bool wide = P.max_nn > 4;
    const int64_t lanes = wide ? 32 : 8;
    DBuf<int64_t> deg;
    deg.alloc(ctx->pool, nn + 1);
    if (nn > 0) {
        (wide ? &degree_kernel<32> : &degree_kernel<8>)<<<blocks_for(nn * lanes, 256), 256, 0, st>>>(
            nn, P.max_nn, P.slot_ptr.p, P.slot_elem.p, op->conn_ptr.p, op->conn.p, deg.p,
            flags.p + 1);
        SVX_LAUNCH_CHECK();
    }
    P.adj_ptr.alloc(ctx->pool, nn + 1);
    exclusive_scan_i64(ctx, deg.p, P.adj_ptr.p, nn);

    // 3. rows, and the one wait of the pattern: the sizes that follow
    DBuf<int64_t> node_nnz;
    node_nnz.alloc(ctx->pool, nn + 1);
    if (nn > 0) {
        node_nnz_kernel<<<blocks_for(nn, 256), 256, 0, st>>>(nn, op->ndof, P.adj_ptr.p,
                                                             node_nnz.p);
        SVX_LAUNCH_CHECK();
    }
    P.node_base.alloc(ctx->pool, nn + 1);
    exclusive_scan_i64(ctx, node_nnz.p, P.node_base.p, nn);
    struct Sizes {
        int64_t n_adj, nnz;
        int flags[2];
    };
    Sizes* h = static_cast<Sizes*>(ctx->h_scalars);
    SVX_CUDA(cudaMemcpyAsync(&h->n_adj, P.adj_ptr.p + nn, sizeof(int64_t),
                             cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaMemcpyAsync(&h->nnz, P.node_base.p + nn, sizeof(int64_t),
                             cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaMemcpyAsync(h->flags, flags.p, sizeof(h->flags), cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaStreamSynchronize(st));
    const int64_t n_adj = h->n_adj, nnz = h->nnz;
    P.max_slots = h->flags[0];
    P.max_deg = h->flags[1];
    if (nnz >= int64_t(INT_MAX))
        throw ModelFail{SVX_OOM, 0, -1,
                        "stiffness has " + std::to_string(nnz) +
                            " nonzeros; the int32 CSR indices of the device path hold < 2^31"};
    if (P.max_deg > 65535)
        throw ModelFail{SVX_INVALID_MODEL, 0, -1,
                        "a node shares elements with more than 65535 nodes"};
    P.adj.alloc(ctx->pool, n_adj + 1);
    P.nnz = nnz;
    P.row_ptr.alloc(ctx->pool, P.n + 1);
    P.col_idx.alloc(ctx->pool, nnz + 1);
    P.diag_pos.alloc(ctx->pool, P.n + 1);
    // 4. and the element -> nonzero map, from the same list
    P.slot_map.alloc(ctx->pool, size_t(n_slots) * P.max_nn + 1);
    if (nn > 0) {
        auto* const kernel = op->ndof == 3   ? wide ? &rows_kernel<3, 32> : &rows_kernel<3, 8>
                             : op->ndof == 2 ? wide ? &rows_kernel<2, 32> : &rows_kernel<2, 8>
                             : wide          ? &rows_kernel<1, 32>
                                             : &rows_kernel<1, 8>;
        kernel<<<blocks_for(nn * lanes, 256), 256, 0, st>>>(
            nn, P.max_nn, P.slot_ptr.p, P.slot_elem.p, op->conn_ptr.p, op->conn.p, P.adj_ptr.p,
            P.adj.p, P.node_base.p, P.slot_map.p, P.row_ptr.p, P.col_idx.p, P.diag_pos.p);
        SVX_LAUNCH_CHECK();
    }
}

}  // namespace svx
