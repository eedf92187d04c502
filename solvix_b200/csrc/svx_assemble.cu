// svx_assemble.cu - K2 fixed-order assembly and K4 Dirichlet / Jacobi
// diagonal.
//
// K2 replaces scatter + csr_from_triplets (crates/solvix-core/src/
// assembly.rs:87-133) without triplets and without float atomics.  One warp
// owns one node: its ndof CSR rows are a contiguous block of
// ndof * ndof * deg values (the pattern is node adjacency x dense ndof
// blocks).  The warp walks the node's incident (element, local position)
// slots in ascending order and adds the element's ndof rows of Ke into a
// shared-memory copy of the block, each value landing at the position the
// precomputed element-to-nonzero map gives.  Every CSR value is therefore
//   0.0 + Ke_e1 + Ke_e2 + ...   in ascending element order,
// which is the reference's triplet-stream order (diagonal seed first, then
// elements in enumeration order): deterministic run to run, and bit-equal to
// the oracle's stable-order assembly.
//
// K4 replaces apply_dirichlet (solver.rs:45-62), the inverse diagonal of
// pcg (solver.rs:96-107) and jacobi_cond (lib.rs:634-644).  The rows of the
// unmodified K at constrained dofs are kept in a compact CSR for reactions
// (stress.rs:103-118) instead of cloning all of K (lib.rs:623-628).

#include "svx_internal.h"

#include <algorithm>
#include <cmath>

namespace svx {

namespace {

constexpr int ASM_WARPS = 8;

// The sums of one slot: rows (ND x NN ND) of the element's Ke onto the node's
// block, the lanes of its group one value each.
template <int ND, int NN, int G>
__device__ __forceinline__ void add_rows(double* acc, int rowlen, const uint16_t* map,
                                         const double* rows, int gl) {
    constexpr int N = NN * ND;
#pragma unroll
    for (int t0 = 0; t0 < ND * N; t0 += G) {
        const int t = t0 + gl;
        if (ND * N % G != 0 && t >= ND * N) break;
        const int da = t / N, col = t - da * N, c = col / ND, db = col - c * ND;
        acc[da * rowlen + int(map[c]) * ND + db] += rows[t];
    }
}

// G lanes a node: a warp for plane and solid rows, eight lanes for one dof a
// node (an element's row is at most eight values then; a warp a node left 24
// lanes idle: 899 us for the 240 x 24 x 24 conduction block, 92 now).  Whether an
// element repeats a node is found by one match over its map (reading the map
// pair by pair was most of this kernel's loads; with the sizes of an element
// known at compile time the 160 x 16 x 16 solid assembles in 1.37 ms instead of
// 1.56, the 40 solids of a batch in 8.2 instead of 9.7).
template <int ND>
__global__ void __launch_bounds__(ASM_WARPS * 32)
assemble_kernel(int64_t n_nodes, int max_nn, int acc_stride,
                const int64_t* __restrict__ slot_ptr, const int32_t* __restrict__ slot_elem,
                const uint8_t* __restrict__ slot_local, const uint16_t* __restrict__ slot_map,
                const int64_t* __restrict__ conn_ptr, const int64_t* __restrict__ adj_ptr,
                const int64_t* __restrict__ node_base, const double* __restrict__ ke,
                int ke_stride, double* __restrict__ vals) {
    constexpr int G = ND == 1 ? 8 : 32, PER = 32 / G;
    extern __shared__ double acc_all[];
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), grp = lane / G;
    const int w = threadIdx.x >> 5;
    double* acc = acc_all + size_t(w * PER + grp) * acc_stride;
    const int warps = int(blockDim.x) >> 5;
    const int64_t step = int64_t(gridDim.x) * warps * PER;
    for (int64_t i0 = (int64_t(blockIdx.x) * warps + w) * PER; i0 < n_nodes; i0 += step) {
        const int64_t i = i0 + grp;
        const bool node = i < n_nodes;
        const int64_t deg = node ? adj_ptr[i + 1] - adj_ptr[i] : 0;
        const int64_t base = node ? node_base[i] : 0;
        if (node && deg == 0 && gl < ND) vals[base + gl] = 0.0;  // only the diagonal seeds
        const int rowlen = int(ND * deg);
        const int total = ND * rowlen;
        for (int q = gl; q < total; q += G) acc[q] = 0.0;
        const int64_t s0 = deg > 0 ? slot_ptr[i] : 0;
        const int slots = deg > 0 ? int(slot_ptr[i + 1] - s0) : 0;
        const int most = PER == 1 ? slots : __reduce_max_sync(0xffffffffu, slots);
        __syncwarp();
        for (int k = 0; k < most; ++k) {
            const bool on = k < slots;
            const int64_t s = s0 + k;
            const int64_t e = on ? slot_elem[s] : 0;
            const int a = on ? slot_local[s] : 0;
            const int nn = on ? int(conn_ptr[e + 1] - conn_ptr[e]) : 0;
            const int N = nn * ND;
            const uint16_t* map = slot_map + s * max_nn;
            const double* rows = ke + e * int64_t(ke_stride) + int64_t(a) * ND * N;
            // an element that repeats a node maps two columns to one target
            const unsigned key = gl < nn ? (unsigned(grp) << 16 | map[gl]) : 0x80000000u | lane;
            const unsigned same = __match_any_sync(0xffffffffu, key);
            const unsigned twice = __ballot_sync(0xffffffffu, (same & (same - 1)) != 0);
            const unsigned mine = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (grp * G);
            if (!(twice & mine)) {
                if (nn == 8) add_rows<ND, 8, G>(acc, rowlen, map, rows, gl);
                else if (nn == 4) add_rows<ND, 4, G>(acc, rowlen, map, rows, gl);
                else if (nn == 3) add_rows<ND, 3, G>(acc, rowlen, map, rows, gl);
                else
                    for (int t = gl; t < ND * N; t += G) {
                        const int da = t / N, col = t - da * N, c = col / ND, db = col - c * ND;
                        acc[da * rowlen + int(map[c]) * ND + db] += rows[t];
                    }
            } else if (gl == 0) {
                for (int t = 0; t < ND * N; ++t) {
                    const int da = t / N, col = t - da * N, c = col / ND, db = col - c * ND;
                    acc[da * rowlen + int(map[c]) * ND + db] += rows[t];
                }
            }
            __syncwarp();
        }
        for (int q = gl; q < total; q += G) vals[base + q] = acc[q];
        __syncwarp();
    }
}

__global__ void mark_fixed_kernel(int64_t n_fixed, const int64_t* __restrict__ rows,
                                  uint8_t* __restrict__ is_fixed) {
    int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < n_fixed) is_fixed[rows[k]] = 1;
}

// Row lengths of the compact constrained rows.
// ptr[0..m]: exclusive sums of the rows' lengths; one block.
__global__ void __launch_bounds__(1024)
fixed_ptr_kernel(int64_t m, const int64_t* __restrict__ rows, const int32_t* __restrict__ row_ptr,
                 int32_t* __restrict__ ptr) {
    __shared__ int32_t sums[1024];
    const int t = threadIdx.x;
    const int64_t per = (m + 1023) / 1024, k0 = min(m, per * t), k1 = min(m, k0 + per);
    int32_t own = 0;
    for (int64_t k = k0; k < k1; ++k) own += row_ptr[rows[k] + 1] - row_ptr[rows[k]];
    sums[t] = own;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const int32_t v = t >= off ? sums[t - off] : 0;
        __syncthreads();
        sums[t] += v;
        __syncthreads();
    }
    int32_t at = sums[t] - own;
    for (int64_t k = k0; k < k1; ++k) {
        ptr[k] = at;
        at += row_ptr[rows[k] + 1] - row_ptr[rows[k]];
    }
    if (t == 1023) ptr[m] = sums[1023];
}

// Copy the unmodified constrained rows (one warp per row).
__global__ void fixed_copy_kernel(int64_t m, const int64_t* __restrict__ rows,
                                  const int32_t* __restrict__ row_ptr,
                                  const int32_t* __restrict__ col_idx,
                                  const double* __restrict__ vals,
                                  const int32_t* __restrict__ kc_ptr, int32_t* __restrict__ kc_col,
                                  double* __restrict__ kc_val) {
    int64_t k = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (k >= m) return;
    int32_t a = row_ptr[rows[k]], len = row_ptr[rows[k] + 1] - a;
    int32_t o = kc_ptr[k];
    for (int j = lane; j < len; j += 32) {
        kc_col[o + j] = col_idx[a + j];
        kc_val[o + j] = vals[a + j];
    }
}

// Symmetric elimination: an entry dies if its row or column is constrained;
// a constrained diagonal becomes 1 (one warp per row).
__global__ void dirichlet_kernel(int64_t n, const int32_t* __restrict__ row_ptr,
                                 const int32_t* __restrict__ col_idx,
                                 const uint8_t* __restrict__ is_fixed, double* __restrict__ vals,
                                 double* __restrict__ f) {
    int64_t r = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (r >= n) return;
    const bool fr = is_fixed[r] != 0;
    for (int32_t j = row_ptr[r] + lane; j < row_ptr[r + 1]; j += 32) {
        int32_t c = col_idx[j];
        if (fr || is_fixed[c]) vals[j] = (c == r) ? 1.0 : 0.0;
    }
    if (fr && lane == 0) f[r] = 0.0;
}

// inv_diag = 1/K_ii (0 when K_ii == 0) and the extreme |K_ii| per block.
__global__ void diag_kernel(int64_t n, const int32_t* __restrict__ diag_pos,
                            const double* __restrict__ vals, double* __restrict__ inv_diag,
                            double* __restrict__ block_hi, double* __restrict__ block_lo) {
    __shared__ double shi[256], slo[256];
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    double hi = 0.0, lo = INFINITY;
    if (i < n) {
        double d = vals[diag_pos[i]];
        inv_diag[i] = (d == 0.0) ? 0.0 : 1.0 / d;
        double a = fabs(d);
        hi = fmax(hi, a);
        lo = fmin(lo, a);
    }
    shi[threadIdx.x] = hi;
    slo[threadIdx.x] = lo;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) {
            shi[threadIdx.x] = fmax(shi[threadIdx.x], shi[threadIdx.x + off]);
            slo[threadIdx.x] = fmin(slo[threadIdx.x], slo[threadIdx.x + off]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        block_hi[blockIdx.x] = shi[0];
        block_lo[blockIdx.x] = slo[0];
    }
}

// out[0], out[1]: the largest and the smallest of the blocks' extremes (0 and
// infinity without blocks).
__global__ void __launch_bounds__(256)
extremes_kernel(int64_t nb, const double* hi, const double* lo, double* out) {
    __shared__ double shi[256], slo[256];
    double h = 0.0, l = INFINITY;
    for (int64_t k = threadIdx.x; k < nb; k += 256) {
        h = fmax(h, hi[k]);
        l = fmin(l, lo[k]);
    }
    shi[threadIdx.x] = h;
    slo[threadIdx.x] = l;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (threadIdx.x < off) {
            shi[threadIdx.x] = fmax(shi[threadIdx.x], shi[threadIdx.x + off]);
            slo[threadIdx.x] = fmin(slo[threadIdx.x], slo[threadIdx.x + off]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = shi[0];
        out[1] = slo[0];
    }
}

inline unsigned blocks_for(int64_t n, int t) { return unsigned((n + t - 1) / t); }

}  // namespace

void assemble_values(svx_ctx* ctx, svx_op* op, const double* ke, int ke_stride, double* vals) {
    const Pattern& P = op->pat;
    if (op->n_nodes == 0) return;
    const int acc_stride = op->ndof * op->ndof * std::max(1, P.max_deg);
    const int per = op->ndof == 1 ? 4 : 1;  // nodes a warp
    if (size_t(ASM_WARPS) * acc_stride * sizeof(double) > 200 * 1024)
        throw ModelFail{SVX_INVALID_MODEL, 0, -1,
                        "node degree " + std::to_string(P.max_deg) +
                            " exceeds the shared-memory block of the assembly kernel"};
    int warps = ASM_WARPS;  // fewer where four nodes a warp of a large degree need the room
    while (warps > 1 && size_t(warps) * per * acc_stride * sizeof(double) > 200 * 1024) warps /= 2;
    const size_t smem = size_t(warps) * per * acc_stride * sizeof(double);
    auto* const kernel = op->ndof == 3   ? &assemble_kernel<3>
                         : op->ndof == 2 ? &assemble_kernel<2>
                                         : &assemble_kernel<1>;
    if (smem > 48 * 1024)
        SVX_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    int64_t blocks = (op->n_nodes + warps * per - 1) / (warps * per);
    int64_t cap = int64_t(ctx->sm_count) * 32;
    if (blocks > cap) blocks = cap;
    kernel<<<unsigned(blocks), warps * 32, smem, ctx->stream>>>(
        op->n_nodes, P.max_nn, acc_stride, P.slot_ptr.p, P.slot_elem.p, P.slot_local.p,
        P.slot_map.p, op->conn_ptr.p, P.adj_ptr.p, P.node_base.p, ke, ke_stride, vals);
    SVX_LAUNCH_CHECK();
}

void apply_dirichlet(svx_ctx* ctx, svx_op* op) {
    cudaStream_t st = ctx->stream;
    const Pattern& P = op->pat;
    const int64_t n = op->n;
    op->is_fixed.alloc(ctx->pool, n + 1);
    SVX_CUDA(cudaMemsetAsync(op->is_fixed.p, 0, n + 1, st));
    if (op->n_fixed > 0) {
        mark_fixed_kernel<<<blocks_for(op->n_fixed, 256), 256, 0, st>>>(
            op->n_fixed, op->fixed_row.p, op->is_fixed.p);
        SVX_LAUNCH_CHECK();
    }
    // compact copy of the constrained rows of the unmodified K (fixed_uniq and
    // fixed_slot were uploaded with the model)
    const int64_t m = op->n_fixed_rows;
    if (m > 0) {
        op->kc_ptr.alloc(ctx->pool, m + 1);
        fixed_ptr_kernel<<<1, 1024, 0, st>>>(m, op->fixed_uniq.p, P.row_ptr.p, op->kc_ptr.p);
        SVX_LAUNCH_CHECK();
        // room for every row at the largest degree, where that is small (12 MB),
        // saves the wait for the rows' own total
        int64_t room = m * int64_t(op->ndof) * std::max(1, P.max_deg);
        if (room > (int64_t(1) << 20)) {
            int32_t total = 0;
            SVX_CUDA(cudaMemcpyAsync(&total, op->kc_ptr.p + m, sizeof(total),
                                     cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
            room = total;
        }
        op->kc_col.alloc(ctx->pool, size_t(room) + 1);
        op->kc_val.alloc(ctx->pool, size_t(room) + 1);
        fixed_copy_kernel<<<blocks_for(m * 32, 256), 256, 0, st>>>(
            m, op->fixed_uniq.p, P.row_ptr.p, P.col_idx.p, op->vals.p, op->kc_ptr.p,
            op->kc_col.p, op->kc_val.p);
        SVX_LAUNCH_CHECK();
    }
    // f_orig keeps the unmodified loads; f gets the eliminated copy
    op->f.alloc(ctx->pool, n + 1);
    SVX_CUDA(cudaMemcpyAsync(op->f.p, op->f_orig.p, n * sizeof(double), cudaMemcpyDeviceToDevice,
                             st));
    if (n > 0) {
        dirichlet_kernel<<<blocks_for(n * 32, 256), 256, 0, st>>>(
            n, P.row_ptr.p, P.col_idx.p, op->is_fixed.p, op->vals.p, op->f.p);
        SVX_LAUNCH_CHECK();
    }
    jacobi_diagonal(ctx, op);
}

// Jacobi inverse diagonal and cond estimate of the modified K
void jacobi_diagonal(svx_ctx* ctx, svx_op* op) {
    cudaStream_t st = ctx->stream;
    const Pattern& P = op->pat;
    const int64_t n = op->n;
    op->inv_diag.alloc(ctx->pool, n + 1);
    const int64_t nb = (n + 255) / 256;
    DBuf<double> bhi, blo;
    bhi.alloc(ctx->pool, nb + 1);
    blo.alloc(ctx->pool, nb + 2);  // and the extremes of all blocks
    if (n > 0) {
        diag_kernel<<<unsigned(nb), 256, 0, st>>>(n, P.diag_pos.p, op->vals.p, op->inv_diag.p,
                                                  bhi.p, blo.p);
        SVX_LAUNCH_CHECK();
    }
    double* h = reinterpret_cast<double*>(static_cast<char*>(ctx->h_scalars) + svx_ctx::H_DIAG);
    extremes_kernel<<<1, 256, 0, st>>>(nb, bhi.p, blo.p, blo.p + nb);
    SVX_LAUNCH_CHECK();
    SVX_CUDA(cudaMemcpyAsync(h, blo.p + nb, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
}

void jacobi_condition(svx_ctx* ctx, svx_op* op) {
    const double* h = reinterpret_cast<const double*>(static_cast<const char*>(ctx->h_scalars) +
                                                      svx_ctx::H_DIAG);
    op->cond_estimate = h[0] / h[1];
}

}  // namespace svx
