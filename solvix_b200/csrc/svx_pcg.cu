// svx_pcg.cu - K5 SpMV, K6 fused PCG vector kernels, the persistent PCG
// kernels, K7 mixed precision and K8 batched PCG.
//
// The plain form restates solver::pcg_with_threads
// (crates/solvix-core/src/solver.rs:82-149) on the device:
//   per iteration  q = K p ; pap = p.q
//                  alpha = rz / pap ; u += alpha p ; r -= alpha q ;
//                  rr = r.r ; z = r * inv_diag ; rz' = r.z
//                  beta = rz' / rz ; p = z + beta p
// with the same stopping rule (||r|| / ||f|| <= tol, checked after the r
// update; pap <= 0 or NaN is a breakdown) and the same iteration count
// semantics.  Every reduction is deterministic: fixed launch geometry,
// warp-shuffle then shared-memory trees inside a block, and either the last
// block to finish (atomic ticket) or every block after a grid barrier sums
// the per-block partials in index order.
//
// Ways to run an iteration, the first that applies:
//  * plane FP64 models that fit on a cluster: K in its registers
//    (svx_resident.cu);
//  * FP64 C3D8 models from 14,000 nodes (180 as batch members): element by
//    element, in a persistent kernel on bricks of elements (svx_brick.cu) or
//    in the graph form (svx_hex.cu);
//  * the persistent cooperative kernels (systems whose K fits in the L2): one
//    launch runs up to `persistent_chunk` whole iterations, its blocks
//    meeting at bounded grid barriers; one dof a node has its own
//    (pcg_scalar_kernel);
//  * the CUDA-graph form (larger systems): the standalone node-block SpMV
//    (spmv_node_dot), update and p_update kernels, `check_every` iterations
//    per graph launch; kernels return at once after the device status
//    leaves RUNNING, and the host reads the status once per graph launch;
//  * the batched kernels: one CTA, or one 8-CTA cluster, per model.
//
// SpMV layout: K is stored in node blocks (a node's ndof rows over its
// sorted neighbours, contiguous); G lanes own one node and split its
// neighbour blocks, each lane loading one column index, ndof x values and
// ndof^2 K values, all independent of each other; the x gathers go through
// L1/L2 and the lanes combine with shuffles.  The CSR kernels further down
// serve the allocation-free entry point, which takes a caller's CSR.

#include "svx_internal.h"
#include "svx_grid.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

namespace svx {

namespace {

constexpr int BLOCK = 256;
// Resident blocks per SM the node-block SpMV kernels are compiled for; their
// grids are exactly one wave of that many blocks per SM.
constexpr int NODE_BLOCKS_PER_SM = 5;
// The same for the quad-layout FP32 SpMV (ND*ND float4 values a lane).
#ifndef SVX_SPMV32Q_BPS
#define SVX_SPMV32Q_BPS 3
#endif
constexpr int SPMV32Q_BLOCKS_PER_SM = SVX_SPMV32Q_BPS;
// Resident threads per SM the batched kernels are compiled for: 1,024 (at
// most 64 registers a thread) for 3D members, 1,536 for the lighter 2D ones,
// to keep enough node gathers in flight.
constexpr int BATCH_MIN_THREADS = 1024;
// The relative residual below which the mixed forms switch from the FP64 to
// the FP32 operator: tol over the FP32 operator's relative error (~1e-7),
// within [tol, 0.1]; 1e-3 at the reference's tol of 1e-10.
__host__ __device__ inline double mixed_switch_residual(double tol) {
    const double t = tol * 1e7;
    return t < tol ? tol : (t > 0.1 ? 0.1 : t);
}

// ------------------------------------------------------------ reductions
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Block sum of one value (all threads get the result).
__device__ __forceinline__ double block_sum(double v, double* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
    if (w == 0) t = warp_sum(t);
    if (threadIdx.x == 0) sh[0] = t;
    __syncthreads();
    double r = sh[0];
    __syncthreads();
    return r;
}

// Publishes a block partial; returns true in exactly one block (the last
// to arrive), after which that block can read every partial.
__device__ __forceinline__ bool last_block(unsigned int* counter) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int t = atomicAdd(counter, 1u);
        is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// Fixed-order sum of partials[0..n) by one block.
__device__ __forceinline__ double sum_partials(const double* partials, int n, double* sh) {
    double v = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) v += ((volatile const double*)partials)[k];
    return block_sum(v, sh);
}

// ------------------------------------------------------------ kernels
template <int G, class V>
__device__ __forceinline__ double row_dot(const int32_t* __restrict__ col_idx,
                                          const V* __restrict__ vals, const V* __restrict__ x,
                                          int32_t a, int32_t b, int gl) {
    double acc0 = 0.0, acc1 = 0.0;
    int32_t j = a + gl;
    for (; j + G < b; j += 2 * G) {
        int32_t c0 = __ldg(col_idx + j), c1 = __ldg(col_idx + j + G);
        double v0 = double(__ldg(vals + j)), v1 = double(__ldg(vals + j + G));
        acc0 += v0 * double(x[c0]);
        acc1 += v1 * double(x[c1]);
    }
    if (j < b) acc0 += double(__ldg(vals + j)) * double(x[__ldg(col_idx + j)]);
    return acc0 + acc1;
}

// First row of this warp's 32/G row groups in the block-strided loop; it is
// the same for all lanes of the warp.
template <int G>
__device__ __forceinline__ int64_t warp_first_row(int64_t groups_per_block) {
    return int64_t(blockIdx.x) * groups_per_block + int64_t(threadIdx.x >> 5) * (32 / G);
}

// q = K p and per-block partial of p.q; the last block forms pap and alpha.
template <int G, class V>
__global__ void __launch_bounds__(BLOCK)
spmv_dot_kernel(int64_t n, const int32_t* __restrict__ row_ptr,
                const int32_t* __restrict__ col_idx, const V* __restrict__ vals,
                const V* __restrict__ p, V* __restrict__ q, double* __restrict__ partials,
                PcgScalars* __restrict__ s) {
    __shared__ double sh[32];
    if (s->status != PCG_RUNNING) return;
    const int gl = threadIdx.x & (G - 1);
    const int64_t groups_per_block = BLOCK / G;
    double dot = 0.0;
    // warp-uniform trip count: every lane reaches the shuffles together
    for (int64_t rb = warp_first_row<G>(groups_per_block); rb < n;
         rb += int64_t(gridDim.x) * groups_per_block) {
        const int64_t r = rb + ((threadIdx.x & 31) / G);
        const bool valid = r < n;
        double v = valid ? row_dot<G, V>(col_idx, vals, p, row_ptr[r], row_ptr[r + 1], gl) : 0.0;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (valid && gl == 0) {
            V qv = V(v);
            q[r] = qv;
            dot += double(p[r]) * double(qv);
        }
    }
    double bs = block_sum(dot, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    if (last_block(&s->count_a)) {
        double pap = sum_partials(partials, gridDim.x, sh);
        if (threadIdx.x == 0) {
            s->count_a = 0;
            s->pap = pap;
            if (pap <= 0.0 || isnan(pap)) {
                s->status = PCG_BREAKDOWN;
                s->it = s->it + 1;
                s->res = sqrt(s->rr) / s->bnorm;
            } else {
                s->alpha = s->rz / pap;
            }
        }
    }
}


// ------------------------------------------------------------ node-block SpMV
// The pattern is node adjacency x dense ndof blocks, so the ND rows of node i
// share one column list: adj[adj_ptr[i] .. adj_ptr[i+1]).  These kernels read
// the column of each ND x ND block once from adj (4 B per block instead of
// 4 B per nonzero) and the values in the CSR order of the node's rows:
//   y[i*ND + da] = sum_k sum_db vals[node_base[i] + da*ND*d + k*ND + db]
//                                * x[adj[k]*ND + db]
// G lanes own one node and split its d blocks; lane k loads one index, ND
// x values and ND*ND matrix values, all independent of each other.
// M = float is the difference-form FP32 operator (compensated_fp32_kernel):
// every neighbour but the node itself multiplies x_j - x_i.
template <int ND, int G, class M, class V>
__device__ __forceinline__ void node_rows(const int64_t* __restrict__ adj_ptr,
                                          const int32_t* __restrict__ adj,
                                          const int64_t* __restrict__ node_base,
                                          const M* __restrict__ vals, const V* __restrict__ x,
                                          int64_t i, int gl, double* acc) {
    const int64_t a0 = adj_ptr[i];
    const int d = int(adj_ptr[i + 1] - a0);
    const M* __restrict__ v = vals + node_base[i];
    if (d == 0) {  // an unreferenced node: rows of length 1 (the diagonal)
        if (gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = double(v[da]) * double(x[i * ND + da]);
        return;
    }
    const int rowlen = ND * d;
    constexpr bool DIFF = std::is_same<M, float>::value;
    double xi[ND];
    if constexpr (DIFF) {
#pragma unroll
        for (int db = 0; db < ND; ++db) xi[db] = double(x[i * ND + db]);
    }
    for (int k = gl; k < d; k += G) {
        const int32_t j = __ldg(adj + a0 + k);
        const int64_t c = int64_t(j) * ND;
        double xv[ND];
#pragma unroll
        for (int db = 0; db < ND; ++db) xv[db] = double(x[c + db]);
        if constexpr (DIFF) {
            if (j != int32_t(i))
#pragma unroll
                for (int db = 0; db < ND; ++db) xv[db] -= xi[db];
        }
#pragma unroll
        for (int da = 0; da < ND; ++da)
#pragma unroll
            for (int db = 0; db < ND; ++db)
                acc[da] += double(__ldg(v + da * rowlen + k * ND + db)) * xv[db];
    }
}

template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// q = K p (node blocks) and the per-block partial of p.q; the last block
// forms pap and alpha exactly like spmv_dot_kernel.
template <int ND, int G, class M, class V>
__global__ void __launch_bounds__(BLOCK, NODE_BLOCKS_PER_SM)
spmv_node_dot_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                     const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                     const M* __restrict__ vals, const V* __restrict__ p, V* __restrict__ q,
                     double* __restrict__ partials, PcgScalars* __restrict__ s) {
    __shared__ double sh[32];
    if (s->status != PCG_RUNNING) return;
    const int gl = threadIdx.x & (G - 1);
    const int64_t nodes_per_block = BLOCK / G;
    double dot = 0.0;
    for (int64_t nb = warp_first_row<G>(nodes_per_block); nb < n_nodes;
         nb += int64_t(gridDim.x) * nodes_per_block) {
        const int64_t i = nb + ((threadIdx.x & 31) / G);
        double acc[ND];
#pragma unroll
        for (int da = 0; da < ND; ++da) acc[da] = 0.0;
        if (i < n_nodes) node_rows<ND, G, M, V>(adj_ptr, adj, node_base, vals, p, i, gl, acc);
#pragma unroll
        for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
        if (i < n_nodes && gl == 0) {
#pragma unroll
            for (int da = 0; da < ND; ++da) {
                V qv = V(acc[da]);
                q[i * ND + da] = qv;
                dot += double(p[i * ND + da]) * double(qv);
            }
        }
    }
    double bs = block_sum(dot, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    if (last_block(&s->count_a)) {
        double pap = sum_partials(partials, gridDim.x, sh);
        if (threadIdx.x == 0) {
            s->count_a = 0;
            s->pap = pap;
            if (pap <= 0.0 || isnan(pap)) {
                s->status = PCG_BREAKDOWN;
                s->it = s->it + 1;
                s->res = sqrt(s->rr) / s->bnorm;
            } else {
                s->alpha = s->rz / pap;
            }
        }
    }
}

// y = K x (FP64, node blocks).
template <int ND, int G>
__global__ void __launch_bounds__(BLOCK, NODE_BLOCKS_PER_SM)
spmv_node_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                 const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                 const double* __restrict__ vals, const double* __restrict__ x,
                 double* __restrict__ y) {
    const int gl = threadIdx.x & (G - 1);
    const int64_t nodes_per_block = BLOCK / G;
    for (int64_t nb = warp_first_row<G>(nodes_per_block); nb < n_nodes;
         nb += int64_t(gridDim.x) * nodes_per_block) {
        const int64_t i = nb + ((threadIdx.x & 31) / G);
        double acc[ND];
#pragma unroll
        for (int da = 0; da < ND; ++da) acc[da] = 0.0;
        if (i < n_nodes)
            node_rows<ND, G, double, double>(adj_ptr, adj, node_base, vals, x, i, gl, acc);
#pragma unroll
        for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
        if (i < n_nodes && gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) y[i * ND + da] = acc[da];
    }
}

// ------------------------------------------------------------ compensated residual
// The true residual r = f - K u of a nearly converged solve is a difference
// of two nearly equal sums: in plain FP64 its rounding error is ~1e-16 of
// sum_j |K_ij u_j|, which on a stiff, high-contrast model is larger than
// tol ||f|| itself (about 2e-10 ||f|| on the 480 x 48 x 48 heterogeneous
// cantilever, so no iterate could ever pass a 1e-10 true-residual test).
// Here every product and every addition keeps its exact rounding error:
// the product's by a fused multiply-add (a x - fl(a x)), the sum's by
// Knuth's TwoSum, the running sum carried as an unevaluated pair hi + lo.
// The residual then comes out to ~1e-16 of its own size.  The explicit
// round-to-nearest intrinsics keep the compiler from contracting the pairs'
// arithmetic into fused operations.
__device__ __forceinline__ void dd_add(double& hi, double& lo, double b) {
    const double s = __dadd_rn(hi, b);
    const double bp = __dsub_rn(s, hi);
    const double e = __dadd_rn(__dsub_rn(hi, __dsub_rn(s, bp)), __dsub_rn(b, bp));
    hi = s;
    lo = __dadd_rn(lo, e);
}

__device__ __forceinline__ void dd_mul_add(double& hi, double& lo, double a, double x) {
    const double p = __dmul_rn(a, x);
    dd_add(hi, lo, p);
    lo = __dadd_rn(lo, __fma_rn(a, x, -p));
}

template <int G>
__device__ __forceinline__ void group_sum_dd(double& hi, double& lo) {
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
        const double oh = __shfl_xor_sync(0xffffffffu, hi, off);
        const double ol = __shfl_xor_sync(0xffffffffu, lo, off);
        dd_add(hi, lo, oh);
        lo = __dadd_rn(lo, ol);
    }
}

// f_i - (hi + lo): f_i and hi agree to a few bits near convergence, so the
// first difference is exact
__device__ __forceinline__ double dd_residual(double f, double hi, double lo) {
    return __dsub_rn(__dsub_rn(f, hi), lo);
}

// One node's rows of K u as pairs (hi, lo), G lanes splitting its neighbour
// blocks (the node-block layout, as node_rows); CG: u was written by other
// CTAs of the launch and is read from L2.
template <int ND, int G, bool CG>
__device__ __forceinline__ void node_rows_dd(const int64_t* __restrict__ adj_ptr,
                                             const int32_t* __restrict__ adj,
                                             const int64_t* __restrict__ node_base,
                                             const double* __restrict__ vals, const double* u,
                                             int64_t i, int gl, double* hi, double* lo) {
    const int64_t a0 = adj_ptr[i];
    const int d = int(adj_ptr[i + 1] - a0);
    const double* __restrict__ v = vals + node_base[i];
    auto ld = [&](int64_t c) { return CG ? __ldcg(u + c) : u[c]; };
    if (d == 0) {  // an unreferenced node: rows of length 1 (the diagonal)
        if (gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) dd_mul_add(hi[da], lo[da], v[da], ld(i * ND + da));
        return;
    }
    const int rowlen = ND * d;
    for (int k = gl; k < d; k += G) {
        const int64_t c = int64_t(__ldg(adj + a0 + k)) * ND;
        double xv[ND];
#pragma unroll
        for (int db = 0; db < ND; ++db) xv[db] = ld(c + db);
#pragma unroll
        for (int da = 0; da < ND; ++da)
#pragma unroll
            for (int db = 0; db < ND; ++db)
                dd_mul_add(hi[da], lo[da], __ldg(v + da * rowlen + k * ND + db), xv[db]);
    }
}

// r = f - K u (FP64, node blocks, compensated sums) and r.r, for the
// reliable updates of the mixed form and the defect correction.
template <int ND, int G>
__global__ void __launch_bounds__(BLOCK, NODE_BLOCKS_PER_SM)
residual_node_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                     const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                     const double* __restrict__ vals, const double* __restrict__ u,
                     const double* __restrict__ f, double* __restrict__ r,
                     double* __restrict__ partials, unsigned int* counter,
                     double* __restrict__ out_rr) {
    __shared__ double sh[32];
    const int gl = threadIdx.x & (G - 1);
    const int64_t nodes_per_block = BLOCK / G;
    double rr = 0.0;
    for (int64_t nb = warp_first_row<G>(nodes_per_block); nb < n_nodes;
         nb += int64_t(gridDim.x) * nodes_per_block) {
        const int64_t i = nb + ((threadIdx.x & 31) / G);
        double hi[ND], lo[ND];
#pragma unroll
        for (int da = 0; da < ND; ++da) hi[da] = lo[da] = 0.0;
        if (i < n_nodes)
            node_rows_dd<ND, G, false>(adj_ptr, adj, node_base, vals, u, i, gl, hi, lo);
#pragma unroll
        for (int da = 0; da < ND; ++da) group_sum_dd<G>(hi[da], lo[da]);
        if (i < n_nodes && gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) {
                const double ri = dd_residual(f[i * ND + da], hi[da], lo[da]);
                r[i * ND + da] = ri;
                rr += ri * ri;
            }
    }
    double b = block_sum(rr, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = b;
    if (last_block(counter)) {
        double t = sum_partials(partials, gridDim.x, sh);
        if (threadIdx.x == 0) {
            *counter = 0;
            *out_rr = t;
        }
    }
}

// u += alpha p ; r -= alpha q ; partials of r.r and r.z (z = r * inv_diag).
template <class V, class U>
__global__ void __launch_bounds__(BLOCK)
update_kernel(int64_t n, U* __restrict__ u, V* __restrict__ r, const V* __restrict__ p,
              const V* __restrict__ q, const V* __restrict__ inv_diag,
              double* __restrict__ partials, PcgScalars* __restrict__ s) {
    __shared__ double sh[32];
    if (s->status != PCG_RUNNING) return;
    const double alpha = s->alpha;
    const V a = V(alpha);
    double rr = 0.0, rz = 0.0;
    // the thread's elements i, i + S, i + 2S, ... in the order of a plain
    // grid-stride loop, two of them loaded before either is updated (more
    // loads in flight: 0.039 against 0.047 ms on 3.46M rows)
    constexpr int UN = 2;
    const int64_t S = int64_t(gridDim.x) * BLOCK;
    for (int64_t i0 = int64_t(blockIdx.x) * BLOCK + threadIdx.x; i0 < n; i0 += UN * S) {
        V pv[UN], qv[UN], rv[UN], dv[UN];
        U uv[UN];
#pragma unroll
        for (int t = 0; t < UN; ++t) {
            const int64_t i = i0 + t * S;
            if (i < n) {
                pv[t] = p[i];
                uv[t] = u[i];
                rv[t] = r[i];
                qv[t] = q[i];
                dv[t] = inv_diag[i];
            }
        }
#pragma unroll
        for (int t = 0; t < UN; ++t) {
            const int64_t i = i0 + t * S;
            if (i < n) {
                V pi = pv[t];
                u[i] = U(uv[t] + U(a) * U(pi));
                V ri = rv[t] - a * qv[t];
                r[i] = ri;
                V zi = ri * dv[t];
                rr += double(ri) * double(ri);
                rz += double(ri) * double(zi);
            }
        }
    }
    double brr = block_sum(rr, sh);
    double brz = block_sum(rz, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = brr;
        partials[2 * blockIdx.x + 1] = brz;
    }
    if (last_block(&s->count_b)) {
        double v0 = 0.0, v1 = 0.0;
        for (int k = threadIdx.x; k < int(gridDim.x); k += blockDim.x) {
            v0 += ((volatile double*)partials)[2 * k];
            v1 += ((volatile double*)partials)[2 * k + 1];
        }
        double trr = block_sum(v0, sh);
        double trz = block_sum(v1, sh);
        if (threadIdx.x == 0) {
            s->count_b = 0;
            s->it = s->it + 1;
            s->rr = trr;
            double res = sqrt(trr) / s->bnorm;
            s->res = res;
            if (res <= s->tol) {
                s->status = PCG_CONVERGED;
            } else if (s->it >= s->max_iter) {
                s->status = PCG_MAXITER;
            } else if (trr <= s->rr_stop) {
                s->status = PCG_RELIABLE;  // s->rz stays r.z of the previous iterate
            } else {
                s->beta = trz / s->rz;
                s->rz = trz;
            }
        }
    }
}

// p = z + beta p with z = r * inv_diag recomputed.
template <class V>
__global__ void __launch_bounds__(BLOCK)
p_update_kernel(int64_t n, V* __restrict__ p, const V* __restrict__ r,
                const V* __restrict__ inv_diag, const PcgScalars* __restrict__ s) {
    if (s->status != PCG_RUNNING) return;
    const V beta = V(s->beta);
    for (int64_t i = int64_t(blockIdx.x) * BLOCK + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * BLOCK)
        p[i] = r[i] * inv_diag[i] + beta * p[i];
}

// r = b ; u = 0 ; p = z = r * inv_diag ; partials of b.b and r.z.
template <class V, class B, class U = V>
__global__ void __launch_bounds__(BLOCK)
init_kernel(int64_t n, const B* __restrict__ b, double b_scale, U* __restrict__ u,
            V* __restrict__ r, V* __restrict__ p, const V* __restrict__ inv_diag,
            double* __restrict__ partials, PcgScalars* __restrict__ s) {
    __shared__ double sh[32];
    double bb = 0.0, rz = 0.0;
    for (int64_t i = int64_t(blockIdx.x) * BLOCK + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * BLOCK) {
        V ri = V(double(b[i]) * b_scale);
        u[i] = U(0);
        r[i] = ri;
        V zi = ri * inv_diag[i];
        p[i] = zi;
        bb += double(ri) * double(ri);
        rz += double(ri) * double(zi);
    }
    double bbb = block_sum(bb, sh);
    double brz = block_sum(rz, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = bbb;
        partials[2 * blockIdx.x + 1] = brz;
    }
    if (last_block(&s->count_c)) {
        double v0 = 0.0, v1 = 0.0;
        for (int k = threadIdx.x; k < int(gridDim.x); k += blockDim.x) {
            v0 += ((volatile double*)partials)[2 * k];
            v1 += ((volatile double*)partials)[2 * k + 1];
        }
        double tbb = block_sum(v0, sh);
        double trz = block_sum(v1, sh);
        if (threadIdx.x == 0) {
            s->count_c = 0;
            s->bnorm = sqrt(tbb);
            s->rr = tbb;
            s->rz = trz;
            s->it = 0;
            s->res = 0.0;
            s->status = (s->bnorm == 0.0) ? PCG_CONVERGED : PCG_RUNNING;
            if (s->bnorm != 0.0) s->res = 1.0;
        }
    }
}

// The FP32 operator of the mixed form.  Rounding each entry of K to FP32
// (relative error ~6e-8) breaks K's translation null space: for a smooth
// field x the product K x is the small difference of large terms, and the
// rounded operator's error eps32 * sum_j |K_ij| |x_j| swamps it on a
// slender, high-contrast model (the true residual of CG on that operator
// stalls near 1e-8).  The stored operator is therefore written in
// difference form around each node's own block:
//   (K x)_i = sum_{j != i} K_ij (x_j - x_i) + R_i x_i,   R_i = sum_j K_ij,
// an identity for any K.  Off-diagonal node blocks are stored as FP32 and
// the slot of the node's own block holds R_i (summed in FP64, then
// rounded), which vanishes in the interior of a free region.  The error of
// the stored operator becomes sum_{j != i} dK_ij (x_j - x_i) + dR_i x_i:
// it scales with the differences of x between neighbouring nodes instead of
// x itself, and a rigid translation is reproduced exactly.  The SpMV of
// this operator (node_rows_cg / node_rows_mv with M = float) subtracts x_i
// from every neighbour but the node itself.
template <int ND>
__global__ void compensated_fp32_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                                        const int32_t* __restrict__ adj,
                                        const int64_t* __restrict__ node_base,
                                        const double* __restrict__ vals,
                                        float* __restrict__ out) {
    const int64_t t = int64_t(blockIdx.x) * BLOCK + threadIdx.x;
    const int64_t i = t / (ND * ND);
    if (i >= n_nodes) return;
    const int da = int(t % (ND * ND)) / ND, db = int(t % ND);
    const int64_t a0 = adj_ptr[i];
    const int d = int(adj_ptr[i + 1] - a0);
    const int64_t base = node_base[i];
    if (d == 0) {  // an unreferenced node: its rows hold only the diagonal
        if (db == 0) out[base + da] = float(vals[base + da]);
        return;
    }
    const int64_t row = base + int64_t(da) * ND * d + db;
    double sum = 0.0;
    int self = -1;
    for (int k = 0; k < d; ++k) {
        const double v = vals[row + k * ND];
        sum += v;
        if (adj[a0 + k] == int32_t(i)) self = k;
        else out[row + k * ND] = float(v);
    }
    if (self >= 0) out[row + self * ND] = float(sum);
}



// vals (row da of node i, neighbour slot k, column db at node_base[i] +
// da ND d + k ND + db) -> valsT, the same values of each node with the slot
// fastest: (da ND + db) d + k.  One thread per (node, da, db); a node no
// element uses keeps its ND diagonal values in place.
template <int ND, class M>
__global__ void transpose_blocks_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                                        const int64_t* __restrict__ node_base,
                                        const M* __restrict__ vals, M* __restrict__ out) {
    const int64_t t = int64_t(blockIdx.x) * BLOCK + threadIdx.x;
    const int64_t i = t / (ND * ND);
    if (i >= n_nodes) return;
    const int e = int(t - i * (ND * ND)), da = e / ND, db = e - da * ND;
    const int d = int(adj_ptr[i + 1] - adj_ptr[i]);
    const int64_t base = node_base[i];
    if (d == 0) {
        if (db == 0) out[base + da] = vals[base + da];
        return;
    }
    const M* src = vals + base + int64_t(da) * ND * d + db;
    M* dst = out + base + int64_t(da * ND + db) * d;
    for (int k = 0; k < d; ++k) dst[k] = src[int64_t(k) * ND];
}

// ------------------------------------------------------------ quad FP32 operator
// vals32 (node-block layout) -> vals32q: node i's ND*ND (da, db) rows over
// its neighbour slots, slot fastest, each padded with zeros to dq =
// round_up(d, 4) slots (4 for a node no element uses, whose own slot holds
// its diagonal); adjq lists the node's neighbours padded with the node
// itself.  baseq[i] is node i's first value; its neighbour list starts at
// baseq[i] / (ND*ND).  Both are 16-byte aligned, so a lane reads four
// slots of one (da, db) row, or four neighbour indices, in one load.
template <int ND>
__global__ void quad_fp32_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                                 const int32_t* __restrict__ adj,
                                 const int64_t* __restrict__ node_base,
                                 const int64_t* __restrict__ baseq,
                                 const float* __restrict__ vals32, float* __restrict__ out,
                                 int32_t* __restrict__ adjq) {
    const int64_t t = int64_t(blockIdx.x) * BLOCK + threadIdx.x;
    const int64_t i = t / (ND * ND);
    if (i >= n_nodes) return;
    const int e = int(t - i * (ND * ND)), da = e / ND, db = e - da * ND;
    const int d = int(adj_ptr[i + 1] - adj_ptr[i]);
    const int dq = d == 0 ? 4 : (d + 3) & ~3;
    const int64_t q0 = baseq[i];
    float* dst = out + q0 + int64_t(e) * dq;
    if (d == 0) {
        for (int k = 0; k < 4; ++k)
            dst[k] = (k == 0 && da == db) ? vals32[node_base[i] + da] : 0.0f;
    } else {
        const float* src = vals32 + node_base[i] + int64_t(da) * ND * d + db;
        for (int k = 0; k < dq; ++k) dst[k] = k < d ? src[int64_t(k) * ND] : 0.0f;
    }
    if (e == 0) {
        int32_t* aq = adjq + q0 / (ND * ND);
        for (int k = 0; k < dq; ++k) aq[k] = k < d ? adj[adj_ptr[i] + k] : int32_t(i);
    }
}

// q = K32 p for the difference-form FP32 operator in the quad layout, and
// the block partial of p.q (the last block forms pap and alpha, as
// spmv_node_dot_kernel does).  Eight lanes per node, four nodes a warp:
// lane g takes the neighbour slots 4g .. 4g+3 (one pass for up to 32
// neighbour blocks), loads their four indices as one int4 and each of the
// node's ND*ND rows as one float4, gathers the four neighbours' p, and
// multiplies in FP64 with p_j - p_i (p_i for the node's own slot and the
// padding, whose values are zero).  Per lane ND*ND 16-byte value loads are
// in flight at once: four times the bytes of the node-block kernel's
// scalar loads, which leave the FP32 operator latency-bound.  A node's quad
// count is (baseq[i+1] - baseq[i]) / (4*ND*ND), and both offsets are loaded
// one node group ahead of their use, so each group's first dependent load
// is its values, not its offsets.
template <int ND, class V>
__global__ void __launch_bounds__(BLOCK, SPMV32Q_BLOCKS_PER_SM)
spmv32q_node_dot_kernel(int64_t n_nodes, const int64_t* __restrict__ baseq,
                        const int32_t* __restrict__ adjq, const float* __restrict__ vals32q,
                        const V* __restrict__ p, V* __restrict__ q,
                        double* __restrict__ partials, PcgScalars* __restrict__ s) {
    constexpr int G = 8;
    __shared__ double sh[32];
    if (s->status != PCG_RUNNING) return;
    const int gl = threadIdx.x & (G - 1);
    const int64_t nodes_per_block = BLOCK / G;
    const int64_t stride = int64_t(gridDim.x) * nodes_per_block;
    double dot = 0.0;
    int64_t nb = warp_first_row<G>(nodes_per_block);
    int64_t qa = 0, qb = 0;  // baseq[i], baseq[i + 1] of this lane's node
    {
        const int64_t i = nb + ((threadIdx.x & 31) / G);
        if (i < n_nodes) {
            qa = __ldg(baseq + i);
            qb = __ldg(baseq + i + 1);
        }
    }
    for (; nb < n_nodes; nb += stride) {
        const int64_t i = nb + ((threadIdx.x & 31) / G);
        const int64_t q0 = qa;
        const int dq4 = int(qb - qa) / (4 * ND * ND);
        if (i + stride < n_nodes) {
            qa = __ldg(baseq + i + stride);
            qb = __ldg(baseq + i + stride + 1);
        }
        double acc[ND];
#pragma unroll
        for (int da = 0; da < ND; ++da) acc[da] = 0.0;
        if (i < n_nodes) {
            const float4* v4 = reinterpret_cast<const float4*>(vals32q + q0);
            const int4* a4 = reinterpret_cast<const int4*>(adjq + q0 / (ND * ND));
            double xi[ND];
#pragma unroll
            for (int db = 0; db < ND; ++db) xi[db] = double(__ldg(p + i * ND + db));
            for (int c = gl; c < dq4; c += G) {
                const int4 jj = __ldg(a4 + c);
                float4 kv[ND * ND];
#pragma unroll
                for (int e = 0; e < ND * ND; ++e) kv[e] = __ldg(v4 + int64_t(e) * dq4 + c);
                const int32_t js[4] = {jj.x, jj.y, jj.z, jj.w};
                double xv[4][ND];
#pragma unroll
                for (int m = 0; m < 4; ++m)
#pragma unroll
                    for (int db = 0; db < ND; ++db) {
                        const double x = double(__ldg(p + int64_t(js[m]) * ND + db));
                        xv[m][db] = (js[m] != int32_t(i)) ? x - xi[db] : x;
                    }
#pragma unroll
                for (int da = 0; da < ND; ++da)
#pragma unroll
                    for (int db = 0; db < ND; ++db) {
                        const float4 k4 = kv[da * ND + db];
                        acc[da] += double(k4.x) * xv[0][db];
                        acc[da] += double(k4.y) * xv[1][db];
                        acc[da] += double(k4.z) * xv[2][db];
                        acc[da] += double(k4.w) * xv[3][db];
                    }
            }
        }
#pragma unroll
        for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
        if (i < n_nodes && gl == 0) {
#pragma unroll
            for (int da = 0; da < ND; ++da) {
                const V qv = V(acc[da]);
                q[i * ND + da] = qv;
                dot += double(__ldg(p + i * ND + da)) * double(qv);
            }
        }
    }
    double bs = block_sum(dot, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    if (last_block(&s->count_a)) {
        double pap = sum_partials(partials, gridDim.x, sh);
        if (threadIdx.x == 0) {
            s->count_a = 0;
            s->pap = pap;
            if (pap <= 0.0 || isnan(pap)) {
                s->status = PCG_BREAKDOWN;
                s->it = s->it + 1;
                s->res = sqrt(s->rr) / s->bnorm;
            } else {
                s->alpha = s->rz / pap;
            }
        }
    }
}


// ------------------------------------------------------------ persistent PCG
// One cooperative launch runs up to `chunk` whole PCG iterations.  Block b
// owns the nodes [n_nodes*b/B, n_nodes*(b+1)/B) for the SpMV and the rows of
// those nodes for the vector updates, so an iteration is
//   A: q = K p on own nodes, partial p.q          -> grid barrier
//   B: alpha; u, r update on own rows, partials    -> grid barrier
//   C: beta; p = z + beta p on own rows            -> grid barrier
// (3D models; 2D models run pcg_persistent2_kernel, which forms p inside A
// and needs only the first two barriers).
// Every block sums the same partials in the same order, so all blocks hold
// bitwise identical scalars and take the same exit (converged, breakdown,
// budget) without a broadcast.  Data written by other blocks during the
// launch (p, q, partials) is read with ld.global.cg (L2), never through L1.
// The barrier spins are bounded: on timeout the kernel raises an error flag
// and returns, and the host reports a device error.
// Persistent kernel shape (build constants): CTA size, CTAs per SM and lanes
// per node for 3D models (2D models use 16).  Measured on the 160x16x16
// C3D8 case (us per iteration): 512 x 2 with 32 lanes 34.9, with 16 lanes
// 39.2, with 8 lanes 36.6; 1024 x 1 35.6-37.5; 256 x 4 41.9; 256 x 6 47.7;
// 128 x 8 54.7 (more CTAs make every grid barrier dearer).  With the
// release/acquire barrier below: 512 x 2 with 32 lanes 30.5-30.7, with 16
// lanes 36.0; 1024 x 1 30.8; 256 x 4 33.4; a poll back-off of 0, 32 or
// 100 ns the same.
#ifndef SVX_PBLOCK
#define SVX_PBLOCK 512
#endif
#ifndef SVX_PBLOCKS_PER_SM
#define SVX_PBLOCKS_PER_SM 2
#endif
#ifndef SVX_PG3D
#define SVX_PG3D 32
#endif
constexpr int PBLOCK = SVX_PBLOCK;
constexpr int PBLOCKS_PER_SM = SVX_PBLOCKS_PER_SM;
// largest per-block shared adjacency copy of the persistent kernels (bytes;
// 0 keeps the adjacency in global memory)
#ifndef SVX_SHARED_ADJ_MAX
#define SVX_SHARED_ADJ_MAX (96 * 1024)
#endif
constexpr long long SHARED_ADJ_MAX = SVX_SHARED_ADJ_MAX;

// One node's rows given its d column node indices (cols: global memory,
// read through the read-only path, or shared memory when SCOLS) and its
// row block v.
template <int ND, int G, class M, class V, bool SCOLS, int UNROLL = 2>
__device__ __forceinline__ void node_rows_cg_at(const int32_t* cols, int d,
                                                const M* __restrict__ v, const V* x, int64_t i,
                                                int gl, double* acc) {
    if (d == 0) {
        if (gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = double(v[da]) * double(__ldcg(x + i * ND + da));
        return;
    }
    const int rowlen = ND * d;
    // FP32 operators are stored in difference form (compensated_fp32_kernel)
    constexpr bool DIFF = std::is_same<M, float>::value;
    double xi[ND];
    if constexpr (DIFF) {
#pragma unroll
        for (int db = 0; db < ND; ++db) xi[db] = double(__ldcg(x + i * ND + db));
    }
#pragma unroll UNROLL
    for (int k = gl; k < d; k += G) {
        const int32_t j = SCOLS ? cols[k] : __ldg(cols + k);
        const int64_t c = int64_t(j) * ND;
        double xv[ND];
#pragma unroll
        for (int db = 0; db < ND; ++db) xv[db] = double(__ldcg(x + c + db));
        if constexpr (DIFF) {
            if (j != int32_t(i))
#pragma unroll
                for (int db = 0; db < ND; ++db) xv[db] -= xi[db];
        }
#pragma unroll
        for (int da = 0; da < ND; ++da)
#pragma unroll
            for (int db = 0; db < ND; ++db)
                acc[da] += double(__ldg(v + da * rowlen + k * ND + db)) * xv[db];
    }
}

template <int ND, int G, class M, class V>
__device__ __forceinline__ void node_rows_cg(const int64_t* __restrict__ adj_ptr,
                                             const int32_t* __restrict__ adj,
                                             const int64_t* __restrict__ node_base,
                                             const M* __restrict__ vals, const V* x,
                                             int64_t i, int gl, double* acc) {
    const int64_t a0 = adj_ptr[i];
    node_rows_cg_at<ND, G, M, V, false>(adj + a0, int(adj_ptr[i + 1] - a0), vals + node_base[i],
                                        x, i, gl, acc);
}

// Fixed-order sum of n partials (stride `stride`, offset `off`) read from L2.
__device__ __forceinline__ double sum_partials_cg(const double* partials, int n, int stride,
                                                  int off, double* sh) {
    double v = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) v += __ldcg(partials + k * stride + off);
    return block_sum(v, sh);
}

// The three-barrier kernel (3D models).
// A persistent block's node range never changes during a launch, so its
// adjacency is copied once per launch into dynamic shared memory: the row
// block offsets (node_base), the column-offset prefix relative to the
// range's first node (nloc + 1 ints) and the column node indices.  Each
// node's SpMV then starts from shared memory instead of two dependent
// global loads before its x gathers.  The host sizes the buffer for
// nodes_cap = ceil(n_nodes / blocks) nodes of at most max_deg neighbours.
// Measured (us per iteration, same iterations and residuals): 160x16x16
// C3D8 30.5 -> 29.7, 200x20 CPS4 9.0 -> 8.9.
struct SharedAdj {
    const int64_t* vbase;
    const int32_t* aptr;
    const int32_t* cols;
};

__device__ __forceinline__ SharedAdj load_shared_adj_at(unsigned char* base,
                                                        const int64_t* __restrict__ adj_ptr,
                                                        const int32_t* __restrict__ adj,
                                                        const int64_t* __restrict__ node_base,
                                                        int64_t nb0, int64_t nb1,
                                                        int nodes_cap) {
    int64_t* vb = reinterpret_cast<int64_t*>(base);
    int32_t* ap = reinterpret_cast<int32_t*>(vb + nodes_cap);
    int32_t* cl = ap + nodes_cap + 1;
    const int nloc = int(nb1 - nb0);
    const int64_t a_start = adj_ptr[nb0];
    for (int t = threadIdx.x; t <= nloc; t += blockDim.x)
        ap[t] = int32_t(adj_ptr[nb0 + t] - a_start);
    for (int t = threadIdx.x; t < nloc; t += blockDim.x) vb[t] = node_base[nb0 + t];
    const int64_t cnt = adj_ptr[nb1] - a_start;
    for (int64_t t = threadIdx.x; t < cnt; t += blockDim.x) cl[t] = adj[a_start + t];
    __syncthreads();
    return SharedAdj{vb, ap, cl};
}

__device__ __forceinline__ SharedAdj load_shared_adj(const int64_t* __restrict__ adj_ptr,
                                                     const int32_t* __restrict__ adj,
                                                     const int64_t* __restrict__ node_base,
                                                     int64_t nb0, int64_t nb1, int nodes_cap) {
    extern __shared__ __align__(16) unsigned char svx_dyn_smem[];
    return load_shared_adj_at(svx_dyn_smem, adj_ptr, adj, node_base, nb0, nb1, nodes_cap);
}

__host__ __device__ inline size_t shared_adj_bytes(int64_t nodes_cap, int max_deg) {
    return size_t(nodes_cap) * 8 + size_t(nodes_cap + 1) * 4 +
           size_t(nodes_cap) * size_t(max_deg > 1 ? max_deg : 1) * 4;
}

template <int ND, int G, class M, class V, class U, bool SADJ>
__global__ void __launch_bounds__(PBLOCK, PBLOCKS_PER_SM)
pcg_persistent_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                      const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                      const M* __restrict__ vals, const V* __restrict__ inv_diag, U* u, V* r,
                      V* p, V* /*p2*/, V* q, double* part_a, double* part_b,
                      PcgScalars* s, GridBarrier* gb, int chunk, int nodes_cap) {
    __shared__ double sh[32];
    const unsigned int B = gridDim.x;
    unsigned int bar_target = 0;  // grid_sync's running arrival target
    const int64_t nb0 = n_nodes * int64_t(blockIdx.x) / B;
    const int64_t nb1 = n_nodes * int64_t(blockIdx.x + 1) / B;
    const int64_t r0 = nb0 * ND, r1 = nb1 * ND;
    volatile PcgScalars* vs = s;
    if (vs->status != PCG_RUNNING) return;
    SharedAdj sa{nullptr, nullptr, nullptr};
    if constexpr (SADJ) sa = load_shared_adj(adj_ptr, adj, node_base, nb0, nb1, nodes_cap);
    double rz = vs->rz, rr = vs->rr, res = vs->res;
    const double bnorm = vs->bnorm, tol = vs->tol, rr_stop = vs->rr_stop;
    long long it = vs->it;
    const long long max_iter = vs->max_iter;
    const int gl = threadIdx.x & (G - 1);
    const int64_t warp_nodes = 32 / G;
    const int64_t step = int64_t(PBLOCK / 32) * warp_nodes;
    const bool writer = (blockIdx.x == 0 && threadIdx.x == 0);
    for (int c = 0; c < chunk; ++c) {
        // A: q = K p on own nodes, p.q
        double dot = 0.0;
        for (int64_t nb = nb0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < nb1; nb += step) {
            const int64_t i = nb + ((threadIdx.x & 31) / G);
            double acc[ND];
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = 0.0;
            if (i < nb1) {
                if constexpr (SADJ) {
                    const int li = int(i - nb0);
                    const int a0 = sa.aptr[li];
                    node_rows_cg_at<ND, G, M, V, true>(sa.cols + a0, sa.aptr[li + 1] - a0,
                                                       vals + sa.vbase[li], p, i, gl, acc);
                } else {
                    node_rows_cg<ND, G, M, V>(adj_ptr, adj, node_base, vals, p, i, gl, acc);
                }
            }
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
            if (i < nb1 && gl == 0) {
#pragma unroll
                for (int da = 0; da < ND; ++da) {
                    V qv = V(acc[da]);
                    q[i * ND + da] = qv;
                    dot += double(__ldcg(p + i * ND + da)) * double(qv);
                }
            }
        }
        double bs = block_sum(dot, sh);
        if (threadIdx.x == 0) part_a[blockIdx.x] = bs;
        if (!grid_sync(gb, B, bar_target)) return;
        const double pap = sum_partials_cg(part_a, int(B), 1, 0, sh);
        if (!(pap > 0.0)) {  // pap <= 0 or NaN: breakdown
            if (writer) {
                s->pap = pap;
                s->it = it + 1;
                s->res = sqrt(rr) / bnorm;
                s->rr = rr;
                s->rz = rz;
                __threadfence();
                s->status = PCG_BREAKDOWN;
            }
            return;
        }
        const double alpha = rz / pap;
        // B: u += alpha p, r -= alpha q on own rows; r.r, r.z
        const V a = V(alpha);
        double lrr = 0.0, lrz = 0.0;
        for (int64_t row = r0 + threadIdx.x; row < r1; row += PBLOCK) {
            const V pi = __ldcg(p + row);
            u[row] = U(u[row] + U(a) * U(pi));
            const V ri = __ldcg(r + row) - a * __ldcg(q + row);
            r[row] = ri;
            const V zi = ri * inv_diag[row];
            lrr += double(ri) * double(ri);
            lrz += double(ri) * double(zi);
        }
        const double brr = block_sum(lrr, sh);
        const double brz = block_sum(lrz, sh);
        if (threadIdx.x == 0) {
            part_b[2 * blockIdx.x] = brr;
            part_b[2 * blockIdx.x + 1] = brz;
        }
        if (!grid_sync(gb, B, bar_target)) return;
        const double rr_new = sum_partials_cg(part_b, int(B), 2, 0, sh);
        const double rz_new = sum_partials_cg(part_b, int(B), 2, 1, sh);
        it += 1;
        rr = rr_new;
        res = sqrt(rr) / bnorm;
        if (res <= tol || it >= max_iter || rr <= rr_stop) {
            if (writer) {
                s->it = it;
                s->res = res;
                s->rr = rr;
                s->rz = rz;         // r.z of the previous iterate (beta's denominator)
                s->pap = rz_new;    // r.z of this iterate
                s->alpha = alpha;
                __threadfence();
                s->status = (res <= tol) ? PCG_CONVERGED
                                         : (it >= max_iter ? PCG_MAXITER : PCG_RELIABLE);
            }
            return;
        }
        const double beta = rz_new / rz;
        rz = rz_new;
        // C: p = z + beta p on own rows
        const V bt = V(beta);
        for (int64_t row = r0 + threadIdx.x; row < r1; row += PBLOCK)
            p[row] = __ldcg(r + row) * inv_diag[row] + bt * __ldcg(p + row);
        if (!grid_sync(gb, B, bar_target)) return;
    }
    if (writer) {
        s->it = it;
        s->res = res;
        s->rr = rr;
        s->rz = rz;
    }
}

// Node rows of the persistent kernel with the search direction formed on
// the fly: x_j = r_j * inv_diag_j + beta * pprev_j (p of this iteration,
// from the previous p, this iteration's r and beta), so no pass and no grid
// barrier is spent writing p before the SpMV reads it.
template <int ND, int G, class M, class V, bool SCOLS>
__device__ __forceinline__ void node_rows_pp_at(const int32_t* cols, int d,
                                                const M* __restrict__ v, const V* r,
                                                const V* __restrict__ inv_diag, const V* pprev,
                                                V bprev, int64_t i, int gl, double* acc) {
    auto pdir = [&](int64_t row) -> double {
        return double(__ldcg(r + row) * __ldg(inv_diag + row) + bprev * __ldcg(pprev + row));
    };
    if (d == 0) {
        if (gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = double(v[da]) * pdir(i * ND + da);
        return;
    }
    const int rowlen = ND * d;
    // FP32 operators are stored in difference form (compensated_fp32_kernel)
    constexpr bool DIFF = std::is_same<M, float>::value;
    double xi[ND];
    if constexpr (DIFF) {
#pragma unroll
        for (int db = 0; db < ND; ++db) xi[db] = pdir(i * ND + db);
    }
#pragma unroll 2
    for (int k = gl; k < d; k += G) {
        const int32_t j = SCOLS ? cols[k] : __ldg(cols + k);
        const int64_t c = int64_t(j) * ND;
        double xv[ND];
#pragma unroll
        for (int db = 0; db < ND; ++db) xv[db] = pdir(c + db);
        if constexpr (DIFF) {
            if (j != int32_t(i))
#pragma unroll
                for (int db = 0; db < ND; ++db) xv[db] -= xi[db];
        }
#pragma unroll
        for (int da = 0; da < ND; ++da)
#pragma unroll
            for (int db = 0; db < ND; ++db)
                acc[da] += double(__ldg(v + da * rowlen + k * ND + db)) * xv[db];
    }
}

template <int ND, int G, class M, class V>
__device__ __forceinline__ void node_rows_pp(const int64_t* __restrict__ adj_ptr,
                                             const int32_t* __restrict__ adj,
                                             const int64_t* __restrict__ node_base,
                                             const M* __restrict__ vals, const V* r,
                                             const V* __restrict__ inv_diag, const V* pprev,
                                             V bprev, int64_t i, int gl, double* acc) {
    const int64_t a0 = adj_ptr[i];
    node_rows_pp_at<ND, G, M, V, false>(adj + a0, int(adj_ptr[i + 1] - a0), vals + node_base[i],
                                        r, inv_diag, pprev, bprev, i, gl, acc);
}

// Two grid barriers per iteration (2D models).  Iteration k keeps p_k in buf[k & 1]
// (buf[0] = p, buf[1] = p2) and forms it on the fly from p_{k-1} in the
// other buffer: at the start of iteration k, r_k, beta_{k-1} (PcgScalars.beta)
// and p_{k-1} are final; p_{-1} is zero and beta_{-1} = 0, so p_0 = z_0.
//   A: q = K p_k on own nodes (neighbours' p_k formed from their r and
//      p_{k-1}), p_k of own rows stored, p_k.q     -> grid barrier
//   B: alpha; u += alpha p_k, r -= alpha q on own rows; r.r, r.z
//                                                   -> grid barrier
// then beta_k = r.z / r.z_prev and the next iteration.  A block writes one
// buffer while every block reads the other, and r is written only in B, so
// the two barriers order every access.  Forming p on the fly triples the
// gathered vector loads of the SpMV: on the 200x20 CPS4 case (9 neighbour
// blocks a node) an iteration takes 11.7 us against 14.2 us with three
// barriers, on the 160x16x16 C3D8 case (27 blocks) 48.9 us against 34.9 us,
// so 3D models keep the three-barrier kernel.
template <int ND, int G, class M, class V, class U, bool SADJ>
__global__ void __launch_bounds__(PBLOCK, PBLOCKS_PER_SM)
pcg_persistent2_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                       const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                       const M* __restrict__ vals, const V* __restrict__ inv_diag, U* u, V* r,
                       V* p, V* p2, V* q, double* part_a, double* part_b, PcgScalars* s,
                       GridBarrier* gb, int chunk, int nodes_cap) {
    __shared__ double sh[32];
    const unsigned int B = gridDim.x;
    unsigned int bar_target = 0;  // grid_sync's running arrival target
    const int64_t nb0 = n_nodes * int64_t(blockIdx.x) / B;
    const int64_t nb1 = n_nodes * int64_t(blockIdx.x + 1) / B;
    const int64_t r0 = nb0 * ND, r1 = nb1 * ND;
    volatile PcgScalars* vs = s;
    if (vs->status != PCG_RUNNING) return;
    SharedAdj sa{nullptr, nullptr, nullptr};
    if constexpr (SADJ) sa = load_shared_adj(adj_ptr, adj, node_base, nb0, nb1, nodes_cap);
    double rz = vs->rz, rr = vs->rr, res = vs->res, beta = vs->beta;
    const double bnorm = vs->bnorm, tol = vs->tol, rr_stop = vs->rr_stop;
    long long it = vs->it;
    const long long max_iter = vs->max_iter;
    const int gl = threadIdx.x & (G - 1);
    const int64_t warp_nodes = 32 / G;
    const int64_t step = int64_t(PBLOCK / 32) * warp_nodes;
    const bool writer = (blockIdx.x == 0 && threadIdx.x == 0);
    for (int c = 0; c < chunk; ++c) {
        V* pcur = (it & 1) ? p2 : p;
        const V* pprev = (it & 1) ? p : p2;
        const V bprev = V(beta);
        // A: q = K p_k on own nodes, p_k of own rows, p_k.q
        double dot = 0.0;
        for (int64_t nb = nb0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < nb1; nb += step) {
            const int64_t i = nb + ((threadIdx.x & 31) / G);
            double acc[ND];
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = 0.0;
            if (i < nb1) {
                if constexpr (SADJ) {
                    const int li = int(i - nb0);
                    const int a0 = sa.aptr[li];
                    node_rows_pp_at<ND, G, M, V, true>(sa.cols + a0, sa.aptr[li + 1] - a0,
                                                       vals + sa.vbase[li], r, inv_diag, pprev,
                                                       bprev, i, gl, acc);
                } else {
                    node_rows_pp<ND, G, M, V>(adj_ptr, adj, node_base, vals, r, inv_diag, pprev,
                                              bprev, i, gl, acc);
                }
            }
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
            if (i < nb1 && gl == 0) {
#pragma unroll
                for (int da = 0; da < ND; ++da) {
                    const int64_t row = i * ND + da;
                    const V pk = __ldcg(r + row) * inv_diag[row] + bprev * __ldcg(pprev + row);
                    pcur[row] = pk;
                    const V qv = V(acc[da]);
                    q[row] = qv;
                    dot += double(pk) * double(qv);
                }
            }
        }
        double bs = block_sum(dot, sh);
        if (threadIdx.x == 0) part_a[blockIdx.x] = bs;
        if (!grid_sync(gb, B, bar_target)) return;
        const double pap = sum_partials_cg(part_a, int(B), 1, 0, sh);
        if (!(pap > 0.0)) {  // pap <= 0 or NaN: breakdown
            if (writer) {
                s->pap = pap;
                s->it = it + 1;
                s->res = sqrt(rr) / bnorm;
                s->rr = rr;
                s->rz = rz;
                __threadfence();
                s->status = PCG_BREAKDOWN;
            }
            return;
        }
        const double alpha = rz / pap;
        // B: u += alpha p_k, r -= alpha q on own rows; r.r, r.z
        const V a = V(alpha);
        double lrr = 0.0, lrz = 0.0;
        for (int64_t row = r0 + threadIdx.x; row < r1; row += PBLOCK) {
            const V pi = __ldcg(pcur + row);
            u[row] = U(u[row] + U(a) * U(pi));
            const V ri = __ldcg(r + row) - a * __ldcg(q + row);
            r[row] = ri;
            const V zi = ri * inv_diag[row];
            lrr += double(ri) * double(ri);
            lrz += double(ri) * double(zi);
        }
        const double brr = block_sum(lrr, sh);
        const double brz = block_sum(lrz, sh);
        if (threadIdx.x == 0) {
            part_b[2 * blockIdx.x] = brr;
            part_b[2 * blockIdx.x + 1] = brz;
        }
        if (!grid_sync(gb, B, bar_target)) return;
        const double rr_new = sum_partials_cg(part_b, int(B), 2, 0, sh);
        const double rz_new = sum_partials_cg(part_b, int(B), 2, 1, sh);
        it += 1;
        rr = rr_new;
        res = sqrt(rr) / bnorm;
        if (res <= tol || it >= max_iter || rr <= rr_stop) {
            if (writer) {
                s->it = it;
                s->res = res;
                s->rr = rr;
                s->rz = rz;         // r.z of the previous iterate (beta's denominator)
                s->pap = rz_new;    // r.z of this iterate
                s->alpha = alpha;
                __threadfence();
                s->status = (res <= tol) ? PCG_CONVERGED
                                         : (it >= max_iter ? PCG_MAXITER : PCG_RELIABLE);
            }
            return;
        }
        beta = rz_new / rz;
        rz = rz_new;
    }
    if (writer) {
        s->it = it;
        s->res = res;
        s->rr = rr;
        s->rz = rz;
        s->beta = beta;
    }
}

// ------------------------------------------------------------ shared-memory persistent PCG
// The plain FP64 solve below GRAPH_MIN_NNZ (pcg_fp64).
// A block owns the nodes [n_nodes*b/B, n_nodes*(b+1)/B) and their rows for a
// whole launch.  Its adjacency (row-block offsets, column prefix, column
// node indices) and its rows of u, r, p, q, z and 1/K_ii live in dynamic
// shared memory across the launch; what neighbouring blocks gather goes to
// global memory every iteration, u, r and p at the end of the launch.  Each
// warp computes q = K p for a contiguous run of the block's nodes (G lanes
// per node, partial sums combined by shuffles within the lane group) and
// writes the node's rows of q to shared memory; the vector updates run over
// the block's rows, one thread per row.  The recurrence is solver.rs:82-149
// exactly (q = K p, alpha = r.z / p.q, u += alpha p, r -= alpha q, z = r /
// K_ii, beta = r.z' / r.z, p = z + beta p), so the iterates round like the
// reference's but for the order of the dot-product sums.  Two forms:
//  * ALG 0: p is stored for the neighbours after its update, so an
//    iteration has three grid barriers (p stored; p.q; r.r and r.z);
//  * ALG 1: the SpMV forms each gathered p_j = z_j + beta p_prev_j itself
//    from z (stored with the r update) and the previous p (a second buffer,
//    alternating between iterations), so the barrier after the p update
//    goes away: two grid barriers, two gathered vectors.  Every block forms
//    p_j with the same fused multiply-add, so a row's p is bitwise the same
//    in its owner and in every neighbour.
// Reductions are in a fixed order (warp shuffles, shared memory, then every
// block sums the block partials in index order), so repeated runs are
// bitwise identical.

// The three-barrier form stages the p values its SpMV gathers: the window of
// nodes [lowest, highest neighbour of the block's nodes] is copied from L2
// into shared memory once an iteration (coalesced), instead of every node
// gathering its neighbours' p from L2.  The window holds up to
// STAGE_NODES_PER_NODE x nodes_cap nodes; a block whose window is wider
// (an unstructured node order) gathers from L2 as before.  (On the
// 160 x 16 x 16 C3D8 cantilever a block's window spans 5,800 nodes; staging
// it whole in the shared memory left over, 139 KB, measured 26.5 against
// 25.4 us an iteration gathering from L2, both with 32 lanes a node.)
constexpr int STAGE_NODES_PER_NODE = 4;

__host__ __device__ inline size_t smem_adj_offset(int64_t nodes_cap, int nd, size_t value) {
    return size_t(nodes_cap) * size_t(nd) * value * 6;
}

// Dynamic shared memory of pcg_smem_kernel for `nodes_cap` nodes of `nd`
// dofs and at most max_deg neighbours: six vectors of nodes_cap * nd
// values of `value` bytes, the adjacency in load_shared_adj's layout (rounded up to 16
// bytes), then the staging window of stage_nodes nodes.
size_t smem_pcg_bytes(int64_t nodes_cap, int nd, int max_deg, int64_t stage_nodes, size_t value) {
    const size_t adj = (shared_adj_bytes(nodes_cap, max_deg) + 15) / 16 * 16;
    return smem_adj_offset(nodes_cap, nd, value) + adj + size_t(stage_nodes) * size_t(nd) * value;
}

__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// The gathered value of column c: p_c itself (ALG 0) or z_c + beta pprev_c
// formed with one fused multiply-add of the vectors' type (ALG 1).
// XS: x is the shared-memory staging window of the nodes from xoff / ND on.
template <int ALG, bool XS, class V>
__device__ __forceinline__ double gathered(const V* x, const V* z, const V* pprev, V beta,
                                           int64_t c, int64_t xoff) {
    if constexpr (ALG == 0) {
        if constexpr (XS) return double(x[c - xoff]);
        else return double(__ldcg(x + c));
    }
    return double(fma_rn(beta, __ldcg(pprev + c), __ldcg(z + c)));
}

// One node's rows, lane gl of its G-lane group taking neighbour blocks gl,
// gl + G, ...  The values come from the transposed copy (entry (da, db) of
// neighbour slot k at (da ND + db) d + k from the node's base), so the loads
// of one (da, db) by the lanes of a group are consecutive values, where in
// the row layout they stride ND.  The first block is loaded under a
// predicate rather than a branch, so that the U nodes of a warp step issue
// its loads before their first multiply-add; the blocks past the first G (a
// C3D8 node's 27 at G = 8) loop.  An FP32 operator is in difference form:
// the node's own x (own) is taken from every other neighbour's.
template <int ND, int G, int ALG, bool XS, class M, class V>
__device__ __forceinline__ void node_rows_pred(bool valid, const int32_t* cols, int d, const M* v,
                                               const V* x, const V* z, const V* pprev, V beta,
                                               int64_t i, int gl, double* acc, int64_t xoff,
                                               const V* own) {
    constexpr bool DIFF = std::is_same<M, float>::value;
    const bool act = valid && gl < d;
    const int32_t j0 = act ? cols[gl] : 0;
    const int64_t c0 = int64_t(j0) * ND;
    double xv[ND], xi[ND];
#pragma unroll
    for (int db = 0; db < ND; ++db) {
        xv[db] = act ? gathered<ALG, XS>(x, z, pprev, beta, c0 + db, xoff) : 0.0;
        xi[db] = DIFF ? double(own[db]) : 0.0;
        if (DIFF && act && j0 != int32_t(i)) xv[db] -= xi[db];
    }
#pragma unroll
    for (int da = 0; da < ND; ++da)
#pragma unroll
        for (int db = 0; db < ND; ++db)
            acc[da] += (act ? double(__ldg(v + (da * ND + db) * d + gl)) : 0.0) * xv[db];
    if (valid && d > G) {
        for (int k = gl + G; k < d; k += G) {
            const int32_t j = cols[k];
            const int64_t c = int64_t(j) * ND;
#pragma unroll
            for (int db = 0; db < ND; ++db) {
                xv[db] = gathered<ALG, XS>(x, z, pprev, beta, c + db, xoff);
                if (DIFF && j != int32_t(i)) xv[db] -= xi[db];
            }
#pragma unroll
            for (int da = 0; da < ND; ++da)
#pragma unroll
                for (int db = 0; db < ND; ++db)
                    acc[da] += double(__ldg(v + (da * ND + db) * d + k)) * xv[db];
        }
    }
    if (valid && d == 0 && gl == 0)  // an unreferenced node: rows of length 1
#pragma unroll
        for (int da = 0; da < ND; ++da)
            acc[da] = double(v[da]) * gathered<ALG, XS>(x, z, pprev, beta, i * ND + da, xoff);
}

template <int ND, int G, int PB, int BPS, int ALG, int U, class M, class V>
__global__ void __launch_bounds__(PB, BPS)
pcg_smem_kernel(int64_t n_nodes, const int64_t* __restrict__ adj_ptr,
                const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                const M* __restrict__ vals, const V* __restrict__ inv_diag,
                V* u_g, V* r_g, V* p_g, V* p2_g, V* z_g,
                double* part, PcgScalars* s, GridBarrier* gb, int chunk, int nodes_cap,
                int max_deg, int stage, int first) {
    extern __shared__ __align__(16) unsigned char svx_dyn_smem[];
    __shared__ double sh[66];
    // block-uniform values kept out of registers: ||f||, tol, the last
    // iterate's ||r|| / ||f|| and r.r (thread 0 keeps them), the reliable
    // update's r.r, max_iter
    __shared__ double s_c[5];
    __shared__ long long s_max_iter;
    constexpr int NPS = 32 / G;  // nodes per warp step
    constexpr int W = PB / 32;
    const unsigned int B = gridDim.x;
    unsigned int bar_target = 0;
    volatile PcgScalars* vs = s;
    if (vs->status != PCG_RUNNING) return;
    // nodes and rows fit in int32 (the CSR indices are int32)
    const int nb0 = int(n_nodes * int64_t(blockIdx.x) / B);
    const int nb1 = int(n_nodes * int64_t(blockIdx.x + 1) / B);
    const int nloc = nb1 - nb0, rows = nloc * ND, row0 = nb0 * ND;
    const int rcap = nodes_cap * ND;
    V* u_s = reinterpret_cast<V*>(svx_dyn_smem);
    V* r_s = u_s + rcap;
    V* p_s = r_s + rcap;
    V* q_s = p_s + rcap;
    V* z_s = q_s + rcap;
    V* d_s = z_s + rcap;
    const SharedAdj sa = load_shared_adj_at(reinterpret_cast<unsigned char*>(d_s + rcap),
                                            adj_ptr, adj, node_base, nb0, nb1, nodes_cap);
    // the staging window (three-barrier form): nodes [jlo, jhi] of every
    // column the block's rows reach, its own nodes included
    __shared__ int s_jlo, s_jhi;
    V* xs = reinterpret_cast<V*>(
        svx_dyn_smem + smem_adj_offset(nodes_cap, ND, sizeof(V)) +
        (shared_adj_bytes(nodes_cap, max_deg) + 15) / 16 * 16);
    bool staged = false;
    int jlo = 0, jhi = -1;
    if constexpr (ALG == 0) {
        if (threadIdx.x == 0) {
            s_jlo = nb0;
            s_jhi = nb1 - 1;
        }
        __syncthreads();
        const int cnt = nloc > 0 ? sa.aptr[nloc] : 0;
        int lo = nb0, hi = nb1 - 1;
        for (int t = threadIdx.x; t < cnt; t += PB) {
            lo = min(lo, sa.cols[t]);
            hi = max(hi, sa.cols[t]);
        }
        atomicMin(&s_jlo, lo);
        atomicMax(&s_jhi, hi);
        __syncthreads();
        jlo = s_jlo;
        jhi = s_jhi;
        staged = nloc > 0 && (jhi - jlo + 1) <= stage;
    }
    if (threadIdx.x == 0) {
        s_c[0] = vs->bnorm;
        s_c[1] = vs->tol;
        s_c[2] = vs->res;
        s_c[3] = vs->rr;
        s_c[4] = vs->rr_stop;
        s_max_iter = vs->max_iter;
    }
    long long it = vs->it;
    double rz = vs->rz, beta = vs->beta;
    // ALG 1 alternates the previous-p buffers: iteration it reads p_{it-1}
    // from buf(it) and writes p_it to buf(it + 1)
    auto buf = [&](long long k) -> V* { return (k & 1) ? p2_g : p_g; };
    for (int t = threadIdx.x; t < rows; t += PB) {
        const int row = row0 + t;
        const V di = inv_diag[row];
        const V ri = r_g[row];
        d_s[t] = di;
        r_s[t] = ri;
        z_s[t] = ri * di;
        u_s[t] = u_g[row];
        // the first launch starts from p = z (the init kernel's p); later
        // launches from the stored direction
        p_s[t] = ALG == 1 ? (first ? V(0) : buf(it)[row]) : p_g[row];
    }
    if (ALG == 1 && first) beta = 0.0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wn0 = nb0 + nloc * warp / W, wn1 = nb0 + nloc * (warp + 1) / W;
    const int gl = lane & (G - 1), grp = lane / G;
    const bool writer = (blockIdx.x == 0 && threadIdx.x == 0);
    __syncthreads();
    // the two reductions of an iteration use two slots of `part`.  (Posting the
    // sums as numbered words that every block polls, instead of the counting
    // barrier, measured slower: 8.8 against 7.2 us an iteration at 81 nodes,
    // 12.4 against 8.2 at 6,561.)
    auto grid_totals = [&](int slot, double a, double b, double& ta, double& tb) -> bool {
        return grid_pair_sum(gb, B, bar_target, part + size_t(slot) * 2 * B, sh, a, b, ta, tb);
    };
    if (ALG == 1 && first) {
        // neighbours gather z and the previous p (zero): store z, barrier
        for (int t = threadIdx.x; t < rows; t += PB) {
            z_g[row0 + t] = z_s[t];
            p_g[row0 + t] = V(0);
        }
        if (!grid_sync(gb, B, bar_target)) return;
    }
    auto finish = [&](int status) {
        for (int t = threadIdx.x; t < rows; t += PB) {
            const int row = row0 + t;
            u_g[row] = u_s[t];
            r_g[row] = r_s[t];
            if (ALG == 0) p_g[row] = p_s[t];
        }
        if (writer) {
            s->it = it;
            s->res = s_c[2];
            s->rr = s_c[3];
            s->rz = rz;
            s->beta = beta;
            __threadfence();
            if (status != PCG_RUNNING) s->status = status;
        }
    };

    for (int c = 0; c < chunk; ++c) {
        // q = K p on the block's nodes, p.q on its rows
        const V* pprev = buf(it);
        V* pnext = buf(it + 1);
        const V bt = V(beta);
        if (ALG == 0) {
            for (int t = threadIdx.x; t < rows; t += PB) p_g[row0 + t] = p_s[t];
            if (!grid_sync(gb, B, bar_target)) return;
            if (staged) {
                const int x0 = jlo * ND, xn = (jhi - jlo + 1) * ND;
                for (int t = threadIdx.x; t < xn; t += PB) xs[t] = __ldcg(p_g + x0 + t);
                __syncthreads();
            }
        } else {
            for (int t = threadIdx.x; t < rows; t += PB) {
                const V pi = fma_rn(bt, p_s[t], z_s[t]);
                p_s[t] = pi;
                pnext[row0 + t] = pi;
            }
            if (std::is_same<M, float>::value) __syncthreads();  // rows read their own p
        }
        // U steps of the warp's nodes at a time, all their loads in flight
        const int steps = (wn1 - wn0 + NPS - 1) / NPS;
        for (int k = 0; k < steps; k += U) {
            double acc[U][ND];
#pragma unroll
            for (int uu = 0; uu < U; ++uu) {
                const int i = wn0 + (k + uu) * NPS + grp;
                const bool valid = i < wn1;
                const int li = valid ? i - nb0 : 0;
                const int a0 = sa.aptr[li];
                const int d = valid ? sa.aptr[li + 1] - a0 : 0;
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[uu][da] = 0.0;
                const int64_t vb = valid ? sa.vbase[li] : 0;
                if (staged)
                    node_rows_pred<ND, G, ALG, true>(valid, sa.cols + a0, d, vals + vb,
                                                     (const V*)xs, (const V*)z_g, pprev, bt, i, gl,
                                                     acc[uu], int64_t(jlo) * ND,
                                                     (const V*)p_s + li * ND);
                else
                    node_rows_pred<ND, G, ALG, false>(valid, sa.cols + a0, d, vals + vb,
                                                      (const V*)p_g, (const V*)z_g, pprev, bt, i,
                                                      gl, acc[uu], 0, (const V*)p_s + li * ND);
            }
#pragma unroll
            for (int uu = 0; uu < U; ++uu)
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[uu][da] = group_sum<G>(acc[uu][da]);
#pragma unroll
            for (int uu = 0; uu < U; ++uu) {
                const int i = wn0 + (k + uu) * NPS + grp;
                if (i < wn1 && gl < ND) {
                    double qi = acc[uu][0];
#pragma unroll
                    for (int da = 1; da < ND; ++da)
                        if (gl == da) qi = acc[uu][da];
                    q_s[(i - nb0) * ND + gl] = V(qi);
                }
            }
        }
        __syncthreads();
        double pq = 0.0, zero = 0.0;
        for (int t = threadIdx.x; t < rows; t += PB) pq += double(p_s[t]) * double(q_s[t]);
        double pap, unused;
        if (!grid_totals(0, pq, zero, pap, unused)) return;
        if (!(pap > 0.0)) {  // p.Kp <= 0 or NaN: breakdown
            it += 1;
            if (writer) s->pap = pap;
            finish(PCG_BREAKDOWN);
            return;
        }
        const V alpha = V(rz / pap);
        // u += alpha p, r -= alpha q, z = r / K_ii; r.r, r.z
        double lrr = 0.0, lrz = 0.0;
        for (int t = threadIdx.x; t < rows; t += PB) {
            u_s[t] += alpha * p_s[t];
            const V ri = r_s[t] - alpha * q_s[t];
            const V zi = ri * d_s[t];
            r_s[t] = ri;
            z_s[t] = zi;
            if (ALG == 1) z_g[row0 + t] = zi;
            lrr += double(ri) * double(ri);
            lrz += double(ri) * double(zi);
        }
        double rr, rz_new;
        if (!grid_totals(1, lrr, lrz, rr, rz_new)) return;
        it += 1;
        const double res = sqrt(rr) / s_c[0];
        if (threadIdx.x == 0) {
            s_c[2] = res;
            s_c[3] = rr;
        }
        if (res <= s_c[1] || it >= s_max_iter) {
            if (ALG == 1) beta = rz_new / rz;  // the next p of a resumed solve
            rz = rz_new;
            finish(res <= s_c[1] ? PCG_CONVERGED : PCG_MAXITER);
            return;
        }
        if (rr <= s_c[4]) {  // rz stays r.z of the previous iterate
            finish(PCG_RELIABLE);
            return;
        }
        beta = rz_new / rz;
        rz = rz_new;
        if (ALG == 0)
            for (int t = threadIdx.x; t < rows; t += PB) p_s[t] = z_s[t] + V(beta) * p_s[t];
    }
    finish(PCG_RUNNING);
}


// ------------------------------------------------------------ one dof a node
// The persistent PCG of conduction systems.  A scalar row has one value a
// neighbour, so with several lanes a node (pcg_smem_kernel) the loads of the
// gathers bound it: eight lanes a node, four nodes a warp touch a dozen cache
// lines a load, 22.5 us an iteration at 240 x 24 x 24.  Here a lane owns a
// node and a warp a slice of 32 consecutive nodes, K stored slice by slice
// with the neighbour slot outermost ([slice][slot][lane], rows padded with
// zeros to the largest degree), so a warp reads K and its columns in full
// lines and, the k-th neighbours of consecutive nodes being consecutive nodes
// in a structured mesh, gathers nearly so, through the L1 (the grid barrier's
// acquire leaves no stale line there).  z and the previous p are one pair, so
// that a neighbour is one load: the pairs of an iteration are written before
// its second barrier and gathered only before the next one's first, so one
// buffer is enough.  Two barriers an iteration as in ALG 1 above, whose
// recurrence this is: 10.7 us an iteration at 240 x 24 x 24 (3.48 ms a solve
// of 326, 7.35 before), of which the two grid sums take 5 and reading K
// (33 MB) from the L2 most of the rest; 7.0 at 120 x 12 x 12 (8.8 before).
// 1,024 threads a block, 5 or 14 neighbours in flight, and the columns left
// in the L2 measured within 5% of this or slower.
constexpr int SCALAR_THREADS = 512;
constexpr int SCALAR_BATCH = 9;  // neighbours in flight: a third of a solid's 27, a plate's 9
constexpr size_t SCALAR_SMEM = 200 * 1024;
// Rows wider than a solid's 27 keep pcg_smem_kernel, and so does a system that
// padding every row to the widest would make more than twice as large (the
// kernel streams it each iteration; a small one is not bound by that).
constexpr int SCALAR_MAX_DEG = 32;
constexpr int64_t SCALAR_SMALL = 65536;

__global__ void slice_rows_kernel(int64_t n, int width, const int64_t* __restrict__ adj_ptr,
                                  const int32_t* __restrict__ adj,
                                  const int64_t* __restrict__ node_base,
                                  const double* __restrict__ vals, double* __restrict__ out,
                                  int32_t* __restrict__ cols) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;  // rounded up to slices
    const int64_t s = i / 32, lane = i % 32;
    if (s * 32 >= n) return;
    const int64_t a0 = i < n ? adj_ptr[i] : 0;
    const int d = i < n ? int(adj_ptr[i + 1] - a0) : 0;
    const int32_t self = int32_t(i < n ? i : n - 1);
    const double* v = i < n ? vals + node_base[i] : vals;
    for (int k = 0; k < width; ++k) {
        const int64_t at = (s * width + k) * 32 + lane;
        // a node no element uses has a row of its diagonal alone
        out[at] = k < d ? v[k] : (d == 0 && i < n && k == 0 ? v[0] : 0.0);
        cols[at] = k < d ? adj[a0 + k] : self;
    }
}

template <int PB>
__global__ void __launch_bounds__(PB, 1)
pcg_scalar_kernel(int64_t n, int width, const double* __restrict__ vals,
                  const int32_t* __restrict__ cols, const double* __restrict__ inv_diag,
                  double* u_g, double* r_g, double2* zp, double* part, PcgScalars* s,
                  GridBarrier* gb, int chunk, int cap, int cols_here, int first) {
    extern __shared__ __align__(16) unsigned char svx_dyn_smem[];
    __shared__ double sh[66];
    constexpr int W = PB / 32, U = SCALAR_BATCH;
    const unsigned int B = gridDim.x;
    unsigned int bar_target = 0;
    volatile PcgScalars* vs = s;
    if (vs->status != PCG_RUNNING) return;
    const int slices = int((n + 31) / 32);
    const int s0 = int(int64_t(slices) * blockIdx.x / B),
              s1 = int(int64_t(slices) * (blockIdx.x + 1) / B);
    const int row0 = s0 * 32, rows = min(int(n), s1 * 32) - row0;
    double* u_s = reinterpret_cast<double*>(svx_dyn_smem);
    double* r_s = u_s + cap;
    double* p_s = r_s + cap;
    double* q_s = p_s + cap;
    double* z_s = q_s + cap;
    double* d_s = z_s + cap;
    int32_t* c_s = reinterpret_cast<int32_t*>(d_s + cap);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double bnorm = vs->bnorm, tol = vs->tol;
    const long long max_iter = vs->max_iter;
    long long it = vs->it;
    double rz = vs->rz, beta = vs->beta, rr = vs->rr, res = vs->res;
    if (first) beta = 0.0;
    for (int t = threadIdx.x; t < rows; t += PB) {
        const int row = row0 + t;
        const double di = inv_diag[row], ri = r_g[row];
        d_s[t] = di;
        r_s[t] = ri;
        z_s[t] = ri * di;
        u_s[t] = u_g[row];
        p_s[t] = first ? 0.0 : zp[row].y;
        if (first) zp[row] = make_double2(ri * di, 0.0);
    }
    if (cols_here)
        for (int t = threadIdx.x; t < (s1 - s0) * width * 32; t += PB)
            c_s[t] = cols[int64_t(s0) * width * 32 + t];
    if (!grid_sync(gb, B, bar_target)) return;
    int status = PCG_RUNNING;
    for (int c = 0; c < chunk && status == PCG_RUNNING; ++c) {
        for (int sl = s0 + warp; sl < s1; sl += W) {
            const double* v = vals + int64_t(sl) * width * 32 + lane;
            const int32_t* cl = cols_here ? c_s + (sl - s0) * width * 32 + lane
                                          : cols + int64_t(sl) * width * 32 + lane;
            double acc[3] = {0.0, 0.0, 0.0};
            int k = 0;
            for (; k + U <= width; k += U) {
                double kv[U];
                double2 x[U];
#pragma unroll
                for (int m = 0; m < U; ++m) kv[m] = __ldg(v + (k + m) * 32);
#pragma unroll
                for (int m = 0; m < U; ++m) x[m] = zp[cl[(k + m) * 32]];
#pragma unroll
                for (int m = 0; m < U; ++m) acc[m % 3] += kv[m] * __fma_rn(beta, x[m].y, x[m].x);
            }
            for (; k < width; ++k) {
                const double2 x = zp[cl[k * 32]];
                acc[0] += __ldg(v + k * 32) * __fma_rn(beta, x.y, x.x);
            }
            const int t = (sl - s0) * 32 + lane;
            if (t < rows) q_s[t] = (acc[0] + acc[1]) + acc[2];
        }
        __syncthreads();
        double pq = 0.0, pap, unused;
        for (int t = threadIdx.x; t < rows; t += PB) {
            const double pi = __fma_rn(beta, p_s[t], z_s[t]);
            p_s[t] = pi;
            pq += pi * q_s[t];
        }
        if (!grid_pair_sum(gb, B, bar_target, part, sh, pq, 0.0, pap, unused)) return;
        if (!(pap > 0.0)) {  // p.Kp <= 0 or NaN: breakdown
            it += 1;
            status = PCG_BREAKDOWN;
            break;
        }
        const double alpha = rz / pap;
        double lrr = 0.0, lrz = 0.0, rz_new;
        for (int t = threadIdx.x; t < rows; t += PB) {
            const double pi = p_s[t];
            u_s[t] += alpha * pi;
            const double ri = r_s[t] - alpha * q_s[t];
            const double zi = ri * d_s[t];
            r_s[t] = ri;
            z_s[t] = zi;
            zp[row0 + t] = make_double2(zi, pi);
            lrr += ri * ri;
            lrz += ri * zi;
        }
        if (!grid_pair_sum(gb, B, bar_target, part + 2 * size_t(B), sh, lrr, lrz, rr, rz_new))
            return;
        it += 1;
        res = sqrt(rr) / bnorm;
        beta = rz_new / rz;
        rz = rz_new;
        status = res <= tol ? PCG_CONVERGED : it >= max_iter ? PCG_MAXITER : PCG_RUNNING;
    }
    for (int t = threadIdx.x; t < rows; t += PB) {
        u_g[row0 + t] = u_s[t];
        r_g[row0 + t] = r_s[t];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->it = it;
        s->res = res;
        s->rr = rr;
        s->rz = rz;
        s->beta = beta;
        __threadfence();
        if (status != PCG_RUNNING) s->status = status;
    }
}

// ------------------------------------------------------------ batched PCG
// Thousands of independent models concatenated into one block-diagonal
// operator.  One launch with one CTA per instance (instances ordered by
// size, largest first, so the block scheduler hands out the longest work
// first); the CTA runs that instance's whole Jacobi-PCG with CTA-local
// reductions, so every instance has its own alpha/beta, its own convergence
// test and its own iteration count, and no CTA ever waits for another.  The
// grid is not persistent: CTAs of other streams' kernels (the assembly of
// the next served batch, on a higher-priority stream) are scheduled as soon
// as any instance finishes.  An instance is always computed by one CTA of
// the same shape, so its result does not depend on what else is in the
// batch.
template <int ND, int G, class M>
__device__ __forceinline__ void node_rows_mv(const int64_t* __restrict__ adj_ptr,
                                             const int32_t* __restrict__ adj,
                                             const int64_t* __restrict__ node_base,
                                             const M* __restrict__ vals, const double* x,
                                             int64_t i, int gl, double* acc) {
    const int64_t a0 = adj_ptr[i];
    const int d = int(adj_ptr[i + 1] - a0);
    const M* __restrict__ v = vals + node_base[i];
    if (d == 0) {
        if (gl == 0)
#pragma unroll
            for (int da = 0; da < ND; ++da) acc[da] = double(v[da]) * x[i * ND + da];
        return;
    }
    const int rowlen = ND * d;
    constexpr bool DIFF = std::is_same<M, float>::value;  // difference form
    double xi[ND];
    if constexpr (DIFF) {
#pragma unroll
        for (int db = 0; db < ND; ++db) xi[db] = x[i * ND + db];
    }
    for (int k = gl; k < d; k += G) {
        const int32_t j = __ldg(adj + a0 + k);
        const int64_t c = int64_t(j) * ND;
        double xv[ND];
#pragma unroll
        for (int db = 0; db < ND; ++db) xv[db] = x[c + db];
        if constexpr (DIFF) {
            if (j != int32_t(i))
#pragma unroll
                for (int db = 0; db < ND; ++db) xv[db] -= xi[db];
        }
#pragma unroll
        for (int da = 0; da < ND; ++da)
#pragma unroll
            for (int db = 0; db < ND; ++db)
                acc[da] += double(__ldg(v + da * rowlen + k * ND + db)) * xv[db];
    }
}

template <int ND, int G, int BS, class M>
__global__ void __launch_bounds__(BS, (ND == 2 ? 1536 : BATCH_MIN_THREADS) / BS)
batch_pcg_kernel(int count, const int32_t* __restrict__ order, const int64_t* __restrict__ node_off,
                 const int64_t* __restrict__ adj_ptr, const int32_t* __restrict__ adj,
                 const int64_t* __restrict__ node_base, const M* __restrict__ vals,
                 const double* __restrict__ inv_diag, const double* __restrict__ f, double* u,
                 double* r, double* p, double* q, const double* __restrict__ tol,
                 const int64_t* __restrict__ max_iter, int64_t* __restrict__ out_it,
                 double* __restrict__ out_res, int32_t* __restrict__ out_status) {
    __shared__ double sh[32];
    const int gl = threadIdx.x & (G - 1);
    const int64_t warp_nodes = 32 / G;
    const int64_t step = int64_t(BS / 32) * warp_nodes;
    for (int k = blockIdx.x; k < count; k += gridDim.x) {
        const int inst = order[k];
        const int64_t n0 = node_off[inst], n1 = node_off[inst + 1];
        const int64_t r0 = n0 * ND, r1 = n1 * ND;
        const double tl = tol[inst];
        const int64_t mi = max_iter[inst];
        double rr = 0.0, rz = 0.0;
        for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
            const double ri = f[row];
            u[row] = 0.0;
            r[row] = ri;
            const double zi = ri * inv_diag[row];
            p[row] = zi;
            rr += ri * ri;
            rz += ri * zi;
        }
        rr = block_sum(rr, sh);
        rz = block_sum(rz, sh);
        const double bnorm = sqrt(rr);
        int64_t it = 0;
        int status = (bnorm == 0.0) ? PCG_CONVERGED : PCG_RUNNING;
        double res = (bnorm == 0.0) ? 0.0 : 1.0;
        while (status == PCG_RUNNING) {
            double dot = 0.0;
            for (int64_t nb = n0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < n1; nb += step) {
                const int64_t i = nb + ((threadIdx.x & 31) / G);
                double acc[ND];
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[da] = 0.0;
                if (i < n1) node_rows_mv<ND, G, M>(adj_ptr, adj, node_base, vals, p, i, gl, acc);
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
                if (i < n1 && gl == 0) {
#pragma unroll
                    for (int da = 0; da < ND; ++da) {
                        q[i * ND + da] = acc[da];
                        dot += p[i * ND + da] * acc[da];
                    }
                }
            }
            const double pap = block_sum(dot, sh);
            if (!(pap > 0.0)) {  // pap <= 0 or NaN: breakdown
                status = PCG_BREAKDOWN;
                it += 1;
                res = sqrt(rr) / bnorm;
                break;
            }
            const double alpha = rz / pap;
            double lrr = 0.0, lrz = 0.0;
            for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                u[row] += alpha * p[row];
                const double ri = r[row] - alpha * q[row];
                r[row] = ri;
                const double zi = ri * inv_diag[row];
                lrr += ri * ri;
                lrz += ri * zi;
            }
            rr = block_sum(lrr, sh);
            const double rz_new = block_sum(lrz, sh);
            it += 1;
            res = sqrt(rr) / bnorm;
            if (res <= tl) {
                status = PCG_CONVERGED;
                break;
            }
            if (it >= mi) {
                status = PCG_MAXITER;
                break;
            }
            const double beta = rz_new / rz;
            rz = rz_new;
            for (int64_t row = r0 + threadIdx.x; row < r1; row += BS)
                p[row] = r[row] * inv_diag[row] + beta * p[row];
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            out_it[inst] = it;
            out_res[inst] = res;
            out_status[inst] = status;
        }
    }
}

// Mixed form of the batched PCG, per instance the rule of pcg_mixed: the
// FP64 operator until ||r|| / ||f|| <= mixed_switch_residual(tol), where
// the iterate (u, r, p and the scalars) is kept in u_sv / r_sv / p_sv, then
// the FP32 difference-form operator (vals32) on the same search directions
// to the tolerance, for at most as many iterations as the FP64 phase took;
// the true residual f - K64 u decides, and when the FP32 phase runs out of
// budget or its true residual is short of tol, the instance rolls back to
// the kept iterate and finishes on the FP64 operator.  All of it is
// CTA-local, so
// every instance keeps its own scalars and its result does not depend on
// the rest of the batch.
template <int ND, int G, int BS>
__global__ void __launch_bounds__(BS, BATCH_MIN_THREADS / BS)
batch_pcg_mixed_kernel(int count, const int32_t* __restrict__ order,
                       const int64_t* __restrict__ node_off, const int64_t* __restrict__ adj_ptr,
                       const int32_t* __restrict__ adj, const int64_t* __restrict__ node_base,
                       const double* __restrict__ vals, const float* __restrict__ vals32,
                       const double* __restrict__ inv_diag, const double* __restrict__ f,
                       double* u, double* r, double* p, double* q, const double* __restrict__ tol,
                       const int64_t* __restrict__ max_iter, int64_t* __restrict__ out_it,
                       double* __restrict__ out_res, int32_t* __restrict__ out_status,
                       int64_t* __restrict__ out_fp32_it, double* __restrict__ u_sv,
                       double* __restrict__ r_sv, double* __restrict__ p_sv) {
    __shared__ double sh[32];
    const int gl = threadIdx.x & (G - 1);
    const int64_t warp_nodes = 32 / G;
    const int64_t step = int64_t(BS / 32) * warp_nodes;
    for (int k = blockIdx.x; k < count; k += gridDim.x) {
        const int inst = order[k];
        const int64_t n0 = node_off[inst], n1 = node_off[inst + 1];
        const int64_t r0 = n0 * ND, r1 = n1 * ND;
        const double tl = tol[inst], tau = mixed_switch_residual(tl);
        const int64_t mi = max_iter[inst];
        double rr = 0.0, rz = 0.0;
        for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
            const double ri = f[row];
            u[row] = 0.0;
            r[row] = ri;
            const double zi = ri * inv_diag[row];
            p[row] = zi;
            rr += ri * ri;
            rz += ri * zi;
        }
        rr = block_sum(rr, sh);
        rz = block_sum(rz, sh);
        const double bnorm = sqrt(rr);
        int64_t it = 0, fp32_it = 0;
        int status = (bnorm == 0.0) ? PCG_CONVERGED : PCG_RUNNING;
        double res = (bnorm == 0.0) ? 0.0 : 1.0;
        bool exact = true, switched = false, save = false;
        int64_t cap_end = 0;
        double rz_sv = 0.0, rr_sv = 0.0;
        while (status == PCG_RUNNING) {
            double dot = 0.0;
            for (int64_t nb = n0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < n1; nb += step) {
                const int64_t i = nb + ((threadIdx.x & 31) / G);
                double acc[ND];
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[da] = 0.0;
                if (i < n1) {
                    if (exact)
                        node_rows_mv<ND, G, double>(adj_ptr, adj, node_base, vals, p, i, gl, acc);
                    else
                        node_rows_mv<ND, G, float>(adj_ptr, adj, node_base, vals32, p, i, gl,
                                                   acc);
                }
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
                if (i < n1 && gl == 0) {
#pragma unroll
                    for (int da = 0; da < ND; ++da) {
                        q[i * ND + da] = acc[da];
                        dot += p[i * ND + da] * acc[da];
                    }
                }
            }
            const double pap = block_sum(dot, sh);
            if (!(pap > 0.0)) {  // pap <= 0 or NaN: breakdown
                status = PCG_BREAKDOWN;
                it += 1;
                res = sqrt(rr) / bnorm;
                break;
            }
            const double alpha = rz / pap;
            double lrr = 0.0, lrz = 0.0;
            for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                u[row] += alpha * p[row];
                const double ri = r[row] - alpha * q[row];
                r[row] = ri;
                const double zi = ri * inv_diag[row];
                lrr += ri * ri;
                lrz += ri * zi;
            }
            rr = block_sum(lrr, sh);
            double rz_new = block_sum(lrz, sh);
            it += 1;
            if (!exact) ++fp32_it;
            res = sqrt(rr) / bnorm;
            bool rollback = false;
            if (exact && !switched && res <= tau && res > tl) {
                exact = false;  // the FP32 operator from here, same search directions
                switched = true;
                save = true;       // this iterate is kept for a rollback
                cap_end = 2 * it;  // FP32 budget: as many iterations as the FP64 phase
            } else if (!exact && it >= cap_end && res > tl) {
                rollback = true;  // budget spent
            }
            if (res <= tl && !exact) {
                // reliable update: r = f - K64 u, then r.r and r.z of it
                __syncthreads();
                double trr = 0.0, trz = 0.0;
                for (int64_t nb = n0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < n1;
                     nb += step) {
                    const int64_t i = nb + ((threadIdx.x & 31) / G);
                    double hi[ND], lo[ND];
#pragma unroll
                    for (int da = 0; da < ND; ++da) hi[da] = lo[da] = 0.0;
                    if (i < n1)
                        node_rows_dd<ND, G, false>(adj_ptr, adj, node_base, vals, u, i, gl, hi,
                                                   lo);
#pragma unroll
                    for (int da = 0; da < ND; ++da) group_sum_dd<G>(hi[da], lo[da]);
                    if (i < n1 && gl == 0) {
#pragma unroll
                        for (int da = 0; da < ND; ++da) {
                            const int64_t row = i * ND + da;
                            const double ri = dd_residual(f[row], hi[da], lo[da]);
                            r[row] = ri;
                            trr += ri * ri;
                            trz += ri * (ri * inv_diag[row]);
                        }
                    }
                }
                rr = block_sum(trr, sh);
                rz_new = block_sum(trz, sh);
                res = sqrt(rr) / bnorm;
                // the true residual decides; short of tol, the FP32 phase
                // is undone
                rollback = res > tl;
            }
            if (rollback) {
                // back to the iterate of the switch, on the FP64 operator
                // from there: the FP32 phase's updates are discarded
                __syncthreads();  // r rows written by other lanes of this CTA
                for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                    u[row] = u_sv[row];
                    r[row] = r_sv[row];
                    p[row] = p_sv[row];
                }
                rz = rz_sv;
                rr = rr_sv;
                res = sqrt(rr) / bnorm;
                exact = true;
                __syncthreads();  // p rows read by other lanes' SpMV
                if (it >= mi) {
                    status = PCG_MAXITER;
                    break;
                }
                continue;
            }
            if (res <= tl) {
                status = PCG_CONVERGED;
                break;
            }
            if (it >= mi) {
                status = PCG_MAXITER;
                break;
            }
            const double beta = rz_new / rz;
            rz = rz_new;
            __syncthreads();  // r rows written by other lanes of this CTA
            for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                const double pi = r[row] * inv_diag[row] + beta * p[row];
                p[row] = pi;
                if (save) {
                    u_sv[row] = u[row];
                    r_sv[row] = r[row];
                    p_sv[row] = pi;
                }
            }
            if (save) {
                rz_sv = rz;
                rr_sv = rr;
                save = false;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            out_it[inst] = it;
            out_res[inst] = res;
            out_status[inst] = status;
            out_fp32_it[inst] = fp32_it;
        }
    }
}

// Large members of a batch: one thread-block cluster of CS CTAs per
// instance.  A single CTA streams a 100k-DOF member's K at a few tens of
// GB/s, so the largest members would run alone for seconds at the end of a
// batch.  The CTAs of a cluster are co-scheduled by the hardware, split the
// member's nodes into CS contiguous ranges and meet at cluster barriers
// (barrier.cluster arrive.release / wait.acquire, so the p, u and r rows
// other CTAs of the cluster wrote are visible, read through L2).  Dots are
// reduced per CTA, published in shared memory and summed by every CTA over
// the cluster's ranks through distributed shared memory in rank order, so
// all CTAs hold bitwise the same scalars and the result does not depend on
// the rest of the batch.  The partial slots of consecutive phases differ,
// and every slot is rewritten only after a later cluster barrier, so one
// barrier per phase suffices.  MIXED runs the reliable-update form of
// batch_pcg_mixed_kernel with the same rules.
#ifndef SVX_CLUSTER_MIXED_MIN_THREADS
#define SVX_CLUSTER_MIXED_MIN_THREADS 768
#endif
#ifndef SVX_CLUSTER_MIN_THREADS
#define SVX_CLUSTER_MIN_THREADS 1024
#endif
constexpr int CLUSTER_MIXED_MIN_THREADS = SVX_CLUSTER_MIXED_MIN_THREADS;
constexpr int CLUSTER_MIN_THREADS = SVX_CLUSTER_MIN_THREADS;
template <int ND, int G, int BS, int CS, bool MIXED>
__global__ void __launch_bounds__(
    BS, (MIXED ? CLUSTER_MIXED_MIN_THREADS : CLUSTER_MIN_THREADS) / BS > 0
            ? (MIXED ? CLUSTER_MIXED_MIN_THREADS : CLUSTER_MIN_THREADS) / BS
            : 1)
batch_pcg_cluster_kernel(int count, const int32_t* __restrict__ order,
                         const int64_t* __restrict__ node_off,
                         const int64_t* __restrict__ adj_ptr, const int32_t* __restrict__ adj,
                         const int64_t* __restrict__ node_base, const double* __restrict__ vals,
                         const float* __restrict__ vals32, const double* __restrict__ inv_diag,
                         const double* __restrict__ f, double* u, double* r, double* p,
                         double* q, const double* __restrict__ tol,
                         const int64_t* __restrict__ max_iter, int64_t* __restrict__ out_it,
                         double* __restrict__ out_res, int32_t* __restrict__ out_status,
                         int64_t* __restrict__ out_fp32_it, double* __restrict__ u_sv,
                         double* __restrict__ r_sv, double* __restrict__ p_sv) {
    namespace cgx = cooperative_groups;

    cgx::cluster_group cluster = cgx::this_cluster();
    const int crank = int(cluster.block_rank());
    __shared__ double sh[32];
    __shared__ double part[5];  // A: p.q | B: r.r, r.z | T: true r.r, r.z
    __shared__ double tot[2];
    const int gl = threadIdx.x & (G - 1);
    const int64_t warp_nodes = 32 / G;
    const int64_t step = int64_t(BS / 32) * warp_nodes;
    // publish this CTA's block total(s) in part[s0..s0+nv), barrier, sum
    // over the cluster's ranks in rank order
    auto reduce = [&](int s0, int nv) {
        cluster.sync();
        if (threadIdx.x == 0)
            for (int s = 0; s < nv; ++s) {
                double t = 0.0;
                for (int c = 0; c < CS; ++c) t += *cluster.map_shared_rank(&part[s0 + s], c);
                tot[s] = t;
            }
        __syncthreads();
    };
    const int n_clusters = int(gridDim.x) / CS;
    for (int k = int(blockIdx.x) / CS; k < count; k += n_clusters) {
        cluster.sync();  // the previous member's partials are read by now
        const int inst = order[k];
        const int64_t N0 = node_off[inst], N1 = node_off[inst + 1];
        const int64_t n0 = N0 + (N1 - N0) * crank / CS, n1 = N0 + (N1 - N0) * (crank + 1) / CS;
        const int64_t r0 = n0 * ND, r1 = n1 * ND;
        const double tl = tol[inst], tau = mixed_switch_residual(tl);
        const int64_t mi = max_iter[inst];
        double lrr = 0.0, lrz = 0.0;
        for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
            const double ri = f[row];
            u[row] = 0.0;
            r[row] = ri;
            const double zi = ri * inv_diag[row];
            p[row] = zi;
            lrr += ri * ri;
            lrz += ri * zi;
        }
        {
            const double a = block_sum(lrr, sh), b = block_sum(lrz, sh);
            if (threadIdx.x == 0) {
                part[1] = a;
                part[2] = b;
            }
        }
        reduce(1, 2);
        double rr = tot[0], rz = tot[1];
        const double bnorm = sqrt(rr);
        int64_t it = 0, fp32_it = 0;
        int status = (bnorm == 0.0) ? PCG_CONVERGED : PCG_RUNNING;
        double res = (bnorm == 0.0) ? 0.0 : 1.0;
        bool exact = true, switched = false, save = false;
        int64_t cap_end = 0;
        double rz_sv = 0.0, rr_sv = 0.0;
        while (status == PCG_RUNNING) {
            // A: q = K p on own nodes (neighbours' p from L2), p.q
            double dot = 0.0;
            for (int64_t nb = n0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < n1; nb += step) {
                const int64_t i = nb + ((threadIdx.x & 31) / G);
                double acc[ND];
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[da] = 0.0;
                if (i < n1) {
                    if (exact)
                        node_rows_cg<ND, G, double, double>(adj_ptr, adj, node_base, vals, p, i,
                                                            gl, acc);
                    else
                        node_rows_cg<ND, G, float, double>(adj_ptr, adj, node_base, vals32, p, i,
                                                           gl, acc);
                }
#pragma unroll
                for (int da = 0; da < ND; ++da) acc[da] = group_sum<G>(acc[da]);
                if (i < n1 && gl == 0) {
#pragma unroll
                    for (int da = 0; da < ND; ++da) {
                        q[i * ND + da] = acc[da];
                        dot += p[i * ND + da] * acc[da];
                    }
                }
            }
            {
                const double a = block_sum(dot, sh);
                if (threadIdx.x == 0) part[0] = a;
            }
            reduce(0, 1);
            const double pap = tot[0];
            if (!(pap > 0.0)) {  // pap <= 0 or NaN: breakdown
                status = PCG_BREAKDOWN;
                it += 1;
                res = sqrt(rr) / bnorm;
                break;
            }
            const double alpha = rz / pap;
            // B: u, r on own rows; r.r, r.z
            lrr = 0.0;
            lrz = 0.0;
            for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                u[row] += alpha * p[row];
                const double ri = r[row] - alpha * q[row];
                r[row] = ri;
                const double zi = ri * inv_diag[row];
                lrr += ri * ri;
                lrz += ri * zi;
            }
            {
                const double a = block_sum(lrr, sh), b = block_sum(lrz, sh);
                if (threadIdx.x == 0) {
                    part[1] = a;
                    part[2] = b;
                }
            }
            reduce(1, 2);
            rr = tot[0];
            double rz_new = tot[1];
            it += 1;
            if (!exact) ++fp32_it;
            res = sqrt(rr) / bnorm;
            if constexpr (MIXED) {
                bool rollback = false;
                if (exact && !switched && res <= tau && res > tl) {
                    exact = false;  // the FP32 operator from here, same search directions
                    switched = true;
                    save = true;       // this iterate is kept for a rollback
                    cap_end = 2 * it;  // FP32 budget: as many iterations as the FP64 phase
                } else if (!exact && it >= cap_end && res > tl) {
                    rollback = true;  // budget spent
                }
                if (res <= tl && !exact) {
                    // T: r = f - K64 u on own nodes (neighbours' u from L2)
                    double trr = 0.0, trz = 0.0;
                    for (int64_t nb = n0 + int64_t(threadIdx.x >> 5) * warp_nodes; nb < n1;
                         nb += step) {
                        const int64_t i = nb + ((threadIdx.x & 31) / G);
                        double hi[ND], lo[ND];
#pragma unroll
                        for (int da = 0; da < ND; ++da) hi[da] = lo[da] = 0.0;
                        if (i < n1)
                            node_rows_dd<ND, G, true>(adj_ptr, adj, node_base, vals, u, i, gl,
                                                      hi, lo);
#pragma unroll
                        for (int da = 0; da < ND; ++da) group_sum_dd<G>(hi[da], lo[da]);
                        if (i < n1 && gl == 0) {
#pragma unroll
                            for (int da = 0; da < ND; ++da) {
                                const int64_t row = i * ND + da;
                                const double ri = dd_residual(f[row], hi[da], lo[da]);
                                r[row] = ri;
                                trr += ri * ri;
                                trz += ri * (ri * inv_diag[row]);
                            }
                        }
                    }
                    {
                        const double a = block_sum(trr, sh), b = block_sum(trz, sh);
                        if (threadIdx.x == 0) {
                            part[3] = a;
                            part[4] = b;
                        }
                    }
                    reduce(3, 2);
                    rr = tot[0];
                    rz_new = tot[1];
                    res = sqrt(rr) / bnorm;
                    // the true residual decides; short of tol, the FP32
                    // phase is undone
                    rollback = res > tl;
                }
                if (rollback) {
                    // back to the iterate of the switch, on the FP64 operator
                    // from there: the FP32 phase's updates are discarded
                    for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                        u[row] = u_sv[row];
                        r[row] = r_sv[row];
                        p[row] = p_sv[row];
                    }
                    rz = rz_sv;
                    rr = rr_sv;
                    res = sqrt(rr) / bnorm;
                    exact = true;
                    cluster.sync();  // restored p rows read by the neighbours' SpMV
                    if (it >= mi) {
                        status = PCG_MAXITER;
                        break;
                    }
                    continue;
                }
            }
            if (res <= tl) {
                status = PCG_CONVERGED;
                break;
            }
            if (it >= mi) {
                status = PCG_MAXITER;
                break;
            }
            const double beta = rz_new / rz;
            rz = rz_new;
            // C: p = z + beta p on own rows (kept at the switch), then the
            // cluster barrier that makes them visible to the neighbours' SpMV
            for (int64_t row = r0 + threadIdx.x; row < r1; row += BS) {
                const double pi = r[row] * inv_diag[row] + beta * p[row];
                p[row] = pi;
                if (MIXED && save) {
                    u_sv[row] = u[row];
                    r_sv[row] = r[row];
                    p_sv[row] = pi;
                }
            }
            if (MIXED && save) {
                rz_sv = rz;
                rr_sv = rr;
                save = false;
            }
            cluster.sync();
        }
        if (crank == 0 && threadIdx.x == 0) {
            out_it[inst] = it;
            out_res[inst] = res;
            out_status[inst] = status;
            if (out_fp32_it) out_fp32_it[inst] = fp32_it;
        }
    }
    // no CTA leaves while another may still read its partials
    cluster.sync();
}

// Nonzeros of each member: node_base at the members' node offsets.
__global__ void member_nnz_kernel(int count, const int64_t* __restrict__ node_off,
                                  const int64_t* __restrict__ node_base,
                                  int64_t* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < count) out[k] = node_base[node_off[k + 1]] - node_base[node_off[k]];
}

// Extreme |K_ii| of each instance (its cond_estimate), one CTA per instance.
__global__ void instance_diag_kernel(int ndof, const int64_t* __restrict__ node_off,
                                     const int32_t* __restrict__ diag_pos,
                                     const double* __restrict__ vals, double* __restrict__ hi,
                                     double* __restrict__ lo) {
    __shared__ double shi[256], slo[256];
    const int inst = blockIdx.x;
    const int64_t r0 = node_off[inst] * ndof, r1 = node_off[inst + 1] * ndof;
    double h = 0.0, l = INFINITY;
    for (int64_t row = r0 + threadIdx.x; row < r1; row += blockDim.x) {
        const double a = fabs(vals[diag_pos[row]]);
        h = fmax(h, a);
        l = fmin(l, a);
    }
    shi[threadIdx.x] = h;
    slo[threadIdx.x] = l;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) {
            shi[threadIdx.x] = fmax(shi[threadIdx.x], shi[threadIdx.x + off]);
            slo[threadIdx.x] = fmin(slo[threadIdx.x], slo[threadIdx.x + off]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        hi[inst] = shi[0];
        lo[inst] = slo[0];
    }
}

// ------------------------------------------------------------ host side
int pick_group(double mean_row) {
    if (mean_row < 6) return 2;
    if (mean_row < 12) return 4;
    if (mean_row < 40) return 8;
    if (mean_row < 96) return 16;
    return 32;
}

unsigned grid_vec(const svx_ctx* ctx, int64_t n) {
    int64_t need = (n + BLOCK - 1) / BLOCK;
    int64_t cap = int64_t(ctx->sm_count) * 8;
    return unsigned(std::max<int64_t>(1, std::min(need, cap)));
}

// Lanes per node for the node-block kernels: the smallest of 8 / 16 / 32
// that covers the largest node degree (27 for interior C3D8 nodes).
// Lanes per node of the node-block kernels: enough to cover the neighbour
// blocks once for 2D and 3D rows; one dof per node (conduction) gives a
// lane a single value per neighbour, so 8 lanes take several neighbours
// each and a warp 4 nodes (the 480 x 48 x 48 conduction block, 27
// neighbours: 32 lanes per node left the SpMV latency bound at one node a
// warp).
int pick_node_group(int max_deg, int nd) {
    // SVX_NODE_LANES (8, 16 or 32) forces the choice, for measurements
    static const int forced = [] {
        const char* e = std::getenv("SVX_NODE_LANES");
        const int v = e ? std::atoi(e) : 0;
        return (v == 8 || v == 16 || v == 32) ? v : 0;
    }();
    if (forced) return forced;
    if (nd == 1 || max_deg <= 8) return 8;
    if (max_deg <= 16) return 16;
    return 32;
}

unsigned grid_nodes(const svx_ctx* ctx, int64_t n_nodes, int G) {
    int64_t per_block = BLOCK / G;
    int64_t need = (n_nodes + per_block - 1) / per_block;
    int64_t cap = int64_t(ctx->sm_count) * NODE_BLOCKS_PER_SM;
    return unsigned(std::max<int64_t>(1, std::min(need, cap)));
}

#define SVX_NODE_DISPATCH(ND_, G_, KERNEL_CALL)                         \
    do {                                                                \
        if ((ND_) == 3) {                                               \
            if ((G_) == 8) { constexpr int ND = 3, GG = 8; KERNEL_CALL; } \
            else if ((G_) == 16) { constexpr int ND = 3, GG = 16; KERNEL_CALL; } \
            else { constexpr int ND = 3, GG = 32; KERNEL_CALL; }        \
        } else if ((ND_) == 2) {                                        \
            if ((G_) == 8) { constexpr int ND = 2, GG = 8; KERNEL_CALL; } \
            else if ((G_) == 16) { constexpr int ND = 2, GG = 16; KERNEL_CALL; } \
            else { constexpr int ND = 2, GG = 32; KERNEL_CALL; }        \
        } else {                                                        \
            if ((G_) == 8) { constexpr int ND = 1, GG = 8; KERNEL_CALL; } \
            else if ((G_) == 16) { constexpr int ND = 1, GG = 16; KERNEL_CALL; } \
            else { constexpr int ND = 1, GG = 32; KERNEL_CALL; }        \
        }                                                               \
    } while (0)

template <class M, class V>
void launch_spmv_node_dot(const svx_op* op, int G, unsigned grid, cudaStream_t st,
                          const M* vals, const V* p, V* q, double* partials, PcgScalars* s) {
    const Pattern& P = op->pat;
    SVX_NODE_DISPATCH(op->ndof, G,
                      (spmv_node_dot_kernel<ND, GG, M, V><<<grid, BLOCK, 0, st>>>(
                          op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, vals, p, q,
                          partials, s)));
}

// One PCG run in value type V (the vectors and K) with solution type U.
template <class M, class V, class U>
struct PcgRun {
    svx_ctx* ctx;
    const svx_op* op;
    int64_t n;
    int G;
    unsigned grid_r, grid_v;
    const M* vals;
    const V* inv_diag;
    U* u;
    V *r, *p, *q;
    V* p2 = nullptr;  // the persistent kernel's second search-direction buffer (zeroed)
    double* partials;
    PcgScalars* s;
    PcgScalars* h_s;  // pinned
    HexWork* hex = nullptr;  // FP64 C3D8: K applied element by element
    BrickWork* brick = nullptr;  // FP64 C3D8: the persistent form on bricks

    void enqueue_iteration(cudaStream_t st) {
        if constexpr (std::is_same<M, double>::value) {
            if (hex) {
                hex_iteration(op, *hex, st, inv_diag, u, r, p, s);
                return;
            }
        }
        if constexpr (std::is_same<M, float>::value) {
            if (vals == op->vals32.p && op->vals32q.p)
                launch_spmv_fp32(op, G, grid_r, st, p, q, partials, s);
            else
                launch_spmv_node_dot<M, V>(op, G, grid_r, st, vals, p, q, partials, s);
        } else {
            launch_spmv_node_dot<M, V>(op, G, grid_r, st, vals, p, q, partials, s);
        }
        update_kernel<V, U><<<grid_v, BLOCK, 0, st>>>(n, u, r, p, q, inv_diag, partials, s);
        p_update_kernel<V><<<grid_v, BLOCK, 0, st>>>(n, p, r, inv_diag, s);
    }

    // Persistent form: cooperative launches of up to `chunk` iterations each
    // until the device status leaves RUNNING.  Returns -1 when a cooperative
    // launch is not possible on this device (the caller falls back to the
    // graph form).
    int iterate_persistent(int chunk) {
        cudaStream_t st = ctx->stream;
        const int ND = op->ndof;
        const bool narrow = op->pat.max_deg <= 8;
        auto pick = [&](bool sadj) -> void* {
            if (ND == 3) {
                if (sadj)
                    return narrow ? (void*)pcg_persistent_kernel<3, 8, M, V, U, true>
                                  : (void*)pcg_persistent_kernel<3, SVX_PG3D, M, V, U, true>;
                return narrow ? (void*)pcg_persistent_kernel<3, 8, M, V, U, false>
                              : (void*)pcg_persistent_kernel<3, SVX_PG3D, M, V, U, false>;
            }
            if (ND == 1) {  // one dof per node (conduction)
                if (sadj)
                    return narrow ? (void*)pcg_persistent2_kernel<1, 8, M, V, U, true>
                                  : (void*)pcg_persistent2_kernel<1, 16, M, V, U, true>;
                return narrow ? (void*)pcg_persistent2_kernel<1, 8, M, V, U, false>
                              : (void*)pcg_persistent2_kernel<1, 16, M, V, U, false>;
            }
            if (sadj)
                return narrow ? (void*)pcg_persistent2_kernel<2, 8, M, V, U, true>
                              : (void*)pcg_persistent2_kernel<2, 16, M, V, U, true>;
            return narrow ? (void*)pcg_persistent2_kernel<2, 8, M, V, U, false>
                          : (void*)pcg_persistent2_kernel<2, 16, M, V, U, false>;
        };
        void* fn = pick(false);
        int coop = 0, bps = 0;
        SVX_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
        SVX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, PBLOCK, 0));
        if (!coop || bps <= 0) return -1;
        const unsigned int B = unsigned(std::min(bps, PBLOCKS_PER_SM) * ctx->sm_count);
        // each block's adjacency in shared memory, when it fits with as many
        // blocks per SM
        int nodes_cap = int((op->n_nodes + B - 1) / B);
        size_t smem = shared_adj_bytes(nodes_cap, op->pat.max_deg);
        const long long adj_max = ctx->shared_adj_max >= 0 ? ctx->shared_adj_max : SHARED_ADJ_MAX;
        if (smem <= size_t(adj_max)) {
            void* fs = pick(true);
            if (smem > 48 * 1024)
                SVX_CUDA(cudaFuncSetAttribute(fs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              int(smem)));
            int bps_s = 0;
            SVX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps_s, fs, PBLOCK, smem));
            if (bps_s >= std::min(bps, PBLOCKS_PER_SM))
                fn = fs;
            else
                smem = 0;
        } else {
            smem = 0;
        }
        DBuf<double> part_a, part_b;
        DBuf<GridBarrier> gb;
        part_a.alloc(ctx->pool, B + 1);
        part_b.alloc(ctx->pool, 2 * size_t(B) + 2);
        gb.alloc(ctx->pool, 1);
        SVX_CUDA(cudaMemsetAsync(gb.p, 0, sizeof(GridBarrier), st));
        int64_t n_nodes = op->n_nodes;
        const int64_t* a_ptr = op->pat.adj_ptr.p;
        const int32_t* a_idx = op->pat.adj.p;
        const int64_t* nbase = op->pat.node_base.p;
        GridBarrier* gbp = gb.p;
        double* pa = part_a.p;
        double* pb = part_b.p;
        if (!p2) return -1;
        void* args[] = {&n_nodes, (void*)&a_ptr, (void*)&a_idx, (void*)&nbase, (void*)&vals,
                        (void*)&inv_diag, (void*)&u, (void*)&r, (void*)&p, (void*)&p2,
                        (void*)&q, (void*)&pa, (void*)&pb, (void*)&s, (void*)&gbp,
                        (void*)&chunk, (void*)&nodes_cap};
        SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
        SVX_CUDA(cudaStreamSynchronize(st));
        const long long launches_max = h_s->max_iter / chunk + 2;
        GridBarrier hgb{};
        int status = h_s->status;
        for (long long launch = 0; status == PCG_RUNNING; ++launch) {
            if (launch >= launches_max)
                throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                "PCG status did not leave RUNNING within max_iter"};
            // the barrier's arrival count starts from zero in every launch
            SVX_CUDA(cudaMemsetAsync(&gbp->count, 0, sizeof(unsigned int), st));
            SVX_CUDA(cudaLaunchCooperativeKernel(fn, dim3(B), dim3(PBLOCK), args, smem, st));
            g_launches.fetch_add(1, std::memory_order_relaxed);
            SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaMemcpyAsync(&hgb, gbp, sizeof(GridBarrier), cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
            if (hgb.error)
                throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                "persistent PCG: a grid barrier wait ran out (blocks not "
                                "co-resident)"};
            status = h_s->status;
        }
        return status;
    }

    // Shared-memory persistent form (pcg_smem_kernel, plain FP64 only):
    // cooperative launches of up to `chunk` iterations each until the
    // device status leaves RUNNING.  Returns -1 without launching when a
    // block's rows and adjacency do not fit its shared memory (the caller
    // then runs the register-vector persistent kernel).
    // valsT: K in the transposed node-block layout (transposed_values)
    int iterate_smem(int chunk, const M* valsT, int form = -1) {
        if constexpr (!std::is_same<V, U>::value) {
            (void)chunk;
            (void)valsT;
            return -1;
        } else {
            cudaStream_t st = ctx->stream;
            const int ND = op->ndof;
            // 8 lanes per node and one node a lane group per warp step (4
            // nodes a warp), whatever the degree: each lane walks 3-4 of a
            // C3D8 node's 27 neighbour blocks.  Measured against 32 lanes
            // with 4 nodes a warp step (16 for 2D): the 160x16x16 C3D8
            // cantilever 25.4 -> 19.5 us an iteration, its heterogeneous
            // twin 25.4 -> 19.5, the 40x4x4 hex 7.54 -> 7.10, the 200x20
            // CPS4 cantilever 7.26 -> 6.42 (2 and 4 nodes a lane group were
            // slower with 8 lanes).  SVX_PCG_LANES (16 or 32) and
            // SVX_PCG_UNROLL override it for measurements.
            const bool narrow = op->pat.max_deg <= 8;
            const int G = ctx->pcg_lanes == 32 && ND == 3 && !narrow ? 32
                          : ctx->pcg_lanes == 16 && ND != 3 && !narrow ? 16
                                                                        : 8;
            int coop = 0;
            SVX_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
            if (!coop) return -1;
            // one block of 512 threads per SM: fewer arrivals per grid barrier
            // measured faster than 1,024-thread or two-block shapes (with 8
            // lanes a node 1,024 threads fit 64 registers without spills and
            // still ran 21.5 against 19.6 us an iteration on the 160x16x16
            // C3D8 cantilever).  The
            // two-barrier form (ALG 1) gathers two vectors per neighbour
            // value: it wins for 2D and small 3D systems (with 8 lanes a
            // node: the 200x20 CPS4 cantilever 7.81 -> 6.47 us an
            // iteration, the 40x4x4 hex 8.37 -> 7.20) and loses at the
            // 160x16x16 C3D8 size (19.6 -> 25.1 us); SVX_PCG_ALG and
            // SVX_PCG_UNROLL override the choice for measurements.
            constexpr int PB = 512;
            const unsigned int B = unsigned(ctx->sm_count);
            const int nodes_cap = int((op->n_nodes + B - 1) / B);
            const int alg =
                form >= 0           ? form
                : ctx->pcg_alg >= 0 ? ctx->pcg_alg : ((ND <= 2 || nodes_cap <= 64) ? 1 : 0);
            const int unroll = ctx->pcg_unroll > 0 ? ctx->pcg_unroll : 1;
            auto kernel_for = [&]() -> void* {
#define SVX_SMEM_PICK(ND_, G_)                                                           \
    if (ND == ND_ && G == G_) {                                                          \
        if (alg == 0) {                                                                  \
            if (unroll == 1) return (void*)pcg_smem_kernel<ND_, G_, PB, 1, 0, 1, M, V>;        \
            if (unroll == 2) return (void*)pcg_smem_kernel<ND_, G_, PB, 1, 0, 2, M, V>;        \
            return (void*)pcg_smem_kernel<ND_, G_, PB, 1, 0, 4, M, V>;                         \
        }                                                                                \
        if (unroll == 1) return (void*)pcg_smem_kernel<ND_, G_, PB, 1, 1, 1, M, V>;            \
        if (unroll == 2) return (void*)pcg_smem_kernel<ND_, G_, PB, 1, 1, 2, M, V>;            \
        return (void*)pcg_smem_kernel<ND_, G_, PB, 1, 1, 4, M, V>;                             \
    }
                if constexpr (std::is_same<M, float>::value) {
                    // FP32 operators: the default shapes (FP64 vectors, the mixed
                    // form, three barriers only)
                    if (ND == 3 && std::is_same<V, double>::value)
                        return (void*)pcg_smem_kernel<3, 8, PB, 1, 0, 1, M, V>;
                    if (ND == 3)
                        return alg == 0 ? (void*)pcg_smem_kernel<3, 8, PB, 1, 0, 1, M, V>
                                        : (void*)pcg_smem_kernel<3, 8, PB, 1, 1, 1, M, V>;
                    if (ND == 2 && std::is_same<V, float>::value)
                        return (void*)pcg_smem_kernel<2, 8, PB, 1, 1, 1, M, V>;
                    return nullptr;
                } else {
                    SVX_SMEM_PICK(3, 32)
                    SVX_SMEM_PICK(3, 8)
                    SVX_SMEM_PICK(2, 16)
                    SVX_SMEM_PICK(2, 8)
                    SVX_SMEM_PICK(1, 16)
                    SVX_SMEM_PICK(1, 8)
                }
#undef SVX_SMEM_PICK
                return nullptr;
            };
            int max_smem = 0;
            SVX_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                            ctx->device));
            void* fn = kernel_for();
            if (!fn) return -1;
            cudaFuncAttributes fa{};
            SVX_CUDA(cudaFuncGetAttributes(&fa, fn));
            const size_t avail = size_t(max_smem) - std::min(size_t(max_smem), fa.sharedSizeBytes);
            const size_t base = smem_pcg_bytes(nodes_cap, ND, op->pat.max_deg, 0, sizeof(V));
            if (base > avail) return -1;
            // the three-barrier form's staging window
            int stage = (alg == 0 && ctx->pcg_stage) ? STAGE_NODES_PER_NODE * nodes_cap : 0;
            const size_t smem = smem_pcg_bytes(nodes_cap, ND, op->pat.max_deg, stage, sizeof(V));
            if (smem > avail) return -1;
            SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          int(smem)));
            int bps = 0;
            SVX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, PB, smem));
            if (bps < 1) return -1;
            const int pb = PB;
            if (!fn) return -1;
            DBuf<double> part;
            DBuf<V> z;
            DBuf<GridBarrier> gb;
            part.alloc(ctx->pool, 4 * size_t(B) + 2);  // two slots of pairs
            z.alloc(ctx->pool, n + 1);
            gb.alloc(ctx->pool, 1);
            SVX_CUDA(cudaMemsetAsync(gb.p, 0, sizeof(GridBarrier), st));
            int64_t n_nodes = op->n_nodes;
            const int64_t* a_ptr = op->pat.adj_ptr.p;
            const int32_t* a_idx = op->pat.adj.p;
            const int64_t* nbase = op->pat.node_base.p;
            GridBarrier* gbp = gb.p;
            double* pp = part.p;
            V* zp = z.p;
            int first = 1;
            int max_deg = std::max(op->pat.max_deg, 1);
            if (!p2) return -1;
            void* args[] = {&n_nodes, (void*)&a_ptr, (void*)&a_idx, (void*)&nbase,
                            (void*)&valsT, (void*)&inv_diag, (void*)&u, (void*)&r, (void*)&p,
                            (void*)&p2, (void*)&zp, (void*)&pp, (void*)&s, (void*)&gbp,
                            (void*)&chunk, (void*)&nodes_cap, (void*)&max_deg, (void*)&stage,
                            (void*)&first};
            SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
            const long long launches_max = h_s->max_iter / chunk + 2;
            GridBarrier hgb{};
            int status = h_s->status;
            for (long long launch = 0; status == PCG_RUNNING; ++launch) {
                if (launch >= launches_max)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "PCG status did not leave RUNNING within max_iter"};
                SVX_CUDA(cudaMemsetAsync(&gbp->count, 0, sizeof(unsigned int), st));
                SVX_CUDA(cudaLaunchCooperativeKernel(fn, dim3(B), dim3(pb), args, smem, st));
                g_launches.fetch_add(1, std::memory_order_relaxed);
                first = 0;
                SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost,
                                         st));
                SVX_CUDA(cudaMemcpyAsync(&hgb, gbp, sizeof(GridBarrier), cudaMemcpyDeviceToHost,
                                         st));
                SVX_CUDA(cudaStreamSynchronize(st));
                if (hgb.error)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "persistent PCG: a grid barrier wait ran out (blocks not "
                                    "co-resident)"};
                status = h_s->status;
            }
            return status;
        }
    }

    // The persistent form of one dof a node (pcg_scalar_kernel).  Returns -1
    // without launching when the rows do not fit its slices, a block's vectors
    // its shared memory or the slices the device.
    int iterate_scalar(int chunk) {
        if constexpr (std::is_same<M, double>::value && std::is_same<V, double>::value &&
                      std::is_same<U, double>::value) {
            cudaStream_t st = ctx->stream;
            constexpr int PB = SCALAR_THREADS;
            const int width = std::max(op->pat.max_deg, 1);
            int coop = 0;
            SVX_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
            if (!coop || op->ndof != 1 || width > SCALAR_MAX_DEG) return -1;
            const int64_t slices = (n + 31) / 32, padded = slices * width * 32;
            if (padded > std::max(2 * op->pat.nnz, SCALAR_SMALL)) return -1;
            const unsigned int B = unsigned(std::min<int64_t>(ctx->sm_count, slices));
            int cap = int((slices + B - 1) / B) * 32;
            size_t smem = size_t(cap) * 6 * sizeof(double);
            if (smem > SCALAR_SMEM) return -1;
            // the columns stay in shared memory where they fit
            int cols_here = smem + size_t(cap) * width * sizeof(int32_t) <= SCALAR_SMEM;
            if (cols_here) smem += size_t(cap) * width * sizeof(int32_t);
            void* fn = (void*)pcg_scalar_kernel<PB>;
            SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          int(SCALAR_SMEM)));
            DBuf<double> part, sv;
            DBuf<double2> zp;
            DBuf<int32_t> sc;
            DBuf<GridBarrier> gb;
            part.alloc(ctx->pool, 4 * size_t(B) + 2);
            gb.alloc(ctx->pool, 1);
            try {
                zp.alloc(ctx->pool, n);
                sv.alloc(ctx->pool, padded);
                sc.alloc(ctx->pool, padded);
            } catch (const ModelFail& f) {  // a full device: the rows stay where they are
                if (f.code != SVX_OOM) throw;
                return -1;
            }
            SVX_CUDA(cudaMemsetAsync(gb.p, 0, sizeof(GridBarrier), st));
            // rows past n repeat the last node with a zero: any finite pair will do there
            slice_rows_kernel<<<unsigned((slices * 32 + BLOCK - 1) / BLOCK), BLOCK, 0, st>>>(
                n, width, op->pat.adj_ptr.p, op->pat.adj.p, op->pat.node_base.p, vals, sv.p, sc.p);
            SVX_LAUNCH_CHECK();
            int64_t rows = n;
            int w = width, first = 1;
            GridBarrier* gbp = gb.p;
            void* args[] = {&rows, &w, &sv.p, &sc.p, (void*)&inv_diag, (void*)&u, (void*)&r,
                            &zp.p, &part.p, (void*)&s, (void*)&gbp, (void*)&chunk, &cap,
                            &cols_here, &first};
            SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
            const long long launches_max = h_s->max_iter / chunk + 2;
            GridBarrier hgb{};
            int status = h_s->status;
            for (long long launch = 0; status == PCG_RUNNING; ++launch) {
                if (launch >= launches_max)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "PCG status did not leave RUNNING within max_iter"};
                SVX_CUDA(cudaMemsetAsync(&gbp->count, 0, sizeof(unsigned int), st));
                SVX_CUDA(cudaLaunchCooperativeKernel(fn, dim3(B), dim3(PB), args, smem, st));
                g_launches.fetch_add(1, std::memory_order_relaxed);
                first = 0;
                SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost,
                                         st));
                SVX_CUDA(cudaMemcpyAsync(&hgb, gbp, sizeof(GridBarrier), cudaMemcpyDeviceToHost,
                                         st));
                SVX_CUDA(cudaStreamSynchronize(st));
                if (hgb.error)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "persistent PCG: a grid barrier wait ran out (blocks not "
                                    "co-resident)"};
                status = h_s->status;
            }
            return status;
        } else {
            (void)chunk;
            return -1;
        }
    }

    // The persistent form on bricks of elements (svx_brick.cu): cooperative
    // launches of up to `chunk` iterations each.
    int iterate_brick(int chunk) {
        if constexpr (std::is_same<M, double>::value && std::is_same<V, double>::value &&
                      std::is_same<U, double>::value) {
            cudaStream_t st = ctx->stream;
            SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
            const long long launches_max = h_s->max_iter / chunk + 2;
            int status = h_s->status;
            GridBarrier hgb{};
            for (long long launch = 0; status == PCG_RUNNING; ++launch) {
                if (launch >= launches_max)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "PCG status did not leave RUNNING within max_iter"};
                brick_grid_launch(ctx, op, *brick, u, r, p, s, chunk);
                SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost,
                                         st));
                SVX_CUDA(cudaMemcpyAsync(&hgb, brick->gb.p, sizeof(GridBarrier),
                                         cudaMemcpyDeviceToHost, st));
                SVX_CUDA(cudaStreamSynchronize(st));
                if (hgb.error)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "persistent PCG: a grid barrier wait ran out (blocks not "
                                    "co-resident)"};
                status = h_s->status;
            }
            return status;
        } else {
            (void)chunk;
            return -1;
        }
    }

    // Runs until the device status leaves RUNNING; returns the status.
    int iterate(int check_every) {
        cudaStream_t st = ctx->stream;
        if constexpr (std::is_same<M, double>::value && std::is_same<V, double>::value) {
            if (hex) hex_start(op, *hex, st, p);
        }
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        SVX_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        for (int k = 0; k < check_every; ++k) enqueue_iteration(st);
        cudaError_t ce = cudaStreamEndCapture(st, &graph);
        if (ce != cudaSuccess) throw CudaFail{ce, "cudaStreamEndCapture"};
        ce = cudaGraphInstantiate(&exec, graph, 0);
        if (ce != cudaSuccess) {
            cudaGraphDestroy(graph);
            throw CudaFail{ce, "cudaGraphInstantiate"};
        }
        int status = PCG_RUNNING;
        try {
            // the device stops at max_iter; the host bound only guards
            // against a status that never leaves RUNNING
            SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
            const long long launches_max = h_s->max_iter / check_every + 2;
            for (long long launch = 0;; ++launch) {
                if (launch >= launches_max)
                    throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                                    "PCG status did not leave RUNNING within max_iter"};
                SVX_CUDA(cudaGraphLaunch(exec, st));
                g_launches.fetch_add(3LL * check_every, std::memory_order_relaxed);
                SVX_CUDA(cudaMemcpyAsync(h_s, s, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
                SVX_CUDA(cudaStreamSynchronize(st));
                status = h_s->status;
                if (status != PCG_RUNNING) break;
            }
        } catch (...) {
            cudaGraphExecDestroy(exec);
            cudaGraphDestroy(graph);
            throw;
        }
        cudaGraphExecDestroy(exec);
        cudaGraphDestroy(graph);
        return status;
    }
};

static_assert(sizeof(PcgScalars) <= 256, "the context's pinned scalar slot holds 256 bytes");

struct PinnedScalars {
    PcgScalars* h = nullptr;
    // the context's page-locked slot: no cudaMallocHost / cudaFreeHost per
    // solve (each can stall for milliseconds while other processes hold
    // the driver)
    explicit PinnedScalars(svx_ctx* ctx) : h(static_cast<PcgScalars*>(ctx->h_scalars)) {}
};

// Iterations per persistent launch: a few to tens of milliseconds of work,
// so the host sees progress and a long solve is not one unbounded launch.
// Systems whose FP64 K does not fit in L2 (or above GRAPH_MIN_NNZ) iterate
// with the three standalone kernels in a CUDA graph instead of the
// persistent kernel: K streams from HBM every iteration, launch gaps are
// noise, and the standalone node SpMV (5 blocks of 256 threads per SM,
// more loads in flight) runs at ~80% of the HBM copy peak.  While K fits in
// L2 the persistent kernel's absence of launch gaps and grid-wide state in
// shared memory win (the 160 x 16 x 16 C3D8 cantilever, K 83 MB: 19.5
// against 34.1 us an iteration); above it the graph form does (240 x 24 x 24,
// K 277 MB: 79.0 against 82.4 us; the 480 x 48 x 48 conduction block, K
// 250 MB: 11% more DOF-iterations per second over the whole solve).
constexpr int64_t GRAPH_MIN_NNZ = 50000000;

bool use_graph_form(const svx_ctx* ctx, const svx_op* op) {
    if (ctx->graph_min_nnz >= 0) return op->pat.nnz > ctx->graph_min_nnz;
    return op->pat.nnz > GRAPH_MIN_NNZ ||
           (ctx->l2_bytes > 0 && op->pat.nnz * int64_t(sizeof(double)) > ctx->l2_bytes);
}

int persistent_chunk(int64_t nnz) {
    if (nnz > 100000000) return 64;
    if (nnz > 10000000) return 256;
    return 1024;
}

int auto_check_every(int64_t n, int64_t nnz) {
    // ~30 us per iteration at C3D8 3.5M dofs vs ~5 us at 10k dofs: keep one
    // host check per few hundred microseconds of device work.
    (void)n;
    if (nnz > 50000000) return 8;
    if (nnz > 5000000) return 32;
    return 64;
}

}  // namespace

// The transposed copy of K the shared-memory PCG kernel streams (vectors of
// one dof per node need none: both layouts are the same).
template <class M>
static const M* transposed(svx_ctx* ctx, const svx_op* op, const DBuf<M>& vals, DBuf<M>& out) {
    if (op->ndof == 1) return vals.p;
    if (!out.p) {
        out.alloc(ctx->pool, op->pat.nnz + 1);
        const int64_t threads = op->n_nodes * op->ndof * op->ndof;
        const unsigned grid = unsigned(std::max<int64_t>(1, (threads + BLOCK - 1) / BLOCK));
        const Pattern& P = op->pat;
        if (op->ndof == 3)
            transpose_blocks_kernel<3, M><<<grid, BLOCK, 0, ctx->stream>>>(
                op->n_nodes, P.adj_ptr.p, P.node_base.p, vals.p, out.p);
        else
            transpose_blocks_kernel<2, M><<<grid, BLOCK, 0, ctx->stream>>>(
                op->n_nodes, P.adj_ptr.p, P.node_base.p, vals.p, out.p);
        SVX_LAUNCH_CHECK();
    }
    return out.p;
}
const double* transposed_values(svx_ctx* ctx, svx_op* op) {
    return transposed(ctx, op, op->vals, op->valsT);
}

void build_fp32_operator(svx_ctx* ctx, svx_op* op) {
    if (op->vals32.p) return;
    op->vals32.alloc(ctx->pool, op->pat.nnz + 1);
    const int64_t threads = op->n_nodes * op->ndof * op->ndof;
    const unsigned grid = unsigned(std::max<int64_t>(1, (threads + BLOCK - 1) / BLOCK));
    const Pattern& P = op->pat;
    if (op->ndof == 3)
        compensated_fp32_kernel<3><<<grid, BLOCK, 0, ctx->stream>>>(
            op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, op->vals.p, op->vals32.p);
    else
        compensated_fp32_kernel<2><<<grid, BLOCK, 0, ctx->stream>>>(
            op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, op->vals.p, op->vals32.p);
    SVX_LAUNCH_CHECK();
    // a vectorised copy for the graph form's FP32 SpMV (3D, <= 32 neighbour
    // blocks a node); its offsets depend only on the pattern
    if (op->ndof != 3 || P.max_deg > 32 || op->n_nodes == 0 || !ctx->fp32_quads) return;
    {
        if (!op->baseq.p) {
            std::vector<int64_t> ap(size_t(op->n_nodes) + 1), base(size_t(op->n_nodes) + 1);
            SVX_CUDA(cudaMemcpyAsync(ap.data(), P.adj_ptr.p, ap.size() * sizeof(int64_t),
                                     cudaMemcpyDeviceToHost, ctx->stream));
            SVX_CUDA(cudaStreamSynchronize(ctx->stream));
            base[0] = 0;
            for (int64_t i = 0; i < op->n_nodes; ++i) {
                const int64_t d = ap[i + 1] - ap[i];
                base[i + 1] = base[i] + 9 * (d == 0 ? 4 : (d + 3) & ~int64_t(3));
            }
            op->baseq.alloc(ctx->pool, base.size());
            SVX_CUDA(cudaMemcpyAsync(op->baseq.p, base.data(), base.size() * sizeof(int64_t),
                                     cudaMemcpyHostToDevice, ctx->stream));
            op->n32q = base.back();
            op->adjq.alloc(ctx->pool, size_t(op->n32q / 9) + 4);
        }
        op->vals32q.alloc(ctx->pool, size_t(op->n32q) + 4);
        const int64_t threads = op->n_nodes * 9;
        quad_fp32_kernel<3><<<unsigned((threads + BLOCK - 1) / BLOCK), BLOCK, 0, ctx->stream>>>(
            op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, op->baseq.p, op->vals32.p,
            op->vals32q.p, op->adjq.p);
        SVX_LAUNCH_CHECK();
    }
}

// The graph form's FP32 SpMV: a vectorised kernel on its copy of the
// operator when one exists, the node-block kernel otherwise.
template <class V>
void launch_spmv_fp32(const svx_op* op, int G, unsigned grid, cudaStream_t st, const V* p, V* q,
                      double* partials, PcgScalars* s) {
    if (op->vals32q.p) {
        // one wave at this kernel's residency, never more blocks than the
        // caller's partials hold
        grid = unsigned(std::min<int64_t>(
                {int64_t(grid), int64_t(op->ctx->sm_count) * SPMV32Q_BLOCKS_PER_SM,
                 (op->n_nodes + BLOCK / 8 - 1) / (BLOCK / 8)}));
        spmv32q_node_dot_kernel<3, V><<<grid, BLOCK, 0, st>>>(op->n_nodes, op->baseq.p,
                                                               op->adjq.p, op->vals32q.p, p, q,
                                                               partials, s);
    } else {
        launch_spmv_node_dot<float, V>(op, G, grid, st, op->vals32.p, p, q, partials, s);
    }
}
template void launch_spmv_fp32<double>(const svx_op*, int, unsigned, cudaStream_t,
                                       const double*, double*, double*, PcgScalars*);
template void launch_spmv_fp32<float>(const svx_op*, int, unsigned, cudaStream_t, const float*,
                                      float*, double*, PcgScalars*);


std::atomic<long long> g_launches{0};

void time_iteration_kernels(svx_ctx* ctx, svx_op* op, int reps, double* ms4) {
    const int64_t n = op->n;
    cudaStream_t st = ctx->stream;
    DBuf<double> u, r, p, q, partials;
    DBuf<PcgScalars> s;
    u.alloc(ctx->pool, n + 1);
    r.alloc(ctx->pool, n + 1);
    p.alloc(ctx->pool, n + 1);
    q.alloc(ctx->pool, n + 1);
    const int G = pick_node_group(op->pat.max_deg, op->ndof);
    const unsigned grid_r = grid_nodes(ctx, op->n_nodes, G), grid_v = grid_vec(ctx, n);
    partials.alloc(ctx->pool, 2 * size_t(std::max(grid_r, grid_v)) + 2);
    s.alloc(ctx->pool, 1);
    // a running state that never stops: tol 0, unbounded budget
    PcgScalars init{};
    init.tol = 0.0;
    init.max_iter = (1LL << 62);
    init.bnorm = 1.0;
    init.status = PCG_RUNNING;
    SVX_CUDA(cudaMemcpyAsync(s.p, &init, sizeof(init), cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaMemcpyAsync(p.p, op->f.p, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    SVX_CUDA(cudaMemcpyAsync(r.p, op->f.p, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    SVX_CUDA(cudaMemsetAsync(u.p, 0, n * sizeof(double), st));
    auto timed = [&](auto&& launch) -> double {
        launch();  // warm
        SVX_CUDA(cudaEventRecord(ctx->ev[0], st));
        for (int k = 0; k < reps; ++k) launch();
        SVX_CUDA(cudaEventRecord(ctx->ev[1], st));
        SVX_CUDA(cudaEventSynchronize(ctx->ev[1]));
        float ms = 0.f;
        SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
        g_launches.fetch_add(reps + 1, std::memory_order_relaxed);
        return double(ms) / reps;
    };
    ms4[0] = timed([&] {
        launch_spmv_node_dot<double, double>(op, G, grid_r, st, op->vals.p, p.p, q.p, partials.p,
                                             s.p);
    });
    ms4[1] = timed([&] {
        update_kernel<double, double><<<grid_v, BLOCK, 0, st>>>(n, u.p, r.p, p.p, q.p,
                                                                op->inv_diag.p, partials.p, s.p);
    });
    ms4[2] = timed([&] {
        p_update_kernel<double><<<grid_v, BLOCK, 0, st>>>(n, p.p, r.p, op->inv_diag.p, s.p);
    });
    build_fp32_operator(ctx, op);
    ms4[3] = timed([&] {
        launch_spmv_fp32(op, G, grid_r, st, p.p, q.p, partials.p, s.p);
    });
    SVX_CUDA(cudaGetLastError());
}

void spmv_fp64(svx_ctx* ctx, const svx_op* op, const double* vals, const double* x, double* y) {
    const int G = pick_node_group(op->pat.max_deg, op->ndof);
    const unsigned grid = grid_nodes(ctx, op->n_nodes, G);
    cudaStream_t st = ctx->stream;
    const Pattern& P = op->pat;
    SVX_NODE_DISPATCH(op->ndof, G,
                      (spmv_node_kernel<ND, GG><<<grid, BLOCK, 0, st>>>(
                          op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, vals, x, y)));
    SVX_LAUNCH_CHECK();
}

int choose_spmv_group(const svx_op* op) {
    double mean = op->n > 0 ? double(op->pat.nnz) / double(op->n) : 1.0;
    return pick_group(mean);
}

static const char* const RESIDENT_STALL_TEXT =
    "resident PCG: a wait between the CTAs of a cluster ran out";

// One plane model on the chip-resident cluster kernel (svx_resident.cu).
static PcgResult pcg_resident(svx_ctx* ctx, svx_op* op, const ResidentShape& shape, double tol,
                              long long max_iter, double* u_dev, int fault = -1,
                              long long wait_ns = 0) {
    struct Slot {
        int64_t off[2], max_iter, it;
        double tol, res;
        int32_t status, pad;
    };
    static_assert(sizeof(Slot) <= 256, "the context's pinned scalar slot holds 256 bytes");
    cudaStream_t st = ctx->stream;
    DBuf<Slot> d;
    d.alloc(ctx->pool, 1);
    Slot* h = static_cast<Slot*>(ctx->h_scalars);
    *h = Slot{{0, op->n_nodes}, max_iter, 0, tol, 0.0, PCG_RUNNING, 0};
    SVX_CUDA(cudaMemcpyAsync(d.p, h, sizeof(Slot), cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaEventRecord(ctx->ev[0], st));
    resident_pcg(ctx, op, shape, true, st, 1, nullptr, d.p->off, &d.p->tol, &d.p->max_iter, &d.p->it,
                 &d.p->res, &d.p->status, u_dev, fault, wait_ns);
    SVX_CUDA(cudaEventRecord(ctx->ev[1], st));
    SVX_CUDA(cudaMemcpyAsync(h, d.p, sizeof(Slot), cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaStreamSynchronize(st));
    float ms = 0.f;
    SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
    if (h->status == RESIDENT_STALLED) throw ModelFail{SVX_CUDA_ERROR, 0, -1, RESIDENT_STALL_TEXT};
    return PcgResult{h->status, h->it, h->res, ms};
}

// The cluster shape of a plane operator's FP64 solve; false: another form.
static bool resident_single_shape(svx_ctx* ctx, svx_op* op, ResidentShape* shape) {
    if (op->slot_span < 0) {
        std::vector<int64_t> span{0};
        resident_order(ctx, op, true, {0, op->n_nodes}, span);
        op->slot_span = span[0];
    }
    return resident_shape(ctx, op->n_nodes, op->slot_span, true, shape);
}

void resident_stall_diag(svx_ctx* ctx, svx_op* op, int fault, long long wait_ns) {
    ResidentShape shape;
    if (op->ndof != 2 || op->n_nodes >= RESIDENT_MAX_NODES || op->pat.max_deg > RESIDENT_MAX_DEG ||
        !resident_single_shape(ctx, op, &shape) || shape.ctas < 2)
        throw ModelFail{SVX_BAD_ARGUMENT, 0, -1, "not an operator that a cluster solves"};
    DBuf<double> u;
    u.alloc(ctx->pool, op->n);
    pcg_resident(ctx, op, shape, 1e-10, 1000, u.p, fault, wait_ns);
}

// Gives an FP64 run of a C3D8 model its element-by-element form, where it
// has one: bricks while a model's bricks fit the chip, the graph form above.
static void wire_hex_form(svx_ctx* ctx, svx_op* op, PcgRun<double, double, double>& run,
                          HexWork& hex, BrickWork& brick) {
    if (!hex_applies(ctx, op)) return;
    if (!(ctx->graph_min_nnz >= 0 && use_graph_form(ctx, op)) && op->brick.state == 0) {
        int coop = 0;
        SVX_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
        const int64_t per = std::max<int64_t>(ctx->brick_elems,
                                              (op->n_elem + ctx->sm_count - 1) / ctx->sm_count);
        std::vector<int> nbricks{coop && per <= ctx->brick_max_elems
                                     ? int((op->n_elem + per - 1) / per) : 0};
        if (nbricks[0] > 0) brick_build(ctx, op, true, {0, op->n_nodes}, {0, op->n_elem}, nbricks);
        if (nbricks[0] == 0) op->brick = BrickOperator{};  // what was built goes back
        op->brick.state = nbricks[0] > 0 ? 1 : -1;
    }
    if (op->brick.state > 0) {
        if (op->brick.stale) brick_constants(ctx, op);
        brick.alloc(ctx, op, true);
        run.brick = &brick;
        return;
    }
    // a model that the shared-memory kernel holds and that has no bricks keeps
    // its assembled K: a 35^3 cube runs 19.7 us an iteration on it and 22.4 in
    // the graph form's three launches; at 180 x 16 x 16 it is 24.0 and 22.2
    if (!use_graph_form(ctx, op) && op->n_elem < 45000 && ctx->brick_max_elems > 1) return;
    hex_prepare(ctx, op);
    hex.alloc(ctx, op);
    run.hex = &hex;
}

// A device too full for the form's own arrays (about a sixth of the assembled
// K) solves on K, as it could before.
static void wire_hex(svx_ctx* ctx, svx_op* op, PcgRun<double, double, double>& run, HexWork& hex,
                     BrickWork& brick) {
    try {
        wire_hex_form(ctx, op, run, hex, brick);
    } catch (const ModelFail& f) {
        if (f.code != SVX_OOM) throw;
        SVX_CUDA(cudaStreamSynchronize(ctx->stream));
        run.hex = nullptr;
        run.brick = nullptr;
        hex = HexWork{};
        brick = BrickWork{};
        op->hex = HexOperator{};
        op->brick = BrickOperator{};
    }
}

PcgResult pcg_fp64(svx_ctx* ctx, svx_op* op, double tol, long long max_iter, int check_every,
                   double* u_dev) {
    const int64_t n = op->n;
    cudaStream_t st = ctx->stream;
    PcgResult out{PCG_CONVERGED, 0, 0.0, 0.0};
    // plane models that fit on the chip; a budget so large that one launch
    // could run for many seconds keeps the chunked launches below
    if (op->ndof == 2 && op->n_nodes < RESIDENT_MAX_NODES && ctx->resident && ctx->pcg_smem &&
        op->pat.max_deg <= RESIDENT_MAX_DEG && max_iter <= RESIDENT_MAX_ITER &&
        !use_graph_form(ctx, op)) {
        ResidentShape shape;
        if (resident_single_shape(ctx, op, &shape))
            return pcg_resident(ctx, op, shape, tol, max_iter, u_dev);
    }
    if (check_every <= 0) check_every = auto_check_every(n, op->pat.nnz);
    DBuf<double> r, p, p2, q, partials;
    DBuf<PcgScalars> s;
    r.alloc(ctx->pool, n + 1);
    p.alloc(ctx->pool, n + 1);
    q.alloc(ctx->pool, n + 1);
    const bool graph = use_graph_form(ctx, op);
    if (!graph) {
        p2.alloc(ctx->pool, n + 1);
        SVX_CUDA(cudaMemsetAsync(p2.p, 0, (n + 1) * sizeof(double), st));
    }
    const int G = pick_node_group(op->pat.max_deg, op->ndof);
    PcgRun<double, double, double> run;
    run.ctx = ctx;
    run.op = op;
    run.n = n;
    run.G = G;
    run.grid_r = grid_nodes(ctx, op->n_nodes, G);
    run.grid_v = grid_vec(ctx, n);
    partials.alloc(ctx->pool, 2 * size_t(std::max(run.grid_r, run.grid_v)) + 2);
    s.alloc(ctx->pool, 1);
    PinnedScalars hs(ctx);
    PcgScalars init{};
    init.tol = tol;
    init.max_iter = max_iter;
    init.rr_stop = -1.0;
    init.status = PCG_RUNNING;
    SVX_CUDA(cudaMemcpyAsync(s.p, &init, sizeof(init), cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaEventRecord(ctx->ev[0], st));
    init_kernel<double, double><<<run.grid_v, BLOCK, 0, st>>>(n, op->f.p, 1.0, u_dev, r.p, p.p,
                                                             op->inv_diag.p, partials.p, s.p);
    SVX_LAUNCH_CHECK();
    run.vals = op->vals.p;
    run.inv_diag = op->inv_diag.p;
    run.u = u_dev;
    run.r = r.p;
    run.p = p.p;
    run.q = q.p;
    run.p2 = p2.p;
    run.partials = partials.p;
    run.s = s.p;
    run.h_s = hs.h;
    HexWork hex;
    BrickWork brick;
    wire_hex(ctx, op, run, hex, brick);
    SVX_CUDA(cudaMemcpyAsync(hs.h, s.p, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaStreamSynchronize(st));
    int status = hs.h->status;
    if (status == PCG_RUNNING && run.brick) {
        status = run.iterate_brick(persistent_chunk(op->pat.nnz));
    } else if (status == PCG_RUNNING && run.hex) {
        status = run.iterate(check_every);
    } else if (status == PCG_RUNNING) {
        // the graph form starts from the init kernel's p = z0 too: a
        // persistent launch that cannot start leaves p untouched
        status = -1;
        if (!graph && ctx->pcg_smem) status = run.iterate_scalar(persistent_chunk(op->pat.nnz));
        if (!graph && status < 0 && ctx->pcg_smem)
            status = run.iterate_smem(persistent_chunk(op->pat.nnz), transposed_values(ctx, op));
        if (!graph && status < 0) status = run.iterate_persistent(persistent_chunk(op->pat.nnz));
        if (status < 0) status = run.iterate(check_every);
    }
    SVX_CUDA(cudaEventRecord(ctx->ev[1], st));
    SVX_CUDA(cudaEventSynchronize(ctx->ev[1]));
    float ms = 0.f;
    SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
    out.status = status;
    out.iterations = hs.h->it;
    out.residual = hs.h->res;
    out.ms = ms;
    return out;
}

// r = V(r64); partials of r.z; the last block forms beta = r.z / rz_old for
// the reliable update (the search direction p is kept).
template <class V>
__global__ void __launch_bounds__(BLOCK)
reliable_resume_kernel(int64_t n, const double* __restrict__ r64, V* __restrict__ r,
                       const V* __restrict__ inv_diag, double* __restrict__ partials,
                       PcgScalars* __restrict__ s) {
    __shared__ double sh[32];
    double rz = 0.0;
    for (int64_t i = int64_t(blockIdx.x) * BLOCK + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * BLOCK) {
        const V ri = V(r64[i]);
        r[i] = ri;
        rz += double(ri) * double(ri * inv_diag[i]);
    }
    const double b = block_sum(rz, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = b;
    if (last_block(&s->count_c)) {
        const double t = sum_partials(partials, gridDim.x, sh);
        if (threadIdx.x == 0) {
            s->count_c = 0;
            s->beta = t / s->rz;
            s->rz = t;
        }
    }
}

// Mixed precision: FP32-stored K inside one FP64 Jacobi-PCG whose operator
// precision is relaxed as it converges.  The theory of inexact Krylov
// methods (Simoncini and Szyld 2003; van den Eshof and Sleijpen 2004) allows
// the error of iteration k's product K p to grow like tol / ||r_k||: early
// iterations need the exact operator, late ones tolerate FP32 storage.  So
// the solve runs the FP64 operator until ||r|| / ||f|| <= tau
// (mixed_switch_residual: tol / 1e-7, i.e. 1e-3 at tol = 1e-10, the FP32
// operator's relative error being ~1e-7), keeps that iterate, and runs the
// difference-form FP32 operator (compensated_fp32_kernel) on the same
// search directions until the recursive residual meets tol, for at most as
// many iterations as the FP64 phase took.  The true residual f - K64 u
// then decides.  The theory bounds the residual, not the error: on a badly
// conditioned model (condition 1e7-1e10, slender CPS3 strips of the plate
// mix) the FP32 operator leaves errors in the stiffness's soft modes whose
// residual lies below tol, up to 3e-8 against the FP64 solution where the
// FP64 solve is within 5e-11 of the exact one.  Those solves are the ones
// whose FP32 phase misses tol within its budget or fails the true-residual
// test, so in either case the solve rolls back to the kept iterate and
// finishes on the FP64 operator: the FP32 phase's updates are discarded and
// the result is the FP64 solve's.  u, r, p and every dot stay FP64; the
// FP32 iterations stream 4 B instead of 8 B per stored value.
PcgResult pcg_mixed(svx_ctx* ctx, svx_op* op, double tol, long long max_iter, double inner_tol,
                    int check_every, double* u_dev, long long* outer_steps) {
    if (check_every <= 0) check_every = auto_check_every(op->n, op->pat.nnz);
    const bool graph = use_graph_form(ctx, op);
    (void)inner_tol;
    const int64_t n = op->n;
    cudaStream_t st = ctx->stream;
    build_fp32_operator(ctx, op);
    const int G = pick_node_group(op->pat.max_deg, op->ndof);
    DBuf<double> r, p, p2, q, r64, partials, rr_dev;
    DBuf<PcgScalars> s;
    DBuf<unsigned int> counter;
    r.alloc(ctx->pool, n + 1);
    p.alloc(ctx->pool, n + 1);
    q.alloc(ctx->pool, n + 1);
    if (!graph) {
        p2.alloc(ctx->pool, n + 1);
        SVX_CUDA(cudaMemsetAsync(p2.p, 0, (n + 1) * sizeof(double), st));
    }
    r64.alloc(ctx->pool, n + 1);
    rr_dev.alloc(ctx->pool, 1);
    counter.alloc(ctx->pool, 1);
    SVX_CUDA(cudaMemsetAsync(counter.p, 0, sizeof(unsigned int), st));
    const unsigned grid_r = grid_nodes(ctx, op->n_nodes, G), grid_v = grid_vec(ctx, n);
    partials.alloc(ctx->pool, 2 * size_t(std::max(grid_r, grid_v)) + 2);
    s.alloc(ctx->pool, 1);
    PinnedScalars hs(ctx);
    PcgRun<float, double, double> sloppy;
    PcgRun<double, double, double> exact;
    auto wire = [&](auto& run) {
        run.ctx = ctx;
        run.op = op;
        run.n = n;
        run.G = G;
        run.grid_r = grid_r;
        run.grid_v = grid_v;
        run.inv_diag = op->inv_diag.p;
        run.u = u_dev;
        run.r = r.p;
        run.p = p.p;
        run.q = q.p;
        run.p2 = p2.p;
        run.partials = partials.p;
        run.s = s.p;
        run.h_s = hs.h;
    };
    wire(sloppy);
    wire(exact);
    sloppy.vals = op->vals32.p;
    exact.vals = op->vals.p;
    HexWork hex;
    BrickWork brick;
    wire_hex(ctx, op, exact, hex, brick);

    auto true_residual = [&]() -> double {
        const Pattern& P = op->pat;
        SVX_NODE_DISPATCH(op->ndof, G,
                          (residual_node_kernel<ND, GG><<<grid_r, BLOCK, 0, st>>>(
                              op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, op->vals.p, u_dev,
                              op->f.p, r64.p, partials.p, counter.p, rr_dev.p)));
        SVX_LAUNCH_CHECK();
        double h = 0.0;
        SVX_CUDA(cudaMemcpyAsync(&h, rr_dev.p, sizeof(double), cudaMemcpyDeviceToHost, st));
        SVX_CUDA(cudaStreamSynchronize(st));
        return h;
    };
    auto set_field = [&](auto PcgScalars::*field, auto value) {
        SVX_CUDA(cudaMemcpyAsync(&(s.p->*field), &value, sizeof(value), cudaMemcpyHostToDevice,
                                 st));
        SVX_CUDA(cudaStreamSynchronize(st));
    };

    SVX_CUDA(cudaEventRecord(ctx->ev[0], st));
    const double tau = mixed_switch_residual(tol);
    PcgScalars init{};
    init.tol = tol;
    init.max_iter = max_iter;
    init.status = PCG_RUNNING;
    init.rr_stop = -1.0;
    SVX_CUDA(cudaMemcpyAsync(s.p, &init, sizeof(init), cudaMemcpyHostToDevice, st));
    init_kernel<double, double, double><<<grid_v, BLOCK, 0, st>>>(
        n, op->f.p, 1.0, u_dev, r.p, p.p, op->inv_diag.p, partials.p, s.p);
    SVX_LAUNCH_CHECK();
    SVX_CUDA(cudaMemcpyAsync(hs.h, s.p, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaStreamSynchronize(st));
    const double bnorm = hs.h->bnorm;
    int status = hs.h->status;
    long long outer = 0, sloppy_iters = 0;
    double res = hs.h->res;
    const int chunk = persistent_chunk(op->pat.nnz);
    auto valsT_of = [&](auto& pcg) {
        if constexpr (std::is_same<std::decay_t<decltype(*pcg.vals)>, float>::value)
            return transposed(ctx, op, op->vals32, op->vals32T);
        else
            return transposed_values(ctx, op);
    };
    auto run = [&](auto& pcg) -> int {
        if (pcg.brick) return pcg.iterate_brick(chunk);
        if (graph || pcg.hex) return pcg.iterate(check_every);
        // solids: the shared-memory kernel's three-barrier form, which takes
        // and leaves p as the kernel below does (an FP64 iteration of the mixed
        // form at 80 x 16 x 16 19.7 -> 12.4 us; 160 x 16 x 16 has bricks)
        int stt = -1;
        if (op->ndof == 3 && ctx->pcg_smem)
            stt = pcg.iterate_smem(chunk, valsT_of(pcg), 0);
        if (stt < 0) stt = pcg.iterate_persistent(chunk);
        if (stt < 0)
            throw ModelFail{SVX_CUDA_ERROR, 0, -1,
                            "mixed precision below 50M nonzeros needs a cooperative launch"};
        return stt;
    };
    // continue CG from r (replaced from r64) with beta = r.z / rz_prev, or
    // restart it (beta = 0, p = z); the graph form and the three-barrier
    // (3D) persistent kernel update p here, the two-barrier (2D) one forms
    // the next p itself from r, the previous p and beta
    // (p_update_kernel works only while the status is RUNNING)
    auto resume = [&](bool restart) {
        reliable_resume_kernel<double><<<grid_v, BLOCK, 0, st>>>(n, r64.p, r.p, op->inv_diag.p,
                                                                partials.p, s.p);
        SVX_LAUNCH_CHECK();
        if (restart) set_field(&PcgScalars::beta, 0.0);
        set_field(&PcgScalars::status, int(PCG_RUNNING));
        if (graph || op->ndof == 3) {
            p_update_kernel<double><<<grid_v, BLOCK, 0, st>>>(n, p.p, r.p, op->inv_diag.p, s.p);
            SVX_LAUNCH_CHECK();
        }
    };
    // 1. FP64 operator until ||r|| / ||f|| <= tau (status PCG_RELIABLE)
    if (status == PCG_RUNNING) {
        set_field(&PcgScalars::rr_stop, tau * tau * hs.h->rr);
        status = run(exact);
        res = hs.h->res;
    }
    // 2. FP32 operator on the same Krylov space to the tolerance, for at
    // most as many iterations as the FP64 phase took
    if (status == PCG_RELIABLE) {
        SVX_CUDA(cudaMemcpyAsync(r64.p, r.p, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
        set_field(&PcgScalars::rr_stop, -1.0);
        const long long it0 = hs.h->it;
        const long long cap = std::min<long long>(max_iter, 2 * it0);
        // the switch iterate, kept for a rollback: u, r, p (and the 2D
        // kernel's second direction buffer) and the scalars
        DBuf<double> sv;
        DBuf<PcgScalars> s_sv;
        sv.alloc(ctx->pool, 4 * size_t(n) + 1);
        s_sv.alloc(ctx->pool, 1);
        auto copy = [&](double* to, const double* from) {
            SVX_CUDA(cudaMemcpyAsync(to, from, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
        };
        copy(sv.p, u_dev);
        copy(sv.p + n, r64.p);
        copy(sv.p + 2 * n, p.p);
        if (p2.p) copy(sv.p + 3 * n, p2.p);
        SVX_CUDA(cudaMemcpyAsync(s_sv.p, s.p, sizeof(PcgScalars), cudaMemcpyDeviceToDevice, st));
        set_field(&PcgScalars::max_iter, cap);
        resume(false);
        status = run(sloppy);
        sloppy_iters = hs.h->it - it0;
        res = hs.h->res;
        set_field(&PcgScalars::max_iter, max_iter);
        // 3. the true FP64 residual decides
        bool undo = hs.h->it < max_iter && status != PCG_CONVERGED;  // budget or breakdown
        if (status == PCG_CONVERGED) {
            ++outer;
            const double rr_true = true_residual();
            res = std::sqrt(rr_true) / bnorm;
            undo = res > tol;
        }
        if (undo) {
            // back to the switch iterate, on the FP64 operator from there:
            // the FP32 phase's updates are discarded, its iterations counted
            const long long it_now = hs.h->it;
            // the 2D persistent kernel keeps p_k in buffer k & 1: with the
            // count kept, an odd number of discarded iterations swaps them
            const bool flip = !graph && op->ndof != 3 && ((it_now - it0) & 1);
            copy(u_dev, sv.p);
            copy(r64.p, sv.p + n);
            copy(flip ? p2.p : p.p, sv.p + 2 * n);
            if (p2.p) copy(flip ? p.p : p2.p, sv.p + 3 * n);
            SVX_CUDA(cudaMemcpyAsync(s.p, s_sv.p, sizeof(PcgScalars), cudaMemcpyDeviceToDevice,
                                     st));
            set_field(&PcgScalars::it, it_now);
            set_field(&PcgScalars::max_iter, max_iter);
            resume(false);
            status = run(exact);
            res = hs.h->res;
        }
    }
    SVX_CUDA(cudaEventRecord(ctx->ev[1], st));
    SVX_CUDA(cudaEventSynchronize(ctx->ev[1]));
    float ms = 0.f;
    SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
    SVX_CUDA(cudaMemcpyAsync(hs.h, s.p, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaStreamSynchronize(st));
    PcgResult out{status, hs.h->it, res, ms};
    op->mixed_sloppy_iters = sloppy_iters;
    if (outer_steps) *outer_steps = outer;
    return out;
}

// Defect correction with an FP32 inner PCG (SVX_MIXED_DEFECT): the outer
// loop keeps u, the residual r = f - K64 u and its norm in FP64; each
// correction solves K32 e = r / ||r|| with a Jacobi-PCG whose operator
// (the difference-form FP32 K), vectors and inverse diagonal are FP32 and
// whose dots accumulate in FP64, to a relative residual of inner_tol, then
// u += ||r|| e in FP64.  When a correction cuts ||r|| by less than 2x
// twice, the inner solver becomes the FP64 PCG on the same residual
// equation (inner tolerance tol ||f|| / ||r||), so the form converges where
// the FP32 operator's accuracy runs out.  The inner solves run in the CUDA
// graph form.  Iterations count every inner iteration; the FP32 ones are
// reported apart.
__global__ void __launch_bounds__(BLOCK)
to_float_kernel(int64_t n, const double* __restrict__ x, float* __restrict__ y) {
    for (int64_t i = int64_t(blockIdx.x) * BLOCK + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * BLOCK)
        y[i] = float(x[i]);
}

template <class E>
__global__ void __launch_bounds__(BLOCK)
correct_kernel(int64_t n, double a, const E* __restrict__ e, double* __restrict__ u) {
    for (int64_t i = int64_t(blockIdx.x) * BLOCK + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * BLOCK)
        u[i] += a * double(e[i]);
}

PcgResult pcg_defect_correction(svx_ctx* ctx, svx_op* op, double tol, long long max_iter,
                                double inner_tol, int check_every, double* u_dev,
                                long long* outer_steps) {
    if (check_every <= 0) check_every = auto_check_every(op->n, op->pat.nnz);
    if (!(inner_tol > 0.0) || !(inner_tol < 1.0)) inner_tol = 1e-5;
    const int64_t n = op->n;
    cudaStream_t st = ctx->stream;
    build_fp32_operator(ctx, op);
    const int G = pick_node_group(op->pat.max_deg, op->ndof);
    const unsigned grid_r = grid_nodes(ctx, op->n_nodes, G), grid_v = grid_vec(ctx, n);
    DBuf<float> r32, p32, q32, e32, d32, p2;
    DBuf<double> r64, e64, r, p, q, partials, rr_dev;
    DBuf<PcgScalars> s;
    DBuf<unsigned int> counter;
    for (auto* b : {&r32, &p32, &q32, &e32, &d32}) b->alloc(ctx->pool, n + 1);
    r64.alloc(ctx->pool, n + 1);
    rr_dev.alloc(ctx->pool, 1);
    counter.alloc(ctx->pool, 1);
    SVX_CUDA(cudaMemsetAsync(counter.p, 0, sizeof(unsigned int), st));
    partials.alloc(ctx->pool, 2 * size_t(std::max(grid_r, grid_v)) + 2);
    s.alloc(ctx->pool, 1);
    PinnedScalars hs(ctx);
    to_float_kernel<<<grid_v, BLOCK, 0, st>>>(n, op->inv_diag.p, d32.p);
    SVX_LAUNCH_CHECK();

    auto true_residual = [&]() -> double {
        const Pattern& P = op->pat;
        SVX_NODE_DISPATCH(op->ndof, G,
                          (residual_node_kernel<ND, GG><<<grid_r, BLOCK, 0, st>>>(
                              op->n_nodes, P.adj_ptr.p, P.adj.p, P.node_base.p, op->vals.p, u_dev,
                              op->f.p, r64.p, partials.p, counter.p, rr_dev.p)));
        SVX_LAUNCH_CHECK();
        double h = 0.0;
        SVX_CUDA(cudaMemcpyAsync(&h, rr_dev.p, sizeof(double), cudaMemcpyDeviceToHost, st));
        SVX_CUDA(cudaStreamSynchronize(st));
        return h;
    };
    // one inner solve of K e = r64 / ||r64|| to inner relative tolerance
    // `itol` within `budget` iterations; returns its status and iterations
    auto inner = [&](auto& run, auto* e, auto* rr_, auto* pp, auto* qq, const auto* dinv,
                     double scale, double itol, long long budget) {
        using V = std::remove_pointer_t<decltype(pp)>;
        PcgScalars init{};
        init.tol = itol;
        init.max_iter = budget;
        init.status = PCG_RUNNING;
        init.rr_stop = -1.0;
        SVX_CUDA(cudaMemcpyAsync(s.p, &init, sizeof(init), cudaMemcpyHostToDevice, st));
        init_kernel<V, double, V><<<grid_v, BLOCK, 0, st>>>(n, r64.p, scale, e, rr_, pp, dinv,
                                                            partials.p, s.p);
        SVX_LAUNCH_CHECK();
        run.ctx = ctx;
        run.op = op;
        run.n = n;
        run.G = G;
        run.grid_r = grid_r;
        run.grid_v = grid_v;
        run.inv_diag = dinv;
        run.u = e;
        run.r = rr_;
        run.p = pp;
        run.q = qq;
        run.partials = partials.p;
        run.s = s.p;
        run.h_s = hs.h;
        SVX_CUDA(cudaMemcpyAsync(hs.h, s.p, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
        SVX_CUDA(cudaStreamSynchronize(st));
        int status = hs.h->status;
        // below the graph threshold the shared-memory kernel runs the FP32
        // inner solve too: in the graph its three launches' gaps cost more than
        // the arithmetic (80 x 8 x 8: 14.8 us an iteration in the graph, 7.9
        // here; 160 x 16 x 16: 23.3 and 17.4)
        if constexpr (std::is_same<V, float>::value) {
            if (status == PCG_RUNNING && !use_graph_form(ctx, op) && ctx->pcg_smem) {
                if (!p2.p) p2.alloc(ctx->pool, n + 1);
                SVX_CUDA(cudaMemsetAsync(p2.p, 0, (n + 1) * sizeof(float), st));
                run.p2 = p2.p;
                const int got = run.iterate_smem(persistent_chunk(op->pat.nnz),
                                                 transposed(ctx, op, op->vals32, op->vals32T));
                if (got >= 0) status = got;
            }
        }
        if (status == PCG_RUNNING) status = run.iterate(check_every);
        SVX_CUDA(cudaMemcpyAsync(hs.h, s.p, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
        SVX_CUDA(cudaStreamSynchronize(st));
        return std::make_pair(status, (long long)hs.h->it);
    };

    SVX_CUDA(cudaEventRecord(ctx->ev[0], st));
    SVX_CUDA(cudaMemsetAsync(u_dev, 0, n * sizeof(double), st));
    double rr = true_residual();
    const double bnorm = std::sqrt(rr);
    int status = PCG_CONVERGED;
    long long total = 0, fp32_total = 0, outer = 0;
    int stagnant = 0;
    bool fp64 = false;
    double res = bnorm > 0.0 ? 1.0 : 0.0;
    while (bnorm > 0.0) {
        res = std::sqrt(rr) / bnorm;
        if (res <= tol) {
            status = PCG_CONVERGED;
            break;
        }
        if (total >= max_iter) {
            status = PCG_MAXITER;
            break;
        }
        ++outer;
        const double rn = std::sqrt(rr);
        std::pair<int, long long> in;
        if (!fp64) {
            PcgRun<float, float, float> run32;
            run32.vals = op->vals32.p;
            in = inner(run32, e32.p, r32.p, p32.p, q32.p, (const float*)d32.p, 1.0 / rn,
                       inner_tol, max_iter - total);
            fp32_total += in.second;
            correct_kernel<float><<<grid_v, BLOCK, 0, st>>>(n, rn, e32.p, u_dev);
        } else {
            if (!e64.p) {
                for (auto* b : {&e64, &r, &p, &q}) b->alloc(ctx->pool, n + 1);
            }
            PcgRun<double, double, double> run64;
            run64.vals = op->vals.p;
            in = inner(run64, e64.p, r.p, p.p, q.p, (const double*)op->inv_diag.p, 1.0 / rn,
                       std::min(0.5, tol * bnorm / rn), max_iter - total);
            correct_kernel<double><<<grid_v, BLOCK, 0, st>>>(n, rn, e64.p, u_dev);
        }
        SVX_LAUNCH_CHECK();
        total += in.second;
        const double rr_new = true_residual();
        if (in.first == PCG_BREAKDOWN || !(rr_new < 0.25 * rr)) ++stagnant;
        if (!fp64 && stagnant >= 2) fp64 = true;
        else if (fp64 && !(rr_new < rr)) {  // the FP64 solver made no progress either
            rr = rr_new;
            res = std::sqrt(rr) / bnorm;
            status = res <= tol ? PCG_CONVERGED : PCG_BREAKDOWN;
            break;
        }
        rr = rr_new;
    }
    SVX_CUDA(cudaEventRecord(ctx->ev[1], st));
    SVX_CUDA(cudaEventSynchronize(ctx->ev[1]));
    float ms = 0.f;
    SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
    op->mixed_sloppy_iters = fp32_total;
    if (outer_steps) *outer_steps = outer;
    return PcgResult{status, total, res, ms};
}

}  // namespace svx

// ---------------------------------------------------------------------------
// Jacobi-PCG on a caller-owned device CSR that allocates no memory.
//
// Some callers cannot let a library allocate device memory: a host
// application that owns the whole device-memory budget through its own
// arena (a cudaMalloc behind its back fragments that arena and synchronises
// the device), or a caller running a latency-bounded loop in which the
// implicit synchronisation and unpredictable latency of cudaMalloc /
// cudaFree are not acceptable.  For them svx_pcg_solve_noalloc takes every
// input and output as a device pointer and keeps all of its work vectors in
// the file-scope array below, which every GPU that loads the library holds
// until the process exits.
// ---------------------------------------------------------------------------
namespace svx {
namespace {

constexpr int64_t NOALLOC_MAX_N = SVX_NOALLOC_MAX_DOF;
constexpr int64_t NOALLOC_PARTIALS = 4096;  // >= 2 * the largest grid used
constexpr int64_t NOALLOC_SCALARS = 16;     // doubles holding a PcgScalars
constexpr int64_t NOALLOC_DOUBLES = 4 * NOALLOC_MAX_N + NOALLOC_PARTIALS + NOALLOC_SCALARS;
static_assert(sizeof(PcgScalars) <= NOALLOC_SCALARS * sizeof(double), "scalar slot too small");

// r | p | q | inv_diag | block partials | PcgScalars.  Shared by every call
// on a device; its contents are whatever the previous call left.
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_DOUBLES];

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};
int g_noalloc_sms[NOALLOC_MAX_DEVICES] = {};

// 1 / K_ii (0 for a zero or missing diagonal), as the PCG's Jacobi step.
__global__ void noalloc_inv_diag_kernel(int64_t n, const int32_t* __restrict__ row_ptr,
                                        const int32_t* __restrict__ col_idx,
                                        const double* __restrict__ vals,
                                        double* __restrict__ inv_diag) {
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d = 0.0;
    for (int32_t j = row_ptr[i]; j < row_ptr[i + 1]; ++j)
        if (col_idx[j] == i) {
            d = vals[j];
            break;
        }
    inv_diag[i] = (d == 0.0) ? 0.0 : 1.0 / d;
}

void launch_spmv_dot_raw(int G, unsigned grid, cudaStream_t st, int64_t n, const int32_t* rp,
                         const int32_t* ci, const double* vals, const double* p, double* q,
                         double* partials, PcgScalars* s) {
    switch (G) {
        case 2: spmv_dot_kernel<2, double><<<grid, BLOCK, 0, st>>>(n, rp, ci, vals, p, q, partials, s); break;
        case 4: spmv_dot_kernel<4, double><<<grid, BLOCK, 0, st>>>(n, rp, ci, vals, p, q, partials, s); break;
        case 8: spmv_dot_kernel<8, double><<<grid, BLOCK, 0, st>>>(n, rp, ci, vals, p, q, partials, s); break;
        case 16: spmv_dot_kernel<16, double><<<grid, BLOCK, 0, st>>>(n, rp, ci, vals, p, q, partials, s); break;
        default: spmv_dot_kernel<32, double><<<grid, BLOCK, 0, st>>>(n, rp, ci, vals, p, q, partials, s); break;
    }
}

// Device address of the scratch array and the SM count of the current
// device, looked up once per device (the array's name is only a host-side
// stand-in; the kernels need the address cudaGetSymbolAddress returns).
cudaError_t noalloc_setup(int* device, double** scratch, int* sms) {
    cudaError_t e = cudaGetDevice(device);
    if (e != cudaSuccess) return e;
    if (*device < 0 || *device >= NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[*device]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        int count = 0;
        e = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, *device);
        if (e != cudaSuccess) return e;
        g_noalloc_sms[*device] = count;
        g_noalloc_ptr[*device] = static_cast<double*>(p);
    }
    *scratch = g_noalloc_ptr[*device];
    *sms = g_noalloc_sms[*device];
    return cudaSuccess;
}

}  // namespace

}  // namespace svx

extern "C" int svx_pcg_solve_noalloc(int64_t n, const int32_t* row_ptr, const int32_t* col_idx,
                                     const double* vals, const double* f, double tol,
                                     int64_t max_iter, double* u, int64_t* iterations,
                                     double* residual, void* stream) {
    using namespace svx;
    if (n <= 0 || !row_ptr || !col_idx || !vals || !f || !u) return SVX_BAD_ARGUMENT;
    if (n > NOALLOC_MAX_N) return SVX_BAD_ARGUMENT;  // beyond the static scratch
    if (!(tol >= 0.0)) return SVX_BAD_ARGUMENT;      // negative or NaN
    int device = 0, sms = 0;
    double* scratch = nullptr;
    if (noalloc_setup(&device, &scratch, &sms) != cudaSuccess) {
        cudaGetLastError();
        return SVX_CUDA_ERROR;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* r = scratch;
    double* p = r + NOALLOC_MAX_N;
    double* q = p + NOALLOC_MAX_N;
    double* inv_diag = q + NOALLOC_MAX_N;
    double* partials = inv_diag + NOALLOC_MAX_N;
    PcgScalars* s = reinterpret_cast<PcgScalars*>(partials + NOALLOC_PARTIALS);

    // nnz and the launch geometry of the allocating path
    int32_t nnz = 0;
    if (cudaMemcpyAsync(&nnz, row_ptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return SVX_CUDA_ERROR;
    }
    const int G = pick_group(double(nnz) / double(n));
    const int64_t per_block = BLOCK / G;
    // the block partials hold two values per block of the widest grid; the
    // grids stop at that (a device with more SMs only gets fewer blocks)
    const int64_t grid_cap =
        std::min<int64_t>(int64_t(sms) * 8, (NOALLOC_PARTIALS - 2) / 2);
    const unsigned grid_r = unsigned(std::max<int64_t>(
        1, std::min<int64_t>((n + per_block - 1) / per_block, grid_cap)));
    const unsigned grid_v =
        unsigned(std::max<int64_t>(1, std::min<int64_t>((n + BLOCK - 1) / BLOCK, grid_cap)));
    if (max_iter <= 0) max_iter = std::max<int64_t>(1000, 10 * n);
    const int check_every = auto_check_every(n, nnz);

    // the scalars must start from a clean state every call; rr_stop < 0
    // disables the reliable-update stop, as in the allocating FP64 solve
    PcgScalars init{};
    init.tol = tol;
    init.max_iter = max_iter;
    init.status = PCG_RUNNING;
    init.rr_stop = -1.0;
    PcgScalars h{};
    cudaError_t e = cudaMemcpyAsync(s, &init, sizeof(init), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        noalloc_inv_diag_kernel<<<unsigned((n + 255) / 256), 256, 0, st>>>(n, row_ptr, col_idx,
                                                                           vals, inv_diag);
        init_kernel<double, double><<<grid_v, BLOCK, 0, st>>>(n, f, 1.0, u, r, p, inv_diag,
                                                             partials, s);
        g_launches.fetch_add(2, std::memory_order_relaxed);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, s, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    // the device stops at max_iter; the launch bound only guards the host loop
    const long long launches_max = max_iter / check_every + 2;
    for (long long launch = 0; e == cudaSuccess && h.status == PCG_RUNNING; ++launch) {
        if (launch >= launches_max) {
            e = cudaErrorUnknown;
            break;
        }
        for (int k = 0; k < check_every; ++k) {
            launch_spmv_dot_raw(G, grid_r, st, n, row_ptr, col_idx, vals, p, q, partials, s);
            update_kernel<double, double><<<grid_v, BLOCK, 0, st>>>(n, u, r, p, q, inv_diag,
                                                                    partials, s);
            p_update_kernel<double><<<grid_v, BLOCK, 0, st>>>(n, p, r, inv_diag, s);
        }
        g_launches.fetch_add(3LL * check_every, std::memory_order_relaxed);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, s, sizeof(h), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return SVX_CUDA_ERROR;
    }
    if (iterations) *iterations = h.it;
    if (residual) *residual = h.res;
    return h.status == PCG_CONVERGED ? SVX_OK : SVX_NOT_CONVERGED;
}

namespace svx {

// ------------------------------------------------------------ batched host
namespace {

using BatchFn = void (*)(int, const int32_t*, const int64_t*, const int64_t*, const int32_t*,
                         const int64_t*, const double*, const double*, const double*, double*,
                         double*, double*, double*, const double*, const int64_t*, int64_t*,
                         double*, int32_t*);

struct BatchConfig {
    int nd, g, bs;
    BatchFn fn;
};

template <int ND, int G, int BS>
BatchConfig batch_config() {
    return BatchConfig{ND, G, BS, &batch_pcg_kernel<ND, G, BS, double>};
}

using BatchMixedFn = void (*)(int, const int32_t*, const int64_t*, const int64_t*,
                              const int32_t*, const int64_t*, const double*, const float*,
                              const double*, const double*, double*, double*, double*, double*,
                              const double*, const int64_t*, int64_t*, double*, int32_t*,
                              int64_t*, double*, double*, double*);

struct BatchMixedConfig {
    int nd, g, bs;
    BatchMixedFn fn;
};

template <int ND, int G, int BS>
BatchMixedConfig batch_mixed_config() {
    return BatchMixedConfig{ND, G, BS, &batch_pcg_mixed_kernel<ND, G, BS>};
}

// Candidate shapes of the batched kernels, in the same order for both forms;
// the default (used without autotuning) is index 2 for 2D and 1 for 3D.
std::vector<BatchMixedConfig> batch_mixed_candidates(int ndof) {
    if (ndof == 3)
        return {batch_mixed_config<3, 16, 128>(), batch_mixed_config<3, 16, 256>(),
                batch_mixed_config<3, 16, 512>(), batch_mixed_config<3, 32, 256>(),
                batch_mixed_config<3, 32, 512>(), batch_mixed_config<3, 8, 256>(),
                batch_mixed_config<3, 8, 512>()};
    return {batch_mixed_config<2, 8, 128>(), batch_mixed_config<2, 8, 256>(),
            batch_mixed_config<2, 8, 512>(), batch_mixed_config<2, 16, 256>(),
            batch_mixed_config<2, 16, 512>(), batch_mixed_config<2, 4, 256>(),
            batch_mixed_config<2, 4, 512>()};
}

int batch_default_choice(int ndof) { return ndof == 3 ? 1 : 2; }

// Members with at least this many rows run on a cluster of CLUSTER_CTAS CTAs
// (build constants).  Measured on the serving mix: 3D members gain from
// 4k rows up; 2D plates up to 13.5k rows run faster one CTA each (their
// 18 nonzeros a row leave the cluster barriers too little work to hide).
#ifndef SVX_CLUSTER_MIN_DOF_3D
#define SVX_CLUSTER_MIN_DOF_3D 4096
#endif
#ifndef SVX_CLUSTER_MIN_DOF_2D
#define SVX_CLUSTER_MIN_DOF_2D 16384
#endif
int64_t cluster_min_dof(int ndof) {
    return ndof == 3 ? int64_t(SVX_CLUSTER_MIN_DOF_3D) : int64_t(SVX_CLUSTER_MIN_DOF_2D);
}
// CTAs per member cluster, threads per CTA and lanes per 3D node (build
// constants); clusters above the portable 8 CTAs are allowed explicitly at
// launch.  Measured on the first 200 C3D8 cantilevers of the served request
// stream (5.48M DOF, 191 cluster members), device PCG time of one batched
// solve with 16 lanes per node: 8 x 256 626-631 ms, 8 x 512 437-441 ms,
// 8 x 768 499 ms, 8 x 1024 469 ms, 16 x 256 460 ms, 16 x 512 502 ms,
// 4 x 1024 476 ms (32 lanes at 8 x 512: 488 ms); with 8 lanes per node
// 8 x 512 394 ms (4.36 TB/s algorithmic), 8 x 256 534 ms, 8 x 1024 429 ms,
// 16 x 512 459 ms, and 4 lanes at 8 x 512 396 ms.
#ifndef SVX_CLUSTER_CTAS
#define SVX_CLUSTER_CTAS 8
#endif
#ifndef SVX_CLUSTER_BS
#define SVX_CLUSTER_BS 512
#endif
#ifndef SVX_CLUSTER_G3D
#define SVX_CLUSTER_G3D 8
#endif
constexpr int CLUSTER_CTAS = SVX_CLUSTER_CTAS;
constexpr int CLUSTER_G3D = SVX_CLUSTER_G3D;  // lanes per node of 3D members
constexpr int CLUSTER_BS = SVX_CLUSTER_BS;
// the mixed form's cluster kernel carries the reliable-update state in
// more registers; it keeps 256-thread CTAs
#ifndef SVX_CLUSTER_BS_MIXED
#define SVX_CLUSTER_BS_MIXED 256
#endif
constexpr int CLUSTER_BS_MIXED = SVX_CLUSTER_BS_MIXED;
static_assert(CLUSTER_CTAS >= 1 && CLUSTER_CTAS <= 16, "cluster size 1..16");

using ClusterFn = void (*)(int, const int32_t*, const int64_t*, const int64_t*, const int32_t*,
                           const int64_t*, const double*, const float*, const double*,
                           const double*, double*, double*, double*, double*, const double*,
                           const int64_t*, int64_t*, double*, int32_t*, int64_t*, double*,
                           double*, double*);

void launch_batch_cluster(int ndof, bool mixed, cudaStream_t st, int n_inst,
                          const int32_t* order, const int64_t* node_off, const int64_t* adj_ptr,
                          const int32_t* adj, const int64_t* node_base, const double* vals,
                          const float* vals32, const double* inv_diag, const double* f,
                          double* u, double* r, double* p, double* q, const double* tol,
                          const int64_t* max_iter, int64_t* out_it, double* out_res,
                          int32_t* out_status, int64_t* out_fp32, double* u_sv, double* r_sv,
                          double* p_sv) {
    ClusterFn fn;
    if (ndof == 3)
        fn = mixed
                 ? &batch_pcg_cluster_kernel<3, CLUSTER_G3D, CLUSTER_BS_MIXED, CLUSTER_CTAS, true>
                 : &batch_pcg_cluster_kernel<3, CLUSTER_G3D, CLUSTER_BS, CLUSTER_CTAS, false>;
    else
        fn = mixed ? &batch_pcg_cluster_kernel<2, 8, CLUSTER_BS_MIXED, CLUSTER_CTAS, true>
                   : &batch_pcg_cluster_kernel<2, 8, CLUSTER_BS, CLUSTER_CTAS, false>;
    if (CLUSTER_CTAS > 8)
        SVX_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(fn),
                                      cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(mixed ? CLUSTER_BS_MIXED : CLUSTER_BS);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(unsigned(n_inst * CLUSTER_CTAS));  // one cluster per member
    SVX_CUDA(cudaLaunchKernelEx(&cfg, fn, n_inst, order, node_off, adj_ptr, adj, node_base, vals,
                                vals32, inv_diag, f, u, r, p, q, tol, max_iter, out_it, out_res,
                                out_status, out_fp32, u_sv, r_sv, p_sv));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

std::vector<BatchConfig> batch_candidates(int ndof) {
    if (ndof == 3)
        return {batch_config<3, 16, 128>(), batch_config<3, 16, 256>(), batch_config<3, 16, 512>(),
                batch_config<3, 32, 256>(), batch_config<3, 32, 512>(), batch_config<3, 8, 256>(),
                batch_config<3, 8, 512>()};
    return {batch_config<2, 8, 128>(), batch_config<2, 8, 256>(), batch_config<2, 8, 512>(),
            batch_config<2, 16, 256>(), batch_config<2, 16, 512>(), batch_config<2, 4, 256>(),
            batch_config<2, 4, 512>()};
}

}  // namespace

// Largest node degree of each member, one CTA per member.
static __global__ void member_degree_kernel(const int64_t* __restrict__ node_off,
                                            const int64_t* __restrict__ adj_ptr,
                                            int64_t* __restrict__ out) {
    __shared__ int top;
    if (threadIdx.x == 0) top = 0;
    __syncthreads();
    int d = 0;
    for (int64_t i = node_off[blockIdx.x] + threadIdx.x; i < node_off[blockIdx.x + 1];
         i += blockDim.x)
        d = max(d, int(adj_ptr[i + 1] - adj_ptr[i]));
    atomicMax(&top, d);
    __syncthreads();
    if (threadIdx.x == 0) out[blockIdx.x] = top;
}

void batch_pcg(svx_ctx* ctx, svx_op* op, int count, const std::vector<int64_t>& node_off,
               const std::vector<int64_t>& elem_off, const std::vector<double>& tol, const std::vector<int64_t>& max_iter,
               std::vector<int64_t>& it, std::vector<double>& res, std::vector<int32_t>& status,
               std::vector<double>& cond, BatchStats* stats, bool mixed) {
    cudaStream_t st = ctx->stream;
    const int64_t n = op->n;
    const Pattern& P = op->pat;
    // Members of at least cluster_min_dof rows go to the cluster kernel (CS
    // CTAs per member), the rest to the CTA-per-member kernel; each class is
    // queued largest first (longest-processing-time order) and the two
    // kernels run concurrently on the context's two streams.
    std::vector<int32_t> order(count);
    for (int k = 0; k < count; ++k) order[k] = k;
    auto rows_of = [&](int k) { return (node_off[k + 1] - node_off[k]) * op->ndof; };
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return rows_of(a) > rows_of(b); });
    // FP64 plane members that fit on the chip run the resident cluster kernel,
    // one launch per cluster shape
    std::vector<ResidentShape> shapes(op->ndof == 2 && !mixed && ctx->resident ? count : 0);
    if (!shapes.empty()) {
        std::vector<int64_t> degree, span(count, 0);
        resident_order(ctx, op, false, node_off, span);
        if (P.max_deg > RESIDENT_MAX_DEG) {  // some member is out: find which
            DBuf<int64_t> off, top;
            off.alloc(ctx->pool, count + 1);
            top.alloc(ctx->pool, count + 1);
            degree.resize(count);
            SVX_CUDA(cudaMemcpyAsync(off.p, node_off.data(), (count + 1) * sizeof(int64_t),
                                     cudaMemcpyHostToDevice, st));
            member_degree_kernel<<<count, 256, 0, st>>>(off.p, P.adj_ptr.p, top.p);
            SVX_LAUNCH_CHECK();
            SVX_CUDA(cudaMemcpyAsync(degree.data(), top.p, count * sizeof(int64_t),
                                     cudaMemcpyDeviceToHost, st));
            SVX_CUDA(cudaStreamSynchronize(st));
        }
        for (int k = 0; k < count; ++k) {
            if (max_iter[k] > RESIDENT_MAX_ITER ||
                (!degree.empty() && degree[k] > RESIDENT_MAX_DEG) ||
                !resident_shape(ctx, node_off[k + 1] - node_off[k], span[k], false, &shapes[k]))
                shapes[k] = ResidentShape{};
        }
    }
    // FP64 C3D8 members on bricks, a cluster of 1, 2, 4, 8 or 16 CTAs each
    std::vector<int> nbricks;
    BrickWork brick;
    if (op->ndof == 3 && !mixed && ctx->hex && op->all_hex) {
        nbricks.assign(count, 0);
        bool any = false;
        for (int k = 0; k < count; ++k) {
            const int64_t ne = elem_off[k + 1] - elem_off[k];
            if (node_off[k + 1] - node_off[k] < ctx->hex_batch_min_nodes ||
                ne > 16 * int64_t(BRICK_MAX_ELEMS))
                continue;
            int c = 1;
            while (c < 16 && int64_t(c) * ctx->brick_batch_elems < ne) c *= 2;
            nbricks[k] = c;
            any = true;
        }
        if (any) {
            try {
                brick_build(ctx, op, false, node_off, elem_off, nbricks);
                brick.alloc(ctx, op, false);
            } catch (const ModelFail& f) {  // a full device: the members solve on K
                if (f.code != SVX_OOM) throw;
                SVX_CUDA(cudaStreamSynchronize(st));
                brick = BrickWork{};
                op->brick = BrickOperator{};
                std::fill(nbricks.begin(), nbricks.end(), 0);
            }
        }
        for (int k = 0; any && k < count; ++k)
            if (nbricks[k]) {
                shapes.resize(count);
                shapes[k].ctas = nbricks[k];
            }
    }
    auto resident = [&](int k) { return !shapes.empty() && shapes[k].ctas > 0; };
    const auto general_end = std::stable_partition(order.begin(), order.end(),
                                                   [&](int k) { return !resident(k); });
    const int n_general = int(general_end - order.begin());
    // resident members by shape, the largest shapes first, then by size
    std::stable_sort(general_end, order.end(), [&](int x, int y) {
        const ResidentShape &a = shapes[x], &b = shapes[y];
        if (op->ndof == 3) return a.ctas > b.ctas;
        return a.ctas * a.threads != b.ctas * b.threads ? a.ctas * a.threads > b.ctas * b.threads
                                                        : a.threads > b.threads;
    });
    int n_large = 0;
    while (n_large < n_general && rows_of(order[n_large]) >= cluster_min_dof(op->ndof)) ++n_large;
    const int n_small = n_general - n_large;
    // small class first in the order array, then the large class, then the
    // resident members
    std::vector<int32_t> ordered(order.begin() + n_large, order.begin() + n_general);
    ordered.insert(ordered.end(), order.begin(), order.begin() + n_large);
    ordered.insert(ordered.end(), order.begin() + n_general, order.end());
    DBuf<int32_t> d_order, d_status;
    DBuf<int64_t> d_off, d_maxit, d_it, d_cap;
    DBuf<double> d_tol, d_res, r, p, q, d_hi, d_lo;
    d_order.alloc(ctx->pool, count + 1);
    d_off.alloc(ctx->pool, count + 1);
    d_maxit.alloc(ctx->pool, count + 1);
    d_cap.alloc(ctx->pool, count + 1);
    d_it.alloc(ctx->pool, count + 1);
    d_tol.alloc(ctx->pool, count + 1);
    d_res.alloc(ctx->pool, count + 1);
    d_status.alloc(ctx->pool, count + 1);
    d_hi.alloc(ctx->pool, count + 1);
    d_lo.alloc(ctx->pool, count + 1);
    r.alloc(ctx->pool, n + 1);
    p.alloc(ctx->pool, n + 1);
    q.alloc(ctx->pool, n + 1);
    op->u.alloc(ctx->pool, n + 1);
    SVX_CUDA(cudaMemcpyAsync(d_order.p, ordered.data(), count * sizeof(int32_t),
                             cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaMemcpyAsync(d_off.p, node_off.data(), (count + 1) * sizeof(int64_t),
                             cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaMemcpyAsync(d_maxit.p, max_iter.data(), count * sizeof(int64_t),
                             cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaMemcpyAsync(d_tol.p, tol.data(), count * sizeof(double), cudaMemcpyHostToDevice,
                             st));
    DBuf<int64_t> d_fp32;
    DBuf<double> sv;  // the mixed form's iterate at its switch: u, r, p
    if (mixed) {
        build_fp32_operator(ctx, op);
        d_fp32.alloc(ctx->pool, count + 1);
        sv.alloc(ctx->pool, 3 * size_t(n) + 1);
    }
    double* const u_sv = mixed ? sv.p : nullptr;
    double* const r_sv = mixed ? sv.p + n : nullptr;
    double* const p_sv = mixed ? sv.p + 2 * n : nullptr;
    const std::vector<BatchConfig> cands = batch_candidates(op->ndof);
    const std::vector<BatchMixedConfig> mcands = batch_mixed_candidates(op->ndof);
    cudaStream_t pst = ctx->pcg_stream;
    auto launch = [&](int c, const int64_t* maxit, int n_inst) {
        const int bs = cands[c].bs;
        const int grid = std::max(1, n_inst);  // one CTA per member
        if (mixed)
            mcands[c].fn<<<grid, bs, 0, pst>>>(n_inst, d_order.p, d_off.p, P.adj_ptr.p, P.adj.p,
                                               P.node_base.p, op->vals.p, op->vals32.p,
                                               op->inv_diag.p, op->f.p, op->u.p, r.p, p.p, q.p,
                                               d_tol.p, maxit, d_it.p, d_res.p, d_status.p,
                                               d_fp32.p, u_sv, r_sv, p_sv);
        else
            cands[c].fn<<<grid, bs, 0, pst>>>(n_inst, d_order.p, d_off.p, P.adj_ptr.p, P.adj.p,
                                              P.node_base.p, op->vals.p, op->inv_diag.p,
                                              op->f.p, op->u.p, r.p, p.p, q.p, d_tol.p, maxit,
                                              d_it.p, d_res.p, d_status.p);
        SVX_LAUNCH_CHECK();
    };
    // the PCG kernels run on the context's low-priority streams, forked
    // from (and joined back into) its main stream
    SVX_CUDA(cudaEventRecord(ctx->fork_ev, st));
    SVX_CUDA(cudaStreamWaitEvent(pst, ctx->fork_ev, 0));
    // autotune of the CTA-per-member kernel (once per context, form and
    // ndof): threads per CTA and lanes per node, timed on the largest small
    // members with a short iteration budget.  A class smaller than the SM
    // count is too small to time and runs the default shape without fixing
    // the choice.
    int& tuned = ctx->batch_choice[(mixed ? 2 : 0) + (op->ndof == 3 ? 1 : 0)];
    int choice = tuned;
    if (choice < 0 && n_small < ctx->sm_count) choice = batch_default_choice(op->ndof);
    if (choice < 0) {
        const int sample = std::min(n_small, 2 * ctx->sm_count);
        std::vector<int64_t> cap(count, 40);
        SVX_CUDA(cudaMemcpyAsync(d_cap.p, cap.data(), count * sizeof(int64_t),
                                 cudaMemcpyHostToDevice, pst));
        float best = 0.f;
        for (size_t c = 0; c < cands.size(); ++c) {
            launch(int(c), d_cap.p, sample);  // warm
            SVX_CUDA(cudaEventRecord(ctx->ev[0], pst));
            launch(int(c), d_cap.p, sample);
            SVX_CUDA(cudaEventRecord(ctx->ev[1], pst));
            SVX_CUDA(cudaEventSynchronize(ctx->ev[1]));
            float ms = 0.f;
            SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
            if (choice < 0 || ms < best) {
                best = ms;
                choice = int(c);
            }
        }
        tuned = choice;
    }
    const BatchConfig& cfg = cands[choice];
    SVX_CUDA(cudaEventRecord(ctx->ev[0], pst));
    if (n_large > 0) {
        // the cluster kernel on the second low-priority stream
        SVX_CUDA(cudaEventRecord(ctx->fork_ev, pst));
        SVX_CUDA(cudaStreamWaitEvent(ctx->aux_stream, ctx->fork_ev, 0));
        launch_batch_cluster(op->ndof, mixed, ctx->aux_stream, n_large, d_order.p + n_small,
                             d_off.p, P.adj_ptr.p, P.adj.p, P.node_base.p, op->vals.p,
                             mixed ? op->vals32.p : nullptr, op->inv_diag.p, op->f.p, op->u.p,
                             r.p, p.p, q.p, d_tol.p, d_maxit.p, d_it.p, d_res.p, d_status.p,
                             mixed ? d_fp32.p : nullptr, u_sv, r_sv, p_sv);
        SVX_CUDA(cudaEventRecord(ctx->join_ev, ctx->aux_stream));
    }
    // the three kinds run side by side: the classes' streams fork before the
    // one-CTA members are launched, and are joined after
    const bool classes = n_general < count;
    if (classes) SVX_CUDA(cudaEventRecord(ctx->fork_ev, pst));
    if (n_small > 0) launch(choice, d_maxit.p, n_small);
    int n_class = 0;
    for (int k0 = n_general; k0 < count; ++n_class) {
        // the run of members of one shape, its window the largest of them
        ResidentShape shape = shapes[ordered[k0]];
        int k1 = k0 + 1;
        for (; k1 < count && shapes[ordered[k1]].ctas == shape.ctas &&
               shapes[ordered[k1]].threads == shape.threads;
             ++k1) {
            shape.window = std::max(shape.window, shapes[ordered[k1]].window);
            shape.smem = std::max(shape.smem, shapes[ordered[k1]].smem);
        }
        if (int(ctx->class_streams.size()) <= n_class) {
            int least = 0, greatest = 0;
            SVX_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
            cudaStream_t cs = nullptr;
            cudaEvent_t ce = nullptr;
            SVX_CUDA(cudaStreamCreateWithPriority(&cs, cudaStreamNonBlocking, least));
            ctx->class_streams.push_back(cs);
            SVX_CUDA(cudaEventCreateWithFlags(&ce, cudaEventDisableTiming));
            ctx->class_events.push_back(ce);
        }
        cudaStream_t cs = ctx->class_streams[n_class];
        SVX_CUDA(cudaStreamWaitEvent(cs, ctx->fork_ev, 0));
        if (op->ndof == 3)
            brick_batch_launch(op, brick, cs, shape.ctas, k1 - k0, d_order.p + k0, op->u.p,
                               d_tol.p, d_maxit.p, d_it.p, d_res.p, d_status.p);
        else
            resident_pcg(ctx, op, shape, false, cs, k1 - k0, d_order.p + k0, d_off.p, d_tol.p,
                         d_maxit.p, d_it.p, d_res.p, d_status.p, op->u.p);
        SVX_CUDA(cudaEventRecord(ctx->class_events[n_class], cs));
        k0 = k1;
    }
    for (int c = 0; c < n_class; ++c)
        SVX_CUDA(cudaStreamWaitEvent(pst, ctx->class_events[c], 0));
    if (n_large > 0) SVX_CUDA(cudaStreamWaitEvent(pst, ctx->join_ev, 0));
    SVX_CUDA(cudaEventRecord(ctx->ev[1], pst));
    SVX_CUDA(cudaEventRecord(ctx->join_ev, pst));
    SVX_CUDA(cudaStreamWaitEvent(st, ctx->join_ev, 0));
    instance_diag_kernel<<<count, 256, 0, st>>>(op->ndof, d_off.p, P.diag_pos.p, op->vals.p,
                                                d_hi.p, d_lo.p);
    SVX_LAUNCH_CHECK();
    member_nnz_kernel<<<(count + 255) / 256, 256, 0, st>>>(count, d_off.p, P.node_base.p,
                                                            d_cap.p);
    SVX_LAUNCH_CHECK();
    std::vector<int64_t> nnz(count);
    SVX_CUDA(cudaMemcpyAsync(nnz.data(), d_cap.p, count * sizeof(int64_t),
                             cudaMemcpyDeviceToHost, st));
    it.resize(count);
    res.resize(count);
    status.resize(count);
    cond.resize(count);
    std::vector<double> hi(count), lo(count);
    std::vector<int64_t> f32(mixed ? count : 0);
    SVX_CUDA(cudaMemcpyAsync(it.data(), d_it.p, count * sizeof(int64_t), cudaMemcpyDeviceToHost,
                             st));
    SVX_CUDA(cudaMemcpyAsync(res.data(), d_res.p, count * sizeof(double), cudaMemcpyDeviceToHost,
                             st));
    SVX_CUDA(cudaMemcpyAsync(status.data(), d_status.p, count * sizeof(int32_t),
                             cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaMemcpyAsync(hi.data(), d_hi.p, count * sizeof(double), cudaMemcpyDeviceToHost,
                             st));
    SVX_CUDA(cudaMemcpyAsync(lo.data(), d_lo.p, count * sizeof(double), cudaMemcpyDeviceToHost,
                             st));
    if (mixed)
        SVX_CUDA(cudaMemcpyAsync(f32.data(), d_fp32.p, count * sizeof(int64_t),
                                 cudaMemcpyDeviceToHost, st));
    SVX_CUDA(cudaStreamSynchronize(st));
    float ms = 0.f;
    SVX_CUDA(cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
    for (int k = 0; k < count; ++k)
        if (status[k] == RESIDENT_STALLED)
            throw ModelFail{SVX_CUDA_ERROR, 0, -1, RESIDENT_STALL_TEXT};
    for (int k = 0; k < count; ++k) cond[k] = hi[k] / lo[k];
    op->has_solution = true;
    if (stats) {
        stats->fp32_iterations = 0;
        for (int64_t v : f32) stats->fp32_iterations += v;
        stats->ms_solve = ms;
        // the shape of the kernel on the assembled K, whoever runs it
        stats->threads_per_cta = cfg.bs;
        stats->lanes_per_node = cfg.g;
        // members of the documented size (3D >= 4,096 rows, 2D >= 16,384), on
        // bricks or on K: clusters solve them all
        stats->cluster_members = 0;
        for (int k = 0; k < count; ++k)
            stats->cluster_members += rows_of(k) >= cluster_min_dof(op->ndof);
        stats->member_nnz = std::move(nnz);
    }
}

}  // namespace svx

// ------------------------------------------------------------ diagnostics
namespace svx {
namespace {

// One block meets a barrier that expects two: nothing ever releases it, so
// the wait must run out, raise the error flag and return.
__global__ void barrier_timeout_kernel(GridBarrier* gb, long long spin_limit, int* out) {
    unsigned int target = 0;
    const bool ok = grid_sync(gb, 2u, target, spin_limit);
    if (threadIdx.x == 0) out[0] = ok ? 1 : 0;
}

}  // namespace
}  // namespace svx

extern "C" int svx_diag_barrier_timeout(int device, long long spins, int* returned_ok,
                                        int* error_flag) {
    using namespace svx;
    if (spins <= 0 || spins > (1LL << 24) || !returned_ok || !error_flag)
        return SVX_BAD_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return SVX_CUDA_ERROR;
    }
    GridBarrier* gb = nullptr;
    int* out = nullptr;
    cudaError_t e = cudaMalloc(&gb, sizeof(GridBarrier));
    if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(gb, 0, sizeof(GridBarrier));
    if (e == cudaSuccess) e = cudaMemset(out, 0xff, sizeof(int));
    if (e == cudaSuccess) {
        barrier_timeout_kernel<<<1, 32>>>(gb, spins, out);
        g_launches.fetch_add(1, std::memory_order_relaxed);
        e = cudaGetLastError();
    }
    GridBarrier h{};
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&h, gb, sizeof(h), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(returned_ok, out, sizeof(int), cudaMemcpyDeviceToHost);
    if (gb) cudaFree(gb);
    if (out) cudaFree(out);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return SVX_CUDA_ERROR;
    }
    *error_flag = int(h.error);
    return SVX_OK;
}
