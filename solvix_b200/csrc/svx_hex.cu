// svx_hex.cu - the FP64 operator of C3D8 models applied element by element.
//
// What bounds it and why this form.  The assembled K of a solid costs 243
// doubles a node and iteration (1,944 bytes, streamed from HBM above the
// L2's size, from L2 below): the node-block SpMV runs at the copy peak and
// cannot get faster without reading less.  The same product from the mesh
// reads 32 bytes of connectivity, 80 bytes of constants and eight node rows
// an element, about a tenth, and costs some 1,300 FP64 operations, a third
// of the time the bytes of K take.  The operator is the one K1 integrates
// (2 x 2 x 2 Gauss points, the reference's inverse Jacobian with its
// cofactor signs, element.rs:441-521); it differs from the assembled K by
// rounding only, and less of it: strains are formed from differences of the
// displacements, where rows of K cancel large entries.  Against a 64-bit
// solution its solves are as near as K's or nearer.
//
// Layout: one thread an element.  The reference gradients at the eight Gauss
// points are sums and differences of the trilinear modes of the nodal values
// (a 2 x 2 x 2 Hadamard transform), so all of an element's work is in
// registers with no shared memory and no shuffles.  Each element writes its
// 24 nodal forces, component-major over the elements, and the node kernel
// sums every node's slots in ascending element order: no atomics, the same
// bits in every run.

// Measured (one B200, us an iteration in the CUDA graph, the assembled K's
// in brackets): 320 x 32 x 32 99 (171), 240 x 24 x 24 40 (80), 180 x 16 x 16
// 22.2 (24.0).  At 320 x 32 x 32 the force kernel takes 59 us (24 at the FP64
// rate), the node kernel 34 (273 MB through L2), the direction 11.

#include "svx_internal.h"
#include "svx_hex.h"

#include <cmath>

namespace svx {

namespace {

constexpr int HB = 128;   // threads of an element block
constexpr int NB = 256;   // threads of a node block

// Sums a, b over the block; thread 0 has them.
template <int T>
__device__ __forceinline__ void block_pair(double& a, double& b, double* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    __syncthreads();
    if (lane == 0) {
        sh[w] = a;
        sh[32 + w] = b;
    }
    __syncthreads();
    if (w == 0) {
        a = lane < T / 32 ? sh[lane] : 0.0;
        b = lane < T / 32 ? sh[32 + lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, off);
            b += __shfl_xor_sync(0xffffffffu, b, off);
        }
    }
}

// True in the last block to arrive; it may then read every block's partials.
__device__ __forceinline__ bool last_to_arrive(unsigned int* counter) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Per element, once an operator: 1 / det J at the Gauss points and the Lame
// constants, scaled by the transforms' powers of two (8^3).
__global__ void hex_setup_kernel(int64_t n_elem, const int32_t* __restrict__ conn,
                                 const double* __restrict__ xyz,
                                 const double* __restrict__ youngs,
                                 const double* __restrict__ poisson, double* __restrict__ rdet,
                                 double2* __restrict__ lame) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= n_elem) return;
    double x[8][3];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const int64_t nd = conn[8 * e + a];
#pragma unroll
        for (int c = 0; c < 3; ++c) x[a][c] = xyz[3 * nd + c];
    }
    HexModes X(x);
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        double J[3][3];
        X.gradient(g, J);
        rdet[g * n_elem + e] = 1.0 / hex_det(J);
    }
    double lam, mu;
    hex_lame(youngs[e], poisson[e], lam, mu);
    lame[e] = make_double2(lam, mu);
}

// The k-th slot of every node as the offset of its first force component
// (~0: none), node-fastest.
__global__ void hex_slots_kernel(int64_t n_nodes, int64_t n_elem, int max_slots,
                                 const int64_t* __restrict__ slot_ptr,
                                 const int32_t* __restrict__ slot_elem,
                                 const uint8_t* __restrict__ slot_local,
                                 uint32_t* __restrict__ slot) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_nodes) return;
    const int64_t s0 = slot_ptr[i], s1 = slot_ptr[i + 1];
    for (int k = 0; k < max_slots; ++k)
        slot[k * n_nodes + i] =
            s0 + k < s1 ? uint32_t(3 * int64_t(slot_local[s0 + k]) * n_elem + slot_elem[s0 + k])
                        : 0xffffffffu;
}

// Node rows of three doubles to rows of four (32 bytes, one 256-bit load).
__global__ void pad_rows_kernel(int64_t n_nodes, const double* __restrict__ x,
                                double* __restrict__ x4) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_nodes) return;
    store_row(x4 + 4 * i, x[3 * i], x[3 * i + 1], x[3 * i + 2]);
}

// Element forces f_e = K_e p_e and p.Kp; the last block forms alpha.  Two
// blocks an SM: the element's work wants 252 registers (at three blocks and
// 168 it spills 650 bytes and gains nothing).
__global__ void __launch_bounds__(HB, 2)
hex_force_kernel(int64_t n_elem, const int32_t* __restrict__ conn,
                 const double* __restrict__ x4, const double* __restrict__ p4,
                 const double* __restrict__ rdet, const double2* __restrict__ lame,
                 double* __restrict__ fe, double* __restrict__ partials,
                 PcgScalars* __restrict__ s) {
    __shared__ double sh[64];
    if (s->status != PCG_RUNNING) return;
    double dot = 0.0, zero = 0.0;
    const int64_t e = int64_t(blockIdx.x) * HB + threadIdx.x;
    if (e < n_elem) {
        int nd[8];
        const int4 c0 = reinterpret_cast<const int4*>(conn)[2 * e],
                   c1 = reinterpret_cast<const int4*>(conn)[2 * e + 1];
        nd[0] = c0.x; nd[1] = c0.y; nd[2] = c0.z; nd[3] = c0.w;
        nd[4] = c1.x; nd[5] = c1.y; nd[6] = c1.z; nd[7] = c1.w;
        double v[8][3];
#pragma unroll
        for (int a = 0; a < 8; ++a) load_row(x4 + 4 * int64_t(nd[a]), v[a]);
        HexModes X(v);
#pragma unroll
        for (int a = 0; a < 8; ++a) load_row(p4 + 4 * int64_t(nd[a]), v[a]);
        HexModes U(v);
        const double2 lm = lame[e];
        HexForces F;
        hex_integrate(X, U, lm.x, lm.y, [&](int g) { return rdet[g * n_elem + e]; }, F);
        double f[8][3];
        F.nodal(f);
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) fe[(3 * a + c) * n_elem + e] = f[a][c];
        dot = F.work(U);
    }
    block_pair<HB>(dot, zero, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = dot;
    if (last_to_arrive(&s->count_a)) {
        double t = 0.0, u = 0.0;
        for (int k = threadIdx.x; k < int(gridDim.x); k += HB) t += __ldcg(partials + k);
        block_pair<HB>(t, u, sh);
        if (threadIdx.x == 0) {
            s->count_a = 0;
            s->pap = t;
            if (t > 0.0) {
                s->alpha = s->rz / t;
            } else {  // p.Kp <= 0 or NaN: breakdown
                s->it = s->it + 1;
                s->res = sqrt(s->rr) / s->bnorm;
                s->status = PCG_BREAKDOWN;
            }
        }
    }
}

// q from the slots, u += alpha p, r -= alpha q; r.r and r.z, beta by the
// last block (update_kernel's rules).
__global__ void __launch_bounds__(NB)
hex_update_kernel(int64_t n_nodes, int max_slots, const uint32_t* __restrict__ slot,
                  int64_t n_elem, const double* __restrict__ fe,
                  const uint8_t* __restrict__ fixed, const double* __restrict__ inv_diag,
                  const double* __restrict__ p4, double* __restrict__ u, double* __restrict__ r,
                  double* __restrict__ partials, PcgScalars* __restrict__ s) {
    __shared__ double sh[64];
    if (s->status != PCG_RUNNING) return;
    const double alpha = s->alpha;
    double rr = 0.0, rz = 0.0;
    const int64_t i = int64_t(blockIdx.x) * NB + threadIdx.x;
    if (i < n_nodes) {
        double q[3] = {0.0, 0.0, 0.0};
        for (int k0 = 0; k0 < max_slots; k0 += 8) {
            uint32_t o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                o[k] = k0 + k < max_slots ? slot[(k0 + k) * n_nodes + i] : 0xffffffffu;
            double v[8][3];
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    v[k][c] = o[k] != 0xffffffffu ? __ldcg(fe + c * n_elem + o[k]) : 0.0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int c = 0; c < 3; ++c) q[c] += v[k][c];
        }
        double p[3];
        load_row(p4 + 4 * i, p);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int64_t row = 3 * i + c;
            u[row] += alpha * p[c];
            // a constrained row of K is its diagonal, and p is zero there
            const double ri = fixed[row] ? r[row] : r[row] - alpha * q[c];
            r[row] = ri;
            const double zi = ri * inv_diag[row];
            rr += ri * ri;
            rz += ri * zi;
        }
    }
    block_pair<NB>(rr, rz, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = rr;
        partials[2 * blockIdx.x + 1] = rz;
    }
    if (last_to_arrive(&s->count_b)) {
        double a = 0.0, b = 0.0;
        for (int k = threadIdx.x; k < int(gridDim.x); k += NB) {
            a += __ldcg(partials + 2 * k);
            b += __ldcg(partials + 2 * k + 1);
        }
        block_pair<NB>(a, b, sh);
        if (threadIdx.x == 0) {
            s->count_b = 0;
            s->it = s->it + 1;
            s->rr = a;
            const double res = sqrt(a) / s->bnorm;
            s->res = res;
            if (res <= s->tol) {
                s->status = PCG_CONVERGED;
            } else if (s->it >= s->max_iter) {
                s->status = PCG_MAXITER;
            } else if (a <= s->rr_stop) {
                s->status = PCG_RELIABLE;  // s->rz stays r.z of the previous iterate
            } else {
                s->beta = b / s->rz;
                s->rz = b;
            }
        }
    }
}

// p = z + beta p, rows of three and of four.
__global__ void __launch_bounds__(NB)
hex_direction_kernel(int64_t n_nodes, const double* __restrict__ r,
                     const double* __restrict__ inv_diag, double* __restrict__ p,
                     double* __restrict__ p4, const PcgScalars* __restrict__ s) {
    if (s->status != PCG_RUNNING) return;
    const double beta = s->beta;
    const int64_t i = int64_t(blockIdx.x) * NB + threadIdx.x;
    if (i >= n_nodes) return;
    double v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int64_t row = 3 * i + c;
        v[c] = r[row] * inv_diag[row] + beta * p[row];
        p[row] = v[c];
    }
    store_row(p4 + 4 * i, v[0], v[1], v[2]);
}

unsigned blocks(int64_t n, int t) { return unsigned((n + t - 1) / t); }

}  // namespace

bool hex_applies(const svx_ctx* ctx, const svx_op* op) {
    return ctx->hex && op->ndof == 3 && op->all_hex && op->mass_rho < 0.0 &&
           op->n_nodes >= ctx->hex_min_nodes && 24 * op->n_elem < int64_t(0xffffffffu);
}

void hex_prepare(svx_ctx* ctx, svx_op* op) {
    HexOperator& h = op->hex;
    if (h.slot.p && !h.stale) return;
    cudaStream_t st = ctx->stream;
    const Pattern& P = op->pat;
    if (!h.slot.p) {
        h.rdet.alloc(ctx->pool, size_t(op->n_elem) * 8);
        h.lame.alloc(ctx->pool, size_t(op->n_elem));
        h.x4.alloc(ctx->pool, size_t(op->n_nodes) * 4);
        h.slot.alloc(ctx->pool, size_t(op->n_nodes) * std::max(P.max_slots, 1));
        hex_slots_kernel<<<blocks(op->n_nodes, NB), NB, 0, st>>>(
            op->n_nodes, op->n_elem, P.max_slots, P.slot_ptr.p, P.slot_elem.p, P.slot_local.p,
            h.slot.p);
        SVX_LAUNCH_CHECK();
    }
    hex_setup_kernel<<<blocks(op->n_elem, HB), HB, 0, st>>>(
        op->n_elem, op->conn.p, op->xyz.p, op->youngs.p, op->poisson.p, h.rdet.p, h.lame.p);
    SVX_LAUNCH_CHECK();
    pad_rows_kernel<<<blocks(op->n_nodes, NB), NB, 0, st>>>(op->n_nodes, op->xyz.p, h.x4.p);
    SVX_LAUNCH_CHECK();
    h.stale = false;
}

void HexWork::alloc(svx_ctx* ctx, const svx_op* op) {
    fe.alloc(ctx->pool, size_t(op->n_elem) * 24);
    p4.alloc(ctx->pool, size_t(op->n_nodes) * 4);
    partials.alloc(ctx->pool, std::max<size_t>(blocks(op->n_elem, HB),
                                               2 * size_t(blocks(op->n_nodes, NB))) + 2);
}

void hex_start(const svx_op* op, HexWork& w, cudaStream_t st, const double* p) {
    pad_rows_kernel<<<blocks(op->n_nodes, NB), NB, 0, st>>>(op->n_nodes, p, w.p4.p);
    SVX_LAUNCH_CHECK();
}

void hex_iteration(const svx_op* op, HexWork& w, cudaStream_t st, const double* inv_diag,
                   double* u, double* r, double* p, PcgScalars* s) {
    const HexOperator& h = op->hex;
    hex_force_kernel<<<blocks(op->n_elem, HB), HB, 0, st>>>(
        op->n_elem, op->conn.p, h.x4.p, w.p4.p, h.rdet.p, h.lame.p, w.fe.p, w.partials.p, s);
    hex_update_kernel<<<blocks(op->n_nodes, NB), NB, 0, st>>>(
        op->n_nodes, op->pat.max_slots, h.slot.p, op->n_elem, w.fe.p, op->is_fixed.p, inv_diag,
        w.p4.p, u, r, w.partials.p, s);
    hex_direction_kernel<<<blocks(op->n_nodes, NB), NB, 0, st>>>(op->n_nodes, r, inv_diag, p,
                                                                 w.p4.p, s);
}

}  // namespace svx
