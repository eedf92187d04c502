// svx_brick.cu - Jacobi-PCG of C3D8 models on replicated bricks: the
// elements of a model are dealt out to CTAs, and a CTA keeps every node its
// elements touch.
//
// What bounds it and why this split.  With the element-by-element operator
// (svx_hex.h) a model's iteration needs little memory, so below a few
// hundred thousand elements what is left is the FP64 pipe and the waits
// between CTAs.  A brick holds its nodes' p in shared memory and sums its
// own elements' forces there; the one thing bricks exchange is, for a node
// that several of them touch, each one's partial force.  Every brick then
// adds the partials in the same order and updates r, u, z and p of all its
// nodes itself, so the copies of a shared node stay bitwise equal and p is
// never sent: two barriers an iteration, one for p.Kp (the sum of the
// elements' p_e.f_e) and the partial forces, one for r.r and r.z.
//
// Bricks are runs of elements ordered by layers along the model's longest
// side, so a cantilever's bricks are slabs with two neighbours; any order is
// correct.  A brick's elements are taken in chunks of CH, one element a
// thread; forces are staged in shared memory and each node sums its own in
// ascending order, without atomics.
//
// Measured (one B200): 160 x 16 x 16 15.5 us an iteration (19.7 on the
// assembled K from L2), 120 x 12 x 12 10.3 (13.3), 120 x 10 x 10 9.5 (11.3);
// below some 14,000 nodes K from L2 is as fast, above 288 elements a CTA the
// graph form (svx_hex.cu) is.  40 members of 20..120 x 4..16^2 as one batch:
// 99 ms of device time (224 on clusters streaming K from HBM).  An iteration
// of the 160 x 16 x 16 model, in thousands of cycles of a CTA: forces 11.4 (a
// full chunk of two warps a scheduler at the FP64 rate, and one of 21
// elements), their sums 3.2, the two exchanges 12 with the wait for the
// slowest brick, node updates 3.6 (posting the sums as numbered 128-bit words
// that every CTA polls, instead of the counting barrier: 16.4 us).
//
// GRID: one model over the whole device (cooperative launch), chunks of
// iterations on PcgScalars' state like the other persistent
// kernels.  Otherwise: one cluster per batch member, its whole solve.

#include "svx_internal.h"
#include "svx_hex.h"
#include "svx_grid.h"
#include "svx_warp.h"

#include <cmath>

namespace svx {

namespace {

constexpr int CH = 256;             // threads, and elements of a chunk (255 registers each)
constexpr int WARPS = CH / 32;
// staged forces of a chunk: pitch of a component, an element's place (one
// double skipped in 16, or a layer of 16 elements would lie in one bank) and
// the column of zeros
constexpr int FP = CH + CH / 16 + 2, FZERO = CH + CH / 16;
__device__ __forceinline__ int fplace(int e) { return e + e / 16; }
constexpr int CN = 3 * CH;          // nodes a chunk may touch
constexpr int SORT_CHUNK = 4096;    // sort of a chunk's references (a power of two)
constexpr int SORT_BRICK = 16384;   // references of a brick (BRICK_MAX_ELEMS x 8)
constexpr int GEO = 31;             // constants of an element: 21 modes, 8 1/det, lam, mu
constexpr int BT = 512;             // threads of the build kernels
constexpr int SHARE = 8;            // bricks that may touch a node

// ------------------------------------------------------------ building
// The layer of every element along its member's longest side; one CTA a
// member of the list (those with bricks: a batch may have any number of
// others, and more members than a grid's y or z dimension).
__global__ void __launch_bounds__(1024)
layer_kernel(const int32_t* __restrict__ list, const int64_t* __restrict__ node_off,
             const int64_t* __restrict__ elem_off, const int32_t* __restrict__ conn,
             const double* __restrict__ xyz, uint16_t* __restrict__ layer,
             int32_t* __restrict__ hist) {
    __shared__ double box[6][32];
    const int member = list[blockIdx.x];
    const int64_t n0 = node_off[member], n1 = node_off[member + 1];
    const int64_t e0 = elem_off[member], e1 = elem_off[member + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double b[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) b[c] = INFINITY;  // minima of x, y, z, -x, -y, -z
    for (int64_t i = n0 + threadIdx.x; i < n1; i += 1024)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double v = xyz[3 * i + c];
            b[c] = fmin(b[c], v);
            b[3 + c] = fmin(b[3 + c], -v);
        }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        for (int off = 16; off > 0; off >>= 1)
            b[c] = fmin(b[c], __shfl_xor_sync(0xffffffffu, b[c], off));
        if (lane == 0) box[c][warp] = b[c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 6; ++c)
        for (int w = 0; w < 32; ++w) b[c] = fmin(b[c], box[c][w]);
    double ext[3], vol = 1.0, longest = 0.0;
    int axis = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        ext[c] = -b[3 + c] - b[c];
        vol *= ext[c];
        if (ext[c] > longest) {
            longest = ext[c];
            axis = c;
        }
    }
    const double h = cbrt(vol / double(e1 - e0));
    double lay = rint(longest / h);
    lay = lay >= 1.0 ? fmin(lay, double(BRICK_LAYERS)) : 1.0;  // 1 where it is not a number
    const double lo = b[axis], scale = lay / longest;
    for (int64_t e = e0 + threadIdx.x; e < e1; e += 1024) {
        double s = 0.0;
        for (int a = 0; a < 8; ++a) s += xyz[3 * int64_t(conn[8 * e + a]) + axis];
        double q = (s * 0.125 - lo) * scale;
        q = q > 0.0 ? fmin(q, lay - 1.0) : 0.0;
        layer[e] = uint16_t(q);
        atomicAdd(&hist[int64_t(blockIdx.x) * BRICK_LAYERS + int(q)], 1);
    }
}

// Elements by layer, in index order within a layer: gridDim.y CTAs a member
// of the list share its layers (a CTA a layer for a single model; 16 a member
// of a batch, where most of 1,024 would find an empty layer).  pos, if any,
// gets each element's place in the order.
__global__ void __launch_bounds__(256)
layer_order_kernel(const int32_t* __restrict__ list, const int64_t* __restrict__ elem_off,
                   const uint16_t* __restrict__ layer, const int32_t* __restrict__ hist,
                   int32_t* __restrict__ order, int32_t* __restrict__ pos) {
    __shared__ int sums[8], base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int member = list[blockIdx.x];
    const int32_t* h = hist + int64_t(blockIdx.x) * BRICK_LAYERS;
    const int64_t e0 = elem_off[member], e1 = elem_off[member + 1];
    for (int L = blockIdx.y; L < BRICK_LAYERS; L += gridDim.y) {
        if (h[L] == 0) continue;
        if (threadIdx.x == 0) base = 0;
        __syncthreads();
        int before = 0;
        for (int k = threadIdx.x; k < L; k += 256) before += h[k];
        if (before) atomicAdd(&base, before);
        __syncthreads();
        int at = base;
        for (int64_t c = e0; c < e1; c += 256) {
            const int64_t e = c + threadIdx.x;
            const bool in = e < e1 && layer[e] == L;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (lane == 0) sums[warp] = __popc(m);
            __syncthreads();
            int rank = at + __popc(m & ((1u << lane) - 1u)), all = 0;
            for (int w = 0; w < 8; ++w) {
                if (w < warp) rank += sums[w];
                all += sums[w];
            }
            if (in) {
                order[e0 + rank] = int32_t(e);
                if (pos) pos[e] = int32_t(e0 + rank);
            }
            at += all;
            __syncthreads();
        }
    }
}

// Nodes of a single model that more than three of its bricks would share
// (brick k: the elements [n_elem k / bricks, n_elem (k + 1) / bricks) in
// order), from the pattern's incidence lists.
__global__ void crowded_kernel(int64_t n_nodes, int64_t n_elem, int64_t bricks,
                               const int64_t* __restrict__ slot_ptr,
                               const int32_t* __restrict__ slot_elem,
                               const int32_t* __restrict__ pos, int* __restrict__ crowded) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int n = 0;
    if (i < n_nodes) {
        int64_t seen[3] = {-1, -1, -1};
        for (int64_t s = slot_ptr[i]; s < slot_ptr[i + 1] && n <= 3; ++s) {
            const int64_t k = ((int64_t(pos[slot_elem[s]]) + 1) * bricks - 1) / n_elem;
            if (k == seen[0] || k == seen[1] || k == seen[2]) continue;
            if (n < 3) seen[n] = k;
            ++n;
        }
    }
    const int many = __syncthreads_count(n > 3);
    if (threadIdx.x == 0 && many) atomicAdd(crowded, many);
}

__device__ void bitonic(uint32_t* key, int m) {
    for (int k = 2; k <= m; k *= 2)
        for (int j = k / 2; j > 0; j /= 2) {
            for (int q = threadIdx.x; q < m / 2; q += BT) {
                const int i = 2 * q - (q & (j - 1)), p = i + j;
                const uint32_t x = key[i], y = key[p];
                if ((x > y) == ((i & k) == 0)) {
                    key[i] = y;
                    key[p] = x;
                }
            }
            __syncthreads();
        }
}

// Exclusive sum of a per-thread count over the block; total to all.
__device__ int block_scan(int v, int* sh, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < BT / 32; ++w) {
        if (w < warp) before += sh[w];
        total += sh[w];
    }
    __syncthreads();
    return before + x - v;
}

// A brick's node list, its elements' local connectivity and its chunks'
// force sums: one CTA a brick, sorts in shared memory.
__global__ void __launch_bounds__(BT)
brick_build_kernel(BrickView b, const int32_t* __restrict__ conn, int32_t* ent_n, int* fail) {
    extern __shared__ __align__(16) unsigned char dyn[];
    uint32_t* key = reinterpret_cast<uint32_t*>(dyn);  // [SORT_BRICK]
    uint32_t* node = key + SORT_BRICK;                 // [b.ncap]
    __shared__ int sh[BT / 32];
    const int brick = blockIdx.x;
    const int e0 = b.elem0[brick], e1 = b.elem1[brick];
    const int refs = 8 * (e1 - e0);
    int m = 2;
    while (m < refs) m *= 2;
    for (int q = threadIdx.x; q < m; q += BT)
        key[q] = q < refs ? uint32_t(conn[8 * int64_t(b.order[e0 + q / 8]) + q % 8]) : ~0u;
    __syncthreads();
    bitonic(key, m);
    // the distinct nodes, ascending; each thread a contiguous run of keys
    const int per = (refs + BT - 1) / BT, q0 = min(refs, per * int(threadIdx.x)),
              q1 = min(refs, q0 + per);
    int count = 0;
    for (int q = q0; q < q1; ++q) count += q == 0 || key[q] != key[q - 1];
    int nn;
    int at = block_scan(count, sh, nn);
    const uint32_t base = b.node0[brick];
    if (nn > int(b.node0[brick + 1] - base)) {
        if (threadIdx.x == 0) fail[b.member[brick]] = 1;
        return;
    }
    for (int q = q0; q < q1; ++q)
        if (q == 0 || key[q] != key[q - 1]) node[at++] = key[q];
    __syncthreads();
    if (threadIdx.x == 0) b.count[brick] = nn;
    for (int l = threadIdx.x; l < nn; l += BT) {
        const uint32_t nd = node[l];
        b.node[base + l] = int32_t(nd);
        const int k = atomicAdd(&ent_n[nd], 1);
        if (k < SHARE) b.entry[int64_t(nd) * SHARE + k] = base + uint32_t(l);
        else fail[b.member[brick]] = 1;
    }
    for (int q = threadIdx.x; q < refs; q += BT) {
        const uint32_t nd = uint32_t(conn[8 * int64_t(b.order[e0 + q / 8]) + q % 8]);
        int lo = 0, hi = nn - 1;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (node[mid] < nd) lo = mid + 1;
            else hi = mid;
        }
        b.lconn[8 * int64_t(e0) + q] = uint16_t(lo);
    }
    __syncthreads();
    // the chunks: references sorted by (node, element, corner)
    int held_nodes = 0;
    for (int c = 0, f0 = e0; f0 < e1; ++c, f0 += CH) {
        const int cr = 8 * min(CH, e1 - f0);
        const int64_t chunk = b.chunk0[brick] + c;
        __syncthreads();
        for (int q = threadIdx.x; q < SORT_CHUNK; q += BT)
            key[q] = q < cr ? (uint32_t(b.lconn[8 * int64_t(f0) + q]) << 12) | uint32_t(q) : ~0u;
        __syncthreads();
        bitonic(key, SORT_CHUNK);
        const int cp = (cr + BT - 1) / BT, k0 = min(cr, cp * int(threadIdx.x)),
                  k1 = min(cr, k0 + cp);
        int cc = 0;
        for (int q = k0; q < k1; ++q) cc += q == 0 || (key[q] >> 12) != (key[q - 1] >> 12);
        int cn;
        int ca = block_scan(cc, sh, cn);
        held_nodes += (cn + 1) & ~1;
        if (cn > CN || held_nodes > b.lists) {
            if (threadIdx.x == 0) fail[b.member[brick]] = 1;
            return;
        }
        for (int q = k0; q < k1; ++q) {
            const uint32_t l = key[q] >> 12;
            if (q > 0 && l == key[q - 1] >> 12) continue;
            b.cnode[chunk * CN + ca] = uint16_t(l);
            uint16_t* to = b.ref + (chunk * CN + ca) * 8;
            int n = 0;
            for (; q + n < cr && key[q + n] >> 12 == l; ++n)
                if (n < 8) {
                    const int ref = int(key[q + n] & 4095u);  // element * 8 + corner
                    to[n] = uint16_t(3 * (ref & 7) * FP + fplace(ref >> 3));
                }
            if (n > 8) fail[b.member[brick]] = 1;
            for (; n < 8; ++n) to[n] = uint16_t(FZERO);
            ++ca;
        }
        if (threadIdx.x == 0) b.ccount[chunk] = cn;
    }
}

// Every node's entries in ascending brick order; gridDim.y CTAs a member of
// the list.
__global__ void entry_sort_kernel(const int32_t* __restrict__ list,
                                  const int64_t* __restrict__ node_off,
                                  uint32_t* __restrict__ entry,
                                  const int32_t* __restrict__ ent_n, int* __restrict__ fail) {
    const int member = list[blockIdx.x];
    const int64_t n1 = node_off[member + 1];
    for (int64_t i = node_off[member] + int64_t(blockIdx.y) * blockDim.x + threadIdx.x;
         i < n1; i += int64_t(gridDim.y) * blockDim.x) {
        const int n = min(ent_n[i], SHARE);
        if (n == 0) fail[member] = 1;
        uint32_t* e = entry + i * SHARE;
        for (int a = 1; a < n; ++a) {
            const uint32_t v = e[a];
            int k = a;
            for (; k > 0 && e[k - 1] > v; --k) e[k] = e[k - 1];
            e[k] = v;
        }
        for (int a = n; a < SHARE; ++a) e[a] = ~0u;
    }
}

// The elements' constants, in brick order: one CTA a brick.
__global__ void __launch_bounds__(CH)
geometry_kernel(BrickView b, int64_t n_elem, const int32_t* __restrict__ conn,
                const double* __restrict__ xyz, const double* __restrict__ youngs,
                const double* __restrict__ poisson, double* __restrict__ geo) {
    for (int64_t k = b.elem0[blockIdx.x] + int64_t(threadIdx.x); k < b.elem1[blockIdx.x];
         k += CH) {
        const int64_t e = b.order[k];
        double x[8][3];
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int64_t nd = conn[8 * e + a];
#pragma unroll
            for (int c = 0; c < 3; ++c) x[a][c] = xyz[3 * nd + c];
        }
        HexModes X(x);
#pragma unroll
        for (int q = 0; q < 21; ++q) geo[q * n_elem + k] = X.at(q);
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            double J[3][3];
            X.gradient(g, J);
            geo[(21 + g) * n_elem + k] = 1.0 / hex_det(J);
        }
        double lam, mu;
        hex_lame(youngs[e], poisson[e], lam, mu);
        geo[29 * n_elem + k] = lam;
        geo[30 * n_elem + k] = mu;
    }
}

// ------------------------------------------------------------ solving
__device__ __forceinline__ void copy_async4(void* to, const void* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     unsigned(__cvta_generic_to_shared(to))), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_async16(void* to, const void* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     unsigned(__cvta_generic_to_shared(to))), "l"(from) : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}
constexpr int MAX_CHUNKS = (BRICK_MAX_ELEMS + CH - 1) / CH;
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
struct BrickArgs {
    BrickView b;
    int64_t n_elem;
    const double* geo;
    const uint8_t* fixed;
    const double* inv_diag;
    const double* f;          // batch: right-hand side
    double *u, *r, *p;        // node vectors (grid: state between launches)
    double *rb, *ub, *db;     // bricks' copies of r, u, 1 / K_ii (vectors not in shared memory)
    double* rows;             // [2][slots][4] partial forces, in turn
    double* part;             // [3][bricks] sums of each brick: p.Kp, then r.r and r.z
    // grid
    PcgScalars* s;
    GridBarrier* gb;
    int chunk;
    // batch
    const int32_t* order;
    const int32_t* member_brick;
    const double* tol;
    const int64_t* max_iter;
    int64_t* out_it;
    double* out_res;
    int32_t* out_status;
};

// GRID: the whole device works on one model, whose bricks are small enough
// that all they need stays in shared memory (SM).  Otherwise a cluster works
// on a batch member and a CTA may take several chunks.
template <bool GRID>
__global__ void __launch_bounds__(CH, 1) brick_pcg_kernel(BrickArgs a) {
    constexpr bool SM = GRID;
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double wa[WARPS], wb[2 * WARPS], tot[3];
    const BrickView& b = a.b;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int brick, brick0, nb, inst = 0;
    if constexpr (GRID) {
        brick = int(blockIdx.x);
        brick0 = 0;
        nb = int(gridDim.x);
        if (*reinterpret_cast<volatile int*>(&a.s->status) != PCG_RUNNING) return;
    } else {
        unsigned rank, ctas;
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
        inst = a.order[blockIdx.x / ctas];
        brick0 = a.member_brick[inst];
        nb = int(ctas);
        brick = brick0 + int(rank);
    }
    const int e0 = b.elem0[brick], e1 = b.elem1[brick];
    const int nn = b.count[brick];
    // (read from memory, a single model's would cost this kernel 130 bytes of
    // spills and a tenth of its time)
    const int64_t base = GRID ? int64_t(brick) * b.ncap : int64_t(b.node0[brick]);
    const int chunks = (e1 - e0 + CH - 1) / CH;
    // shared memory: staged forces, element constants, force sums (of all
    // chunks in SM, of one otherwise), p, q (and r, u, 1 / K_ii),
    // sharing, mask
    const int held = SM ? b.held : CH;     // elements whose constants are held
    const int lists = SM ? b.lists : CN;   // chunk nodes whose sums are held
    double* fs = reinterpret_cast<double*>(dyn);  // [24][FP]
    double* es = fs + 24 * FP;                    // [GEO][held], or [10][CH] without the modes
    uint4* cref = reinterpret_cast<uint4*>(es + (SM ? GEO : 10) * held);  // [lists]
    uint16_t* cnode = reinterpret_cast<uint16_t*>(cref + lists);         // [lists]
    double* ps = reinterpret_cast<double*>(cnode + lists);
    double* qs = ps + 3 * b.ncap;
    double* rs = SM ? qs + 3 * b.ncap : a.rb + 3 * base;
    double* us = SM ? rs + 3 * b.ncap : a.ub + 3 * base;
    double* ds = SM ? us + 3 * b.ncap : a.db + 3 * base;
    // the other bricks' copies of a node, ascending, up to two (SM) or one
    uint32_t* other = reinterpret_cast<uint32_t*>((SM ? ds : qs) + 3 * b.ncap);
    uint8_t* mask = reinterpret_cast<uint8_t*>(other + (SM ? 2 : 1) * b.ncap);
    // mask bits 0-2: constrained rows; 3: owned (counted in the sums); 4: more
    // bricks share the node than `other` lists
    const unsigned NONE = ~0u;
    double lrr = 0.0, lrz = 0.0;
    for (int l = t; l < nn; l += CH) {
        const int64_t nd = b.node[base + l];
        const uint32_t* ent = b.entry + nd * SHARE;
        const uint32_t own = uint32_t(base + l);
        unsigned m = ent[0] == own ? 8u : 0u;
        if (ent[SM ? 3 : 2] != NONE) m |= 16u;
        other[l] = ent[1] == NONE ? NONE : ent[0] == own ? ent[1] : ent[0];
        if (SM)
            other[b.ncap + l] = ent[1] == NONE || ent[2] == NONE         ? NONE
                                : ent[0] == own || ent[1] == own ? ent[2] : ent[1];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int64_t row = 3 * nd + c;
            if (a.fixed[row]) m |= 1u << c;
            const double d = a.inv_diag[row];
            ds[3 * l + c] = d;
            if constexpr (GRID) {
                rs[3 * l + c] = a.r[row];
                us[3 * l + c] = a.u[row];
                ps[3 * l + c] = a.p[row];
            } else {
                const double ri = a.f[row], zi = ri * d;
                rs[3 * l + c] = ri;
                us[3 * l + c] = 0.0;
                ps[3 * l + c] = zi;
                if (m & 8u) {
                    lrr += ri * ri;
                    lrz += ri * zi;
                }
            }
        }
        mask[l] = uint8_t(m);
    }
    // SM: the elements' constants and the force sums are copied once.
    // Otherwise the lists come by asynchronous copies while the chunk's forces
    // are formed, and the constants of the next chunk through registers while
    // the forces are summed (the modes stay there, the others go to the
    // thread's own shared memory).
    __shared__ int chunk_nodes[MAX_CHUNKS], chunk_at[MAX_CHUNKS];
    HexModes X;
    double late[10];
    uint4 lc = make_uint4(0, 0, 0, 0);
    auto fetch = [&](int c) {
        const int64_t k = e0 + c * CH + t;
        if (k < e1) {
#pragma unroll
            for (int q = 0; q < 21; ++q) X.at(q) = __ldg(a.geo + q * a.n_elem + k);
#pragma unroll
            for (int q = 0; q < 10; ++q) late[q] = __ldg(a.geo + (21 + q) * a.n_elem + k);
            lc = __ldg(reinterpret_cast<const uint4*>(b.lconn) + k);
        }
    };
    auto keep_late = [&]() {
#pragma unroll
        for (int q = 0; q < 10; ++q) es[q * CH + t] = late[q];
    };
    auto fetch_lists = [&](int c, int at) {
        const int64_t ch = b.chunk0[brick] + c;
        const int cc = chunk_nodes[c];
        for (int j = t; j < cc; j += CH) copy_async16(cref + at + j, b.ref + (ch * CN + j) * 8);
        for (int j = t; j < (cc + 1) / 2; j += CH)
            copy_async4(cnode + at + 2 * j, b.cnode + ch * CN + 2 * j);
    };
    for (int c = t; c < chunks; c += CH) chunk_nodes[c] = b.ccount[b.chunk0[brick] + c];
    for (int q = t; q < 3; q += CH) fs[q * FP + FZERO] = 0.0;
    __syncthreads();
    if (t == 0)
        for (int c = 0, at = 0; c < chunks; ++c) {
            chunk_at[c] = SM ? at : 0;
            at += (chunk_nodes[c] + 1) & ~1;
        }
    __syncthreads();
    if constexpr (SM) {
        for (int k = t; k < e1 - e0; k += CH)
            for (int q = 0; q < GEO; ++q) es[q * held + k] = a.geo[q * a.n_elem + e0 + k];
        for (int c = 0; c < chunks; ++c) fetch_lists(c, chunk_at[c]);
    } else {
        fetch(0);
        keep_late();
        fetch_lists(0, 0);
    }
    copies_done();
    unsigned target = 0;
    auto meet = [&]() -> bool {
        if constexpr (GRID) return grid_sync(a.gb, gridDim.x, target);
        cluster_meet();
        return true;
    };
    double* part_a = a.part + brick0;
    double* part_b = a.part + ((b.bricks + 1) & ~1) + 2 * brick0;  // 16-byte aligned
    // r.r and r.z of this CTA to `part_b`; the model's after the CTAs met, read
    // by one warp (all warps of 148 CTAs reading the same few lines took 3,800
    // cycles)
    auto sums_b = [&](double x, double y, double& tx, double& ty) -> bool {
        const double v = lane_sum_pair(x, y, lane);
        if ((lane & 15) == 0) wb[2 * warp + (lane >> 4)] = v;
        __syncthreads();
        if (warp == 0) {
            const double w = lane_sum_pair(lane < WARPS ? wb[2 * lane] : 0.0,
                                           lane < WARPS ? wb[2 * lane + 1] : 0.0, lane);
            if ((lane & 15) == 0) part_b[2 * (brick - brick0) + (lane >> 4)] = w;
        }
        if (!meet()) return false;
        if (warp == 0) {
            double sx = 0.0, sy = 0.0;
            for (int k = lane; k < nb; k += 32) {
                const double2 w = __ldcg(reinterpret_cast<const double2*>(part_b) + k);
                sx += w.x;
                sy += w.y;
            }
            sx = lane_sum(sx);
            sy = lane_sum(sy);
            if (lane == 0) {
                tot[1] = sx;
                tot[2] = sy;
            }
        }
        __syncthreads();
        tx = tot[1];
        ty = tot[2];
        return true;
    };
    __syncthreads();
    double rz, rr, bnorm, tol, rr_stop = -1.0;
    long long it = 0, max_iter;
    int status = PCG_RUNNING;
    if constexpr (GRID) {
        volatile PcgScalars* s = a.s;
        rz = s->rz;
        rr = s->rr;
        bnorm = s->bnorm;
        tol = s->tol;
        rr_stop = s->rr_stop;
        it = s->it;
        max_iter = s->max_iter;
    } else {
        tol = a.tol[inst];
        max_iter = a.max_iter[inst];
        sums_b(lrr, lrz, rr, rz);
        bnorm = sqrt(rr);
        if (bnorm == 0.0) status = PCG_CONVERGED;
    }
    // above this r.r, sqrt(r.r) / ||f|| cannot round to tol or less
    double surely = (tol * bnorm) * (tol * bnorm) * (1.0 + 1e-12);
    if (surely < 1e-280) surely = INFINITY;  // the square left the normal range
    __syncthreads();
    for (int step = 0; status == PCG_RUNNING && (!GRID || step < a.chunk); ++step) {
        const int64_t turn_at = (step & 1) * (GRID ? int64_t(b.bricks) * b.ncap : b.slots);
        double* rows = a.rows + 4 * turn_at;
        auto share = [&](int l, const double (&q)[3]) {
            store_row(rows + 4 * (base + l), q[0], q[1], q[2]);
        };
        // ---- forces of the own elements, summed at the own nodes
        double dot = 0.0;
        if (chunks > 1) {
            for (int l = t; l < 3 * nn; l += CH) qs[l] = 0.0;
        }
        for (int c = 0; c < chunks; ++c) {
            if (e0 + c * CH + t < e1) {
                const double* g0 = SM ? es + c * CH + t : es + t;
                if constexpr (SM) {
                    lc = __ldg(reinterpret_cast<const uint4*>(b.lconn) + e0 + c * CH + t);
#pragma unroll
                    for (int q = 0; q < 21; ++q) X.at(q) = g0[q * held];
                    g0 += 21 * held;
                }
                double v[8][3];
                const unsigned w[4] = {lc.x, lc.y, lc.z, lc.w};
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const double* row = ps + 3 * ((w[q / 2] >> (16 * (q % 2))) & 0xffffu);
#pragma unroll
                    for (int d = 0; d < 3; ++d) v[q][d] = row[d];
                }
                HexModes U(v);
                HexForces F;
                hex_integrate(X, U, g0[8 * held], g0[9 * held],
                              [&](int g) { return g0[g * held]; }, F);
                dot += F.work(U);
                F.nodal(v);
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) fs[(3 * q + d) * FP + fplace(t)] = v[q][d];
            }
            if (!SM && chunks > 1) copies_done();  // this chunk's lists
            __syncthreads();
            const int cc = chunk_nodes[c];
            const int at = SM ? chunk_at[c] : 0, next = c + 1 < chunks ? c + 1 : 0;
            if (!SM && chunks > 1) fetch(next);
            for (int j = t; j < cc; j += CH) {
                const int l = cnode[at + j];
                const uint4 w = cref[at + j];
                const unsigned ref[4] = {w.x, w.y, w.z, w.w};
                double x[8][3];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const double* src = fs + ((ref[k / 2] >> (16 * (k % 2))) & 0xffffu);
#pragma unroll
                    for (int d = 0; d < 3; ++d) x[k][d] = src[d * FP];
                }
                double q[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    q[d] = x[0][d];
#pragma unroll
                    for (int k = 1; k < 8; ++k) q[d] += x[k][d];
                }
                if (chunks > 1)
#pragma unroll
                    for (int d = 0; d < 3; ++d) q[d] += qs[3 * l + d];
#pragma unroll
                for (int d = 0; d < 3; ++d) qs[3 * l + d] = q[d];
                if (chunks == 1 && other[l] != NONE) share(l, q);
            }
            if (chunks > 1) __syncthreads();  // the staged forces are read
            if (!SM && chunks > 1) {
                keep_late();
                fetch_lists(next, 0);
            }
        }
        if (chunks > 1)
            for (int l = t; l < nn; l += CH)
                if (other[l] != NONE) {
                    const double q[3] = {qs[3 * l], qs[3 * l + 1], qs[3 * l + 2]};
                    share(l, q);
                }
        // ---- the CTAs meet: p.Kp, and the partial forces
        dot = lane_sum(dot);
        if (lane == 0) wa[warp] = dot;
        __syncthreads();
        if (warp == 0) {
            const double w = lane_sum(lane < WARPS ? wa[lane] : 0.0);
            if (lane == 0) part_a[brick - brick0] = w;
        }
        if (!meet()) return;
        if (warp == 0) {
            double s = 0.0;
            for (int k = lane; k < nb; k += 32) s += __ldcg(part_a + k);
            s = lane_sum(s);
            if (lane == 0) tot[0] = s;
        }
        __syncthreads();
        const double pap = tot[0];
        if (!(pap > 0.0)) {  // p.Kp <= 0 or NaN: breakdown
            status = PCG_BREAKDOWN;
            it += 1;
            break;
        }
        // ---- complete q of every own node, u, r, and the sums
        lrr = 0.0;
        lrz = 0.0;
        for (int l0 = t; l0 < nn; l0 += 3 * CH) {
            double x[3][3], y[3][3];
            uint2 o[3];
            unsigned m[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int l = l0 + k * CH;
                o[k] = make_uint2(NONE, NONE);
                m[k] = 0;
                if (l < nn) {
                    m[k] = mask[l];
                    if (!(m[k] & 16u)) o[k] = make_uint2(other[l], SM ? other[b.ncap + l] : NONE);
                    if (o[k].x != NONE) load_row_cg(rows + 4 * int64_t(o[k].x), x[k]);
                    if (o[k].y != NONE) load_row_cg(rows + 4 * int64_t(o[k].y), y[k]);
                }
            }
            const double alpha = rz / pap;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int l = l0 + k * CH;
                if (l >= nn) continue;
                const uint32_t own = uint32_t(base + l);
                double q[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) q[d] = qs[3 * l + d];
                if (m[k] & 16u) {
                    // all bricks' parts in ascending order
                    const uint32_t* ent = b.entry + int64_t(b.node[base + l]) * SHARE;
                    double v[3] = {0.0, 0.0, 0.0};
                    for (int j = 0; j < SHARE && ent[j] != NONE; ++j) {
                        double w[3] = {q[0], q[1], q[2]};
                        if (ent[j] != own) load_row_cg(rows + 4 * int64_t(ent[j]), w);
#pragma unroll
                        for (int d = 0; d < 3; ++d) v[d] += w[d];
                    }
#pragma unroll
                    for (int d = 0; d < 3; ++d) q[d] = v[d];
                } else if (o[k].y != NONE) {
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        q[d] = own > o[k].y ? (x[k][d] + y[k][d]) + q[d]
                                            : (q[d] + x[k][d]) + y[k][d];
                } else if (o[k].x != NONE) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) q[d] += x[k][d];
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    us[3 * l + d] += alpha * ps[3 * l + d];
                    // a constrained row of K is its diagonal, and p is zero there
                    const double r0 = rs[3 * l + d];
                    const double ri = (m[k] >> d) & 1u ? r0 : __fma_rn(-alpha, q[d], r0);
                    rs[3 * l + d] = ri;
                    if (m[k] & 8u) {
                        lrr += ri * ri;
                        lrz += ri * (ri * ds[3 * l + d]);
                    }
                }
            }
        }
        // ---- the CTAs meet: r.r and r.z
        double rz_new;
        if (!sums_b(lrr, lrz, rr, rz_new)) return;
        it += 1;
        if (!(rr > surely) && sqrt(rr) / bnorm <= tol) {
            status = PCG_CONVERGED;
        } else if (it >= max_iter) {
            status = PCG_MAXITER;
        } else if (rr <= rr_stop) {
            status = PCG_RELIABLE;  // rz stays r.z of the previous iterate
        } else {
            const double beta = rz_new / rz;
            rz = rz_new;
#pragma unroll 4
            for (int l = t; l < 3 * nn; l += CH)
                ps[l] = __fma_rn(beta, ps[l], rs[l] * ds[l]);
            __syncthreads();
        }
    }
    // the owner's copies are the solution (and the state of a later launch)
    for (int l = t; l < nn; l += CH) {
        if (!(mask[l] & 8u)) continue;
        const int64_t nd = b.node[base + l];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a.u[3 * nd + c] = us[3 * l + c];
            if constexpr (GRID) {
                a.r[3 * nd + c] = rs[3 * l + c];
                a.p[3 * nd + c] = ps[3 * l + c];
            }
        }
    }
    if (t == 0 && brick == brick0) {
        const double res = bnorm == 0.0 ? 0.0 : sqrt(rr) / bnorm;
        if constexpr (GRID) {
            a.s->it = it;
            a.s->res = res;
            a.s->rr = rr;
            a.s->rz = rz;
            __threadfence();
            if (status != PCG_RUNNING) a.s->status = status;
        } else {
            a.out_it[inst] = it;
            a.out_res[inst] = res;
            a.out_status[inst] = status;
        }
    }
}

// sm: the constants of `held` elements, `lists` chunk nodes' sums and all
// vectors in shared memory; otherwise a chunk's, two chunks' and p, q.
size_t brick_smem(int ncap, int held, int lists, bool sm) {
    size_t s = size_t(24) * FP * 8 + size_t(sm ? GEO * held : 10 * CH) * 8 +
               size_t(sm ? lists : CN) * 18 + size_t(sm ? 5 : 2) * 3 * ncap * 8 +
               size_t(ncap) * (sm ? 9 : 5);
    return (s + 15) & ~size_t(15);
}

}  // namespace

// The elements' constants, of the model as it is on the device: with the
// bricks, and again for the first solve after every further assembly.
void brick_constants(svx_ctx* ctx, svx_op* op) {
    BrickOperator& B = op->brick;
    geometry_kernel<<<B.bricks, CH, 0, ctx->stream>>>(B.view(), op->n_elem, op->conn.p, op->xyz.p,
                                                      op->youngs.p, op->poisson.p, B.geo.p);
    SVX_LAUNCH_CHECK();
    B.stale = false;
}

// Bricks of the members of op (one member: the whole model).  nbricks[m]:
// bricks of member m (0: none); set to 0 for a member with a brick whose
// nodes do not fit, a node shared by more bricks than the lists hold, or a
// node that no element uses.
void brick_build(svx_ctx* ctx, svx_op* op, bool single, const std::vector<int64_t>& node_off,
                 const std::vector<int64_t>& elem_off, std::vector<int>& nbricks) {
    BrickOperator& B = op->brick;
    cudaStream_t st = ctx->stream;
    const int members = int(nbricks.size());
    std::vector<int32_t> e0, e1, mb(1, 0), c0, bm, list;  // list: the members with bricks
    int chunks = 0, most = 0;
    for (int m = 0; m < members; ++m)
        if (nbricks[m])
            most = std::max<int>(most, int((elem_off[m + 1] - elem_off[m] + nbricks[m] - 1) /
                                           nbricks[m]));
    for (int m = 0; m < members; ++m) {
        const int64_t lo = elem_off[m], ne = elem_off[m + 1] - lo;
        for (int k = 0; k < nbricks[m]; ++k) {
            const int64_t a = lo + ne * k / nbricks[m], z = lo + ne * (k + 1) / nbricks[m];
            c0.push_back(chunks);
            chunks += int((z - a + CH - 1) / CH);
            e0.push_back(int32_t(a));
            e1.push_back(int32_t(z));
            bm.push_back(m);
        }
        if (nbricks[m]) list.push_back(m);
        mb.push_back(int32_t(c0.size()));
    }
    const int bricks = int(c0.size());
    if (bricks == 0 || most > BRICK_MAX_ELEMS) {
        std::fill(nbricks.begin(), nbricks.end(), 0);
        return;
    }
    // nodes a brick may have: what its shared memory holds
    const int held = (most + 31) / 32 * 32;
    auto lists_of = [&](int n) { return most <= CH ? (n + 7) & ~7 : 3 * held; };
    auto cap = [&](bool sm) {
        int n = 4095;
        while (n > 0 && brick_smem(n, held, lists_of(n), sm) > BRICK_SMEM) n -= 1;
        return n;
    };
    // a slab of `most` elements has about 2.3 nodes an element
    if (single && cap(true) < most * 23 / 10 + 32) {
        nbricks[0] = 0;
        return;
    }
    B.held = held;
    int ncap = std::min(cap(single), 8 * most);
    B.lists = single ? lists_of(ncap) : 1 << 30;
    B.ncap = ncap;
    B.bricks = bricks;
    // slots of the bricks' nodes: in a batch, a brick of few elements takes
    // few, whatever the largest takes; a single model's bricks are alike
    std::vector<uint32_t> n0(1, 0);
    for (int k = 0; k < bricks; ++k)
        n0.push_back(n0.back() + uint32_t(single ? ncap : std::min(ncap, 8 * (e1[k] - e0[k]))));
    B.slots = n0.back();
    DBuf<int64_t> d_noff, d_eoff;
    DBuf<uint16_t> layer;
    DBuf<int32_t> hist, ent_n, d_list, pos;
    DBuf<int> fail;
    const unsigned listed = unsigned(list.size());
    d_noff.alloc(ctx->pool, members + 1);
    d_eoff.alloc(ctx->pool, members + 1);
    layer.alloc(ctx->pool, size_t(op->n_elem));
    d_list.alloc(ctx->pool, listed);
    hist.alloc(ctx->pool, size_t(listed) * BRICK_LAYERS);
    if (single) pos.alloc(ctx->pool, size_t(op->n_elem));
    fail.alloc(ctx->pool, size_t(members) + 1);  // and the nodes many bricks share
    B.order.alloc(ctx->pool, size_t(op->n_elem));
    auto up = [&](auto& dst, const auto& src) {
        SVX_CUDA(cudaMemcpyAsync(dst.p, src.data(), src.size() * sizeof(src[0]),
                                 cudaMemcpyHostToDevice, st));
    };
    std::vector<int> bad(size_t(members) + 1);
    auto read_back = [&]() {
        SVX_CUDA(cudaMemcpyAsync(bad.data(), fail.p, sizeof(int) * bad.size(),
                                 cudaMemcpyDeviceToHost, st));
        SVX_CUDA(cudaStreamSynchronize(st));
    };
    up(d_noff, node_off);
    up(d_eoff, elem_off);
    up(d_list, list);
    SVX_CUDA(cudaMemsetAsync(hist.p, 0, sizeof(int32_t) * size_t(listed) * BRICK_LAYERS, st));
    SVX_CUDA(cudaMemsetAsync(fail.p, 0, sizeof(int) * bad.size(), st));
    layer_kernel<<<listed, 1024, 0, st>>>(d_list.p, d_noff.p, d_eoff.p, op->conn.p, op->xyz.p,
                                          layer.p, hist.p);
    SVX_LAUNCH_CHECK();
    layer_order_kernel<<<dim3(listed, single ? BRICK_LAYERS : 16), 256, 0, st>>>(
        d_list.p, d_eoff.p, layer.p, hist.p, B.order.p, pos.p);
    SVX_LAUNCH_CHECK();
    // A model whose layers take several bricks has nodes that four and more
    // bricks share; their sums go through the lists in global memory.  A 35^3
    // cube runs 27.0 us an iteration that way and 19.7 on its assembled K.  The
    // element order alone tells, so such a model is left before anything is built.
    if (single) {
        crowded_kernel<<<unsigned((op->n_nodes + 255) / 256), 256, 0, st>>>(
            op->n_nodes, op->n_elem, bricks, op->pat.slot_ptr.p, op->pat.slot_elem.p, pos.p,
            fail.p + members);
        SVX_LAUNCH_CHECK();
        read_back();
        if (bad[members] > op->n_nodes / 50) {
            nbricks[0] = 0;
            return;
        }
    }
    ent_n.alloc(ctx->pool, size_t(op->n_nodes));
    B.elem0.alloc(ctx->pool, bricks);
    B.elem1.alloc(ctx->pool, bricks);
    B.member.alloc(ctx->pool, bricks);
    B.chunk0.alloc(ctx->pool, bricks);
    B.member_brick.alloc(ctx->pool, members + 1);
    B.lconn.alloc(ctx->pool, size_t(op->n_elem) * 8);
    B.node0.alloc(ctx->pool, bricks + 1);
    B.node.alloc(ctx->pool, size_t(B.slots));
    B.count.alloc(ctx->pool, bricks);
    B.ref.alloc(ctx->pool, size_t(chunks) * CN * 8);
    B.cnode.alloc(ctx->pool, size_t(chunks) * CN);
    B.ccount.alloc(ctx->pool, chunks);
    B.entry.alloc(ctx->pool, size_t(op->n_nodes) * SHARE);
    B.geo.alloc(ctx->pool, size_t(op->n_elem) * GEO);
    up(B.elem0, e0);
    up(B.elem1, e1);
    up(B.member, bm);
    up(B.chunk0, c0);
    up(B.node0, n0);
    up(B.member_brick, mb);
    SVX_CUDA(cudaMemsetAsync(ent_n.p, 0, sizeof(int32_t) * size_t(op->n_nodes), st));
    const size_t bsm = size_t(SORT_BRICK + ncap) * 4;
    SVX_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(&brick_build_kernel),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int((SORT_BRICK + 4096) * 4)));
    brick_build_kernel<<<bricks, BT, bsm, st>>>(B.view(), op->conn.p, ent_n.p, fail.p);
    SVX_LAUNCH_CHECK();
    entry_sort_kernel<<<dim3(listed, single ? 256 : 16), 256, 0, st>>>(
        d_list.p, d_noff.p, B.entry.p, ent_n.p, fail.p);
    SVX_LAUNCH_CHECK();
    brick_constants(ctx, op);
    read_back();
    for (int m = 0; m < members; ++m)
        if (bad[m]) nbricks[m] = 0;
}

namespace {
BrickArgs brick_args(const svx_op* op, BrickWork& w) {
    BrickArgs a{};
    a.b = op->brick.view();
    a.n_elem = op->n_elem;
    a.geo = op->brick.geo.p;
    a.fixed = op->is_fixed.p;
    a.inv_diag = op->inv_diag.p;
    a.rows = w.exchange.p;
    a.part = w.part.p;
    a.rb = w.vec.p;
    if (w.vec.p) {
        const size_t n = size_t(op->brick.slots) * 3;
        a.ub = w.vec.p + n;
        a.db = w.vec.p + 2 * n;
    }
    return a;
}
}  // namespace

void BrickWork::alloc(svx_ctx* ctx, const svx_op* op, bool single) {
    const BrickOperator& B = op->brick;
    exchange.alloc(ctx->pool, size_t(B.slots) * 8);
    part.alloc(ctx->pool, size_t(B.bricks) * 3 + 4);
    if (!single) vec.alloc(ctx->pool, size_t(B.slots) * 9);
    gb.alloc(ctx->pool, 1);
}

// Up to `chunk` iterations of one model on the whole device, a cooperative
// launch of a CTA per brick.
void brick_grid_launch(svx_ctx* ctx, const svx_op* op, BrickWork& w, double* u, double* r,
                       double* p, PcgScalars* s, int chunk) {
    cudaStream_t st = ctx->stream;
    BrickArgs a = brick_args(op, w);
    a.u = u;
    a.r = r;
    a.p = p;
    a.s = s;
    a.gb = w.gb.p;
    a.chunk = chunk;
    auto* const kernel = &brick_pcg_kernel<true>;
    const void* fn = reinterpret_cast<const void*>(kernel);
    const size_t smem = brick_smem(op->brick.ncap, op->brick.held, op->brick.lists, true);
    SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(BRICK_SMEM)));
    SVX_CUDA(cudaMemsetAsync(w.gb.p, 0, sizeof(GridBarrier), st));
    void* args[] = {&a};
    SVX_CUDA(cudaLaunchCooperativeKernel(fn, dim3(unsigned(op->brick.bricks)),
                                         dim3(CH), args,
                                         smem, st));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

// `count` members (order: device list) of `ctas` bricks each, one cluster a
// member.
void brick_batch_launch(const svx_op* op, BrickWork& w, cudaStream_t st, int ctas, int count,
                        const int32_t* order, double* u, const double* tol,
                        const int64_t* max_iter, int64_t* out_it, double* out_res,
                        int32_t* out_status) {
    BrickArgs a = brick_args(op, w);
    a.f = op->f.p;
    a.u = u;
    a.order = order;
    a.member_brick = op->brick.member_brick.p;
    a.tol = tol;
    a.max_iter = max_iter;
    a.out_it = out_it;
    a.out_res = out_res;
    a.out_status = out_status;
    auto* const kernel = &brick_pcg_kernel<false>;
    const void* fn = reinterpret_cast<const void*>(kernel);
    SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(BRICK_SMEM)));
    SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(count) * unsigned(ctas));
    cfg.blockDim = dim3(CH);
    cfg.dynamicSmemBytes = brick_smem(op->brick.ncap, op->brick.held, 0, false);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SVX_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace svx
