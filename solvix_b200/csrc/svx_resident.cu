// svx_resident.cu - plane (two dofs a node) Jacobi-PCG with the whole system
// resident on the chip: one thread-block cluster per model, K in registers.
//
// What bounds it and why this split.  A plane model of the sizes this path
// sees (up to 8,191 nodes) is too small to fill HBM or L2 with work: its
// iteration is a chain of latencies (gathers, two reductions, the waits
// between blocks).  So everything an iteration touches is kept where it is
// used.  A thread owns one node: the node's 2 x 2 blocks over at most
// nine neighbours (36 doubles, 72 registers) are read once and stay in its
// registers, with its rows of r and p; a structured plate and its split
// triangles have at most nine neighbours, other meshes take the general
// kernels.  A cluster of up to 16 CTAs owns a model, each CTA a contiguous
// node range.  The search direction of every node that a CTA's rows reach
// (its window: own nodes plus the neighbouring ranges' edges) lies in its
// shared memory, so the SpMV gathers from shared memory only.
//
// Two exchanges an iteration, each the reduction's and the halo's at once:
// (A) p.Kp; (B) r.r, r.z and the new z = r / K_ii, which the owner sends
// into the windows of the CTAs that need it.  After B every CTA forms
// p = z + beta p over its whole window, the halo included, with the same
// fused multiply-add as the owner, so a node's p is bitwise the same
// everywhere and no third exchange is needed to publish it.  An exchange is
// a set of st.async stores that complete bytes on the receiver's mbarrier;
// nobody waits for more than the data itself (a cluster barrier with
// release and acquire costs 400-490 cycles here, 280 of them the fence).
// Reductions: a warp sums by two FP64 tensor-core products with a matrix of
// ones (74 cycles against 187 by shuffles), sends its partial to every CTA,
// and every warp sums all partials in the same order, so all threads of a
// cluster hold bitwise the same scalars and take the same branches.
//
// The recurrence, the stopping rule and the iteration count are those of
// the other FP64 forms (solver.rs:82-149) on the same assembled K; the
// shape (CTAs, threads) follows from the model's own size alone, so a
// model's result is the same alone and in any batch.

// Measured (one B200, us an iteration, against the grid-wide persistent
// kernel that these models took before): 55 nodes 0.67 (7.2), 231 nodes 0.87
// (6.8), 1,891 nodes 1.41 (6.7), the 200 x 20 cantilever 1.84 (6.5), 6,601
// nodes 2.43 (6.7).  256 plates of 10..160 x 4..40 as one batch: 14.7 ms of
// device time (140 ms with one CTA a member on the general kernel, whose
// largest members ran alone at the end).  The votes on the waits are 0.03 us of
// a cluster's iteration (flags in shared memory instead: the same within 2%).

#include "svx_internal.h"
#include "svx_quotient.h"
#include "svx_warp.h"

#include <cmath>
#include <cstddef>

namespace svx {

namespace {

constexpr int MAX_CTAS = 16;     // CTAs of a cluster
constexpr int MAX_THREADS = 512; // nodes of a CTA (128 registers a thread)
constexpr int MAX_WARPS = MAX_THREADS / 32;
constexpr int NEIGH = 9;         // neighbour blocks held in registers

struct ResidentArgs {
    const int32_t* order;      // members of this launch (nullptr: member = cluster)
    const int64_t* node_off;   // [members + 1] first node of each member
    const uint16_t* slot_node; // per member: slot -> node and node -> slot
    const uint16_t* node_slot; // (nullptr: slots are the nodes as numbered)
    const int64_t* adj_ptr;
    const int32_t* adj;
    const int64_t* node_base;
    const double* vals;
    const double* inv_diag;
    const double* f;
    double* u;
    const double* tol;         // per member
    const int64_t* max_iter;
    int64_t* out_it;
    double* out_res;
    int32_t* out_status;
    int window_cap;            // nodes a CTA's window may hold
    unsigned long long wait_ns;  // a wait between CTAs runs out after this long
    int fault;                 // DIAG: which exchange goes wrong, and how
};

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return unsigned(__cvta_generic_to_shared(p));
}
// the address of `local` (this CTA's shared memory) in CTA `rank`
__device__ __forceinline__ unsigned peer_addr(unsigned local, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_store(unsigned addr, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// stores to a peer that complete their bytes on the peer's mbarrier
__device__ __forceinline__ void send(unsigned addr, double v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(
                     addr), "d"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void send2(unsigned addr, double x, double y, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, "
                 "[%3];" ::"r"(addr), "d"(x), "d"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// Waits for the phase of the given parity; false when it has not completed
// within wait_ns.  The verdict is this thread's alone: the phase may complete
// between two threads' limits, so nobody acts on it before the CTA has voted.
constexpr unsigned long long WAIT_NS = 2000000000ull;
__device__ __forceinline__ bool bar_done(unsigned bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
__device__ __noinline__ bool bar_wait_long(unsigned bar, unsigned parity,
                                           unsigned long long wait_ns) {
    unsigned long long start, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(start));
    do {
        // polled after the clock is read: a thread that was switched out for
        // longer than the limit still looks once more
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        for (int k = 0; k < 64; ++k)
            if (bar_done(bar, parity)) return true;
    } while (now - start < wait_ns);
    return false;
}
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity,
                                         unsigned long long wait_ns) {
#pragma unroll 1
    for (int k = 0; k < 64; ++k)
        if (bar_done(bar, parity)) return true;
    return bar_wait_long(bar, parity, wait_ns);
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// What the CTAs of a cluster write into each other.
struct Inbox {
    double part_a[MAX_CTAS];             // p.Kp of each CTA
    double2 part_b[MAX_CTAS];            // r.r and r.z of each CTA
    unsigned long long bar_a, bar_b;     // mbarriers of the two exchanges
    int win_lo[MAX_CTAS], win_hi[MAX_CTAS];
};

// SINGLE: one CTA owns the model (the exchanges are stores to its own shared
// memory and block barriers).
// T: most threads of a CTA.  512 leaves a thread 128 registers, so a batch
// also runs two CTAs of 256 on an SM; a single solve's CTAs of up to 256
// threads have their SM to themselves and take all the registers they want.
// DIAG: an early iteration's exchange a.fault & 1 (0: A, 1: B) goes wrong in
// CTA 1, which drops its sums (a.fault < 2) or takes the wait of every third
// thread to have run out (2, 3).
template <bool SINGLE, int T, bool DIAG = false>
__global__ void __launch_bounds__(T, 1) resident_pcg_kernel(ResidentArgs a) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ __align__(16) Inbox box;
    __shared__ double warp_a[MAX_WARPS], warp_b[2 * MAX_WARPS];
    __shared__ int red_lo, red_hi;
    unsigned rank = 0, ctas = 1;
    if constexpr (!SINGLE) {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
    }
    const int member_slot = int(blockIdx.x / ctas);
    const int inst = a.order ? a.order[member_slot] : member_slot;
    const int64_t N0 = a.node_off[inst];
    const int n = int(a.node_off[inst + 1] - N0);
    // this CTA's nodes [n0, n1) within the member
    const int n0 = int(int64_t(n) * rank / ctas), n1 = int(int64_t(n) * (rank + 1) / ctas);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, warps = blockDim.x >> 5;
    // the member's nodes are dealt out in slots, ordered along its longest
    // side (or as numbered): a range of slots has short edges to its
    // neighbours
    const int i = n0 + t;  // this thread's slot
    const bool mine = i < n1;
    const int node = !mine ? 0 : a.slot_node ? int(a.slot_node[N0 + i]) : i;
    double2* pw = reinterpret_cast<double2*>(dyn);      // p over the window
    double2* zw = pw + a.window_cap;                    // z over the halo
    double2* us = zw + (SINGLE ? 0 : a.window_cap);     // u of the own nodes
    double2* ds = us + blockDim.x;                      // 1 / K_ii of the own nodes
    const unsigned bar_a = smem_addr(&box.bar_a), bar_b = smem_addr(&box.bar_b);

    // ---- the node's blocks and neighbours, once
    double k[NEIGH][4];
    int nb[NEIGH];
    int lo = i, hi = i;
#pragma unroll
    for (int j = 0; j < NEIGH; ++j) {
        k[j][0] = k[j][1] = k[j][2] = k[j][3] = 0.0;
        nb[j] = i;
    }
    double2 r = make_double2(0.0, 0.0);
    if (mine) {
        const int64_t a0 = a.adj_ptr[N0 + node];
        const int d = int(a.adj_ptr[N0 + node + 1] - a0);
        const double* v = a.vals + a.node_base[N0 + node];
        if (d == 0) {  // a node no element uses: rows of length 1
            k[0][0] = v[0];
            k[0][3] = v[1];
        }
#pragma unroll
        for (int j = 0; j < NEIGH; ++j)
            if (j < d) {
                nb[j] = a.node_slot ? int(a.node_slot[a.adj[a0 + j]]) : int(a.adj[a0 + j] - N0);
                lo = min(lo, nb[j]);
                hi = max(hi, nb[j]);
                k[j][0] = v[2 * j];
                k[j][1] = v[2 * j + 1];
                k[j][2] = v[2 * d + 2 * j];
                k[j][3] = v[2 * d + 2 * j + 1];
            }
        const int64_t row = (N0 + node) * 2;
        r = make_double2(a.f[row], a.f[row + 1]);
        ds[t] = make_double2(a.inv_diag[row], a.inv_diag[row + 1]);
        us[t] = make_double2(0.0, 0.0);
    }
    // ---- the CTA's window, published to every CTA of the cluster
    int wlo = 0, whi = n - 1;
    unsigned needed = 0;  // CTAs whose window holds this node, own excepted
    if constexpr (!SINGLE) {
        if (t == 0) {
            red_lo = n0;
            red_hi = n1 - 1;
            bar_init(bar_a);
            bar_init(bar_b);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (mine) {
            atomicMin(&red_lo, lo);
            atomicMax(&red_hi, hi);
        }
        cluster_barrier();  // every CTA of the cluster runs; red_* are final
        wlo = red_lo;
        whi = red_hi;
        if (t < int(ctas)) {
            peer_store(peer_addr(smem_addr(&box.win_lo[rank]), unsigned(t)), wlo);
            peer_store(peer_addr(smem_addr(&box.win_hi[rank]), unsigned(t)), whi);
        }
        cluster_barrier();
        if (mine)
            for (unsigned c = 0; c < ctas; ++c)
                if (c != rank && i >= box.win_lo[c] && i <= box.win_hi[c]) needed |= 1u << c;
    }
    // window offsets of the neighbours, two to a register
    unsigned nbp[(NEIGH + 1) / 2];
#pragma unroll
    for (int j = 0; j < NEIGH; j += 2) {
        const unsigned x = mine ? unsigned(nb[j] - wlo) : 0u;
        const unsigned y = (mine && j + 1 < NEIGH) ? unsigned(nb[j + 1 < NEIGH ? j + 1 : j] - wlo)
                                                   : 0u;
        nbp[j / 2] = x | (y << 16);
    }
    const int own = mine ? i - wlo : 0;       // this node's place in the window
    const int below = n0 - wlo;               // halo nodes before the own range
    const int halo = below + (whi - n1 + 1);  // all halo nodes
    for (int h = t; h < halo; h += int(blockDim.x))
        pw[h < below ? h : h - below + (n1 - wlo)] = make_double2(0.0, 0.0);
    // the CTA that a lane of warp 0 sends the CTA's sums to
    const bool sends = !SINGLE && lane < int(ctas);
    const unsigned peer_box = sends ? peer_addr(smem_addr(&box), unsigned(lane)) : 0u;
    const unsigned bytes_a = ctas * 8, bytes_b = (ctas + unsigned(halo)) * 16;
    // sends z into the windows that hold this node
    auto push = [&](const double2& z) {
        if constexpr (!SINGLE) {
            unsigned m = needed;
            while (m) {
                const unsigned c = unsigned(__ffs(int(m))) - 1;
                m &= m - 1;
                send2(peer_addr(smem_addr(zw + (i - box.win_lo[c])), c), z.x, z.y,
                      peer_addr(bar_b, c));
            }
        }
    };
    // p.Kp of the model from the threads' terms: warp sums, their sum in
    // warp 0, one message to every CTA (an exchange costs about 7 cycles for
    // every message a CTA receives), and their sum in every warp
    auto faulty = [&](unsigned parity, int fault) {
        return DIAG && parity == 1u && rank == 1u && a.fault == fault;
    };
    auto reduce_a = [&](double x, unsigned parity, double& total) -> bool {
        x = lane_sum(x);
        if (lane == 0) warp_a[warp] = x;
        __syncthreads();
        if constexpr (SINGLE) {
            total = lane_sum(lane < warps ? warp_a[lane] : 0.0);
            return true;
        } else {
            if (warp == 0) {
                x = lane_sum(lane < warps ? warp_a[lane] : 0.0);
                if (sends && !faulty(parity, 0))
                    send(peer_box + unsigned(offsetof(Inbox, part_a)) + rank * 8, x,
                         peer_box + unsigned(offsetof(Inbox, bar_a)));
            }
            const bool ok = bar_wait(bar_a, parity, a.wait_ns);
            __syncwarp();
            total = lane_sum(lane < int(ctas) ? box.part_a[lane] : 0.0);
            return ok && !(faulty(parity, 2) && t % 3 == 0);
        }
    };
    // r.r and r.z of the model, and the vote on the wait before (ok): the CTA
    // sends its sums, which let the others go on, only if all of its threads
    // came through.  Returns what ends the solve here, the same in every
    // thread: a wait that ran out, or p.Kp <= 0 (broke; all threads have the
    // same p.Kp when none of their waits ran out).
    auto reduce_b = [&](double x, double y, bool& ok, bool broke, unsigned parity, double& tx,
                        double& ty) -> int {
        double v = lane_sum_pair(x, y, lane);
        if ((lane & 15) == 0) warp_b[2 * warp + (lane >> 4)] = v;
        if constexpr (SINGLE) __syncthreads();
        else if (__syncthreads_or(!ok)) return RESIDENT_STALLED;
        if (broke) return PCG_BREAKDOWN;
        double2 w = make_double2(0.0, 0.0);
        if (SINGLE || warp == 0) {
            if (lane < warps) w = make_double2(warp_b[2 * lane], warp_b[2 * lane + 1]);
        }
        if constexpr (!SINGLE) {
            if (warp == 0) {
                v = lane_sum_pair(w.x, w.y, lane);
                const double other = __shfl_xor_sync(0xffffffffu, v, 16);
                if (sends && !faulty(parity, 1))
                    send2(peer_box + unsigned(offsetof(Inbox, part_b)) + rank * 16, v, other,
                          peer_box + unsigned(offsetof(Inbox, bar_b)));
            }
            ok = bar_wait(bar_b, parity, a.wait_ns) && !(faulty(parity, 3) && t % 3 == 0);
            __syncwarp();
            w = lane < int(ctas) ? box.part_b[lane] : make_double2(0.0, 0.0);
        }
        tx = lane_sum(w.x);
        ty = lane_sum(w.y);
        return PCG_RUNNING;
    };
    const double tl = a.tol[inst];
    const int mi = int(a.max_iter[inst]);  // at most RESIDENT_MAX_ITER
    double2 z = make_double2(0.0, 0.0), p = make_double2(0.0, 0.0);
    double lrr = 0.0, lrz = 0.0;
    if (!SINGLE && t == 0) bar_expect(bar_b, bytes_b);
    if (mine) {
        const double2 d = ds[t];
        z = make_double2(r.x * d.x, r.y * d.y);
        lrr = r.x * r.x + r.y * r.y;
        lrz = r.x * z.x + r.y * z.y;
        push(z);
    }
    double rr, rz;
    bool ok = true;  // this thread's last wait
    reduce_b(lrr, lrz, ok, false, 0, rr, rz);
    const double bnorm = sqrt(rr);
    // above this r.r, sqrt(r.r) / ||f|| cannot round to tol or less, so the
    // root and the quotient are left to the last iterations
    double surely = (tl * bnorm) * (tl * bnorm) * (1.0 + 1e-12);
    if (surely < 1e-280) surely = INFINITY;  // the square left the normal range
    int it = 0;
    int status = (bnorm == 0.0) ? PCG_CONVERGED : PCG_RUNNING;
    double beta = 0.0;
    for (;;) {
        if (SINGLE && status != PCG_RUNNING) break;
        // (a thread whose wait ran out has seen no phase end, so it must not
        // open the next one)
        if (!SINGLE && t == 0 && ok) {
            bar_expect(bar_a, bytes_a);
            bar_expect(bar_b, bytes_b);
        }
        // p = z + beta p over the window
        if (mine) {
            p = make_double2(__fma_rn(beta, p.x, z.x), __fma_rn(beta, p.y, z.y));
            pw[own] = p;
        }
        if constexpr (!SINGLE)
            for (int h = t; h < halo; h += int(blockDim.x)) {
                const int w = h < below ? h : h - below + (n1 - wlo);
                const double2 zz = zw[w], pp = pw[w];
                pw[w] = make_double2(__fma_rn(beta, pp.x, zz.x), __fma_rn(beta, pp.y, zz.y));
            }
        if constexpr (SINGLE) {
            __syncthreads();
        } else {
            // the vote on exchange B's wait; its outcome stands only now (the
            // one p too many at the end costs less than a barrier of its own)
            if (__syncthreads_or(!ok)) status = RESIDENT_STALLED;
            if (status != PCG_RUNNING) break;
        }
        // q = K p on the own rows, p.q
        // (two chains a row, over the first five and the last four neighbours:
        // half the latency of one.  Every order of the sum is as near the
        // 64-bit solution; of one, two and four chains this one also stays
        // nearest to the row sums of K that a comparison on a strip of 130 x 4
        // triangles sees: 8e-11 off, against 1.5e-10 to 2.1e-10)
        double2 qc[2] = {};
#pragma unroll
        for (int j = 0; j < NEIGH; ++j) {
            const unsigned o = (j & 1) ? (nbp[j / 2] >> 16) : (nbp[j / 2] & 0xffffu);
            const double2 x = pw[o];
            double2& c = qc[j < 5 ? 0 : 1];
            c.x = __fma_rn(k[j][1], x.y, __fma_rn(k[j][0], x.x, c.x));
            c.y = __fma_rn(k[j][3], x.y, __fma_rn(k[j][2], x.x, c.y));
        }
        const double2 q = make_double2(qc[0].x + qc[1].x, qc[0].y + qc[1].y);
        const double rz_inv = 1.0 / rz;  // for beta, off the chain of the sums
        double pap;
        ok = reduce_a(p.x * q.x + p.y * q.y, unsigned(it) & 1u, pap);
        it += 1;
        const bool broke = !(pap > 0.0);  // p.Kp <= 0 or NaN: breakdown
        const double alpha = rz / pap;
        lrr = 0.0;
        lrz = 0.0;
        if (mine && ok && !broke) {
            r.x -= alpha * q.x;
            r.y -= alpha * q.y;
            const double2 d = ds[t];
            z = make_double2(r.x * d.x, r.y * d.y);
            lrr = r.x * r.x + r.y * r.y;
            lrz = r.x * z.x + r.y * z.y;
            push(z);
            double2 u = us[t];
            u.x += alpha * p.x;
            u.y += alpha * p.y;
            us[t] = u;
        }
        double rz_new;
        status = reduce_b(lrr, lrz, ok, broke, unsigned(it) & 1u, rr, rz_new);
        if (status != PCG_RUNNING) break;
        if (!(rr > surely) && sqrt(rr) / bnorm <= tl) {
            status = PCG_CONVERGED;
        } else if (it >= mi) {
            status = PCG_MAXITER;
        } else {
            beta = quotient(rz_new, rz, rz_inv);
            rz = rz_new;
        }
    }
    // A wait ran out in this CTA.  It has sent nothing since, so the waits of
    // the others run out in turn, and none leaves while another may still
    // store into it.  (Others may have ended the solve on the exchange that
    // came too late here; then the fields are final here too, and they do not
    // wait for this CTA.)
    if (!SINGLE && status == RESIDENT_STALLED) cluster_barrier();
    // no CTA's shared memory is written after the last exchange, so the CTAs
    // of a cluster may leave at different times
    if (mine) reinterpret_cast<double2*>(a.u)[N0 + node] = us[t];
    if (rank == 0 && t == 0) {
        a.out_it[inst] = it;
        a.out_res[inst] = bnorm == 0.0 ? 0.0 : sqrt(rr) / bnorm;
        a.out_status[inst] = status;
    }
}

// The slots of a member of more than one CTA: its nodes sorted along the
// longer side of their bounding box, by number where that is equal; and the
// largest slot difference over the node pairs of K, which bounds a CTA's
// window.  One CTA a member, a bitonic sort of up to 8,192 keys in shared
// memory.  Any order is correct; this one cuts the halo of a 200 x 20 mesh
// numbered along its length from 400 to 44 nodes a CTA of 264.
constexpr int ORDER_THREADS = 1024;
__global__ void __launch_bounds__(ORDER_THREADS)
slot_order_kernel(const int64_t* __restrict__ node_off, const double* __restrict__ xyz,
                  const int64_t* __restrict__ adj_ptr, const int32_t* __restrict__ adj,
                  int min_nodes, uint16_t* slot_node, uint16_t* node_slot,
                  int64_t* __restrict__ span) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long* key = reinterpret_cast<unsigned long long*>(dyn);
    __shared__ double box[4][ORDER_THREADS / 32];
    __shared__ int top;
    const int64_t N0 = node_off[blockIdx.x];
    const int64_t size = node_off[blockIdx.x + 1] - N0;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (size <= min_nodes || size >= RESIDENT_MAX_NODES) return;
    const int n = int(size);
    double b[4] = {INFINITY, INFINITY, INFINITY, INFINITY};  // min x, min y, min -x, min -y
    for (int i = t; i < n; i += ORDER_THREADS) {
        const double x = xyz[3 * (N0 + i)], y = xyz[3 * (N0 + i) + 1];
        b[0] = fmin(b[0], x);
        b[1] = fmin(b[1], y);
        b[2] = fmin(b[2], -x);
        b[3] = fmin(b[3], -y);
    }
    for (int c = 0; c < 4; ++c) {
        for (int off = 16; off > 0; off >>= 1)
            b[c] = fmin(b[c], __shfl_xor_sync(0xffffffffu, b[c], off));
        if (lane == 0) box[c][warp] = b[c];
    }
    if (t == 0) top = 0;
    __syncthreads();
    for (int c = 0; c < 4; ++c)
        for (int w = 0; w < ORDER_THREADS / 32; ++w) b[c] = fmin(b[c], box[c][w]);
    const double ex = -b[2] - b[0], ey = -b[3] - b[1];
    const int axis = ex >= ey ? 0 : 1;
    const double lo = b[axis], scale = 4294967295.0 / (axis == 0 ? ex : ey);
    int m = 1;
    while (m < n) m *= 2;
    for (int i = t; i < m; i += ORDER_THREADS) {
        unsigned long long k = ~0ull;
        if (i < n) {
            // 32 bits of the coordinate (0 where it is not a number)
            double q = (xyz[3 * (N0 + i) + axis] - lo) * scale;
            q = q > 0.0 ? fmin(q, 4294967295.0) : 0.0;
            k = ((unsigned long long)(unsigned)q << 13) | (unsigned)i;
        }
        key[i] = k;
    }
    __syncthreads();
    for (int k = 2; k <= m; k *= 2)
        for (int j = k / 2; j > 0; j /= 2) {
            for (int q = t; q < m / 2; q += ORDER_THREADS) {
                const int i = 2 * q - (q & (j - 1)), p = i + j;
                const unsigned long long x = key[i], y = key[p];
                if ((x > y) == ((i & k) == 0)) {
                    key[i] = y;
                    key[p] = x;
                }
            }
            __syncthreads();
        }
    for (int i = t; i < n; i += ORDER_THREADS) {
        const int node = int(key[i] & 8191u);
        slot_node[N0 + i] = uint16_t(node);
        node_slot[N0 + node] = uint16_t(i);
    }
    __syncthreads();
    int s = 0;
    for (int i = t; i < n; i += ORDER_THREADS) {
        const int mine = node_slot[N0 + i];
        for (int64_t q = adj_ptr[N0 + i]; q < adj_ptr[N0 + i + 1]; ++q)
            s = max(s, abs(int(node_slot[adj[q]]) - mine));
    }
    atomicMax(&top, s);
    __syncthreads();
    if (t == 0) span[blockIdx.x] = top;
}

}  // namespace

// Nodes that one CTA takes before a model is split over a cluster.  A second
// CTA costs a single solve two exchanges an iteration (0.55 us): 231 nodes
// run 0.92 us an iteration on one CTA and 1.27 on two to four; above 256
// nodes the shorter gathers pay for it (861 nodes: 1.30 us on seven CTAs).
static int one_cta_nodes(const svx_ctx* ctx, bool single) {
    return single ? std::max(256, ctx->resident_nodes_single) : ctx->resident_nodes_batch;
}

// Slots of the members of op that take more than one CTA; span[k] becomes
// the member's largest slot difference (unchanged for the others).
void resident_order(svx_ctx* ctx, svx_op* op, bool single, const std::vector<int64_t>& node_off,
                    std::vector<int64_t>& span) {
    const int count = int(node_off.size()) - 1;
    const int target = one_cta_nodes(ctx, single);
    int64_t top = 0;
    for (int k = 0; k < count; ++k) {
        const int64_t n = node_off[k + 1] - node_off[k];
        if (n > target && n < RESIDENT_MAX_NODES) top = std::max(top, n);
    }
    if (top == 0) return;
    cudaStream_t st = ctx->stream;
    op->slot_node.alloc(ctx->pool, size_t(op->n_nodes) + 1);
    op->node_slot.alloc(ctx->pool, size_t(op->n_nodes) + 1);
    DBuf<int64_t> off, out;
    off.alloc(ctx->pool, count + 1);
    out.alloc(ctx->pool, count + 1);
    size_t m = 1;
    while (int64_t(m) < top) m *= 2;
    const void* fn = reinterpret_cast<const void*>(&slot_order_kernel);
    SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(RESIDENT_MAX_NODES * sizeof(unsigned long long))));
    SVX_CUDA(cudaMemcpyAsync(off.p, node_off.data(), (count + 1) * sizeof(int64_t),
                             cudaMemcpyHostToDevice, st));
    SVX_CUDA(cudaMemcpyAsync(out.p, span.data(), count * sizeof(int64_t), cudaMemcpyHostToDevice,
                             st));
    slot_order_kernel<<<count, ORDER_THREADS, m * sizeof(unsigned long long), st>>>(
        off.p, op->xyz.p, op->pat.adj_ptr.p, op->pat.adj.p, target, op->slot_node.p,
        op->node_slot.p, out.p);
    SVX_LAUNCH_CHECK();
    SVX_CUDA(cudaMemcpyAsync(span.data(), out.p, count * sizeof(int64_t), cudaMemcpyDeviceToHost,
                             st));
    SVX_CUDA(cudaStreamSynchronize(st));
}

// The cluster shape of a plane model of n nodes whose elements span at most
// `span` slots; false when the model takes the general kernels.
bool resident_shape(const svx_ctx* ctx, int64_t n, int64_t span, bool single,
                    ResidentShape* out) {
    if (n <= 0 || n >= RESIDENT_MAX_NODES || !ctx->resident) return false;
    const int target = single ? ctx->resident_nodes_single : ctx->resident_nodes_batch;
    int ctas = 1, threads = 64;
    if (n <= one_cta_nodes(ctx, single)) {
        while (threads < n) threads = threads < 256 ? threads * 2 : threads + 128;
    } else {
        static const int sizes[] = {2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16};
        threads = n <= int64_t(MAX_CTAS) * target ? target : MAX_THREADS;
        if (single && threads > target) threads = int((n + MAX_CTAS - 1) / MAX_CTAS);
        for (int c : sizes) {
            ctas = c;
            if (int64_t(c) * threads >= n) break;
        }
    }
    const int per = int((n + ctas - 1) / ctas);
    if (single) threads = (per + 31) / 32 * 32;
    if (threads > MAX_THREADS || per > threads) return false;
    const int64_t window = std::min<int64_t>(n, per + 2 * span);
    const size_t smem = size_t((ctas > 1 ? 2 : 1) * window + 2 * threads) * sizeof(double2);
    if (smem > RESIDENT_SMEM) return false;
    out->ctas = ctas;
    out->threads = threads;
    out->window = int(window);
    out->smem = smem;
    return true;
}

void resident_pcg(svx_ctx* ctx, const svx_op* op, const ResidentShape& shape, bool single, cudaStream_t st,
                  int count, const int32_t* order, const int64_t* node_off, const double* tol,
                  const int64_t* max_iter, int64_t* out_it, double* out_res,
                  int32_t* out_status, double* u, int fault, long long wait_ns) {
    // a single solve takes the registers its thread count leaves free; a
    // batch's CTAs of up to 256 threads share an SM at 128 registers
    const int top = shape.threads <= 256 ? (single ? 256 : MAX_THREADS)
                    : shape.threads <= 384 ? 384 : MAX_THREADS;
    auto* kernel =
        shape.ctas > 1
            ? (top == 256 ? &resident_pcg_kernel<false, 256>
               : top == 384 ? &resident_pcg_kernel<false, 384>
                            : &resident_pcg_kernel<false, MAX_THREADS>)
            : (top == 256 ? &resident_pcg_kernel<true, 256>
               : top == 384 ? &resident_pcg_kernel<true, 384>
                            : &resident_pcg_kernel<true, MAX_THREADS>);
    ResidentArgs a;
    a.order = order;
    a.node_off = node_off;
    a.slot_node = shape.ctas > 1 ? op->slot_node.p : nullptr;
    a.node_slot = shape.ctas > 1 ? op->node_slot.p : nullptr;
    a.adj_ptr = op->pat.adj_ptr.p;
    a.adj = op->pat.adj.p;
    a.node_base = op->pat.node_base.p;
    a.vals = op->vals.p;
    a.inv_diag = op->inv_diag.p;
    a.f = op->f.p;
    a.u = u;
    a.tol = tol;
    a.max_iter = max_iter;
    a.out_it = out_it;
    a.out_res = out_res;
    a.out_status = out_status;
    a.window_cap = shape.window;
    a.wait_ns = fault < 0 ? WAIT_NS : wait_ns;
    a.fault = fault;
    if (fault >= 0) kernel = &resident_pcg_kernel<false, MAX_THREADS, true>;
    const void* fn = reinterpret_cast<const void*>(kernel);
    SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(RESIDENT_SMEM)));
    SVX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(shape.ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(count) * unsigned(shape.ctas));
    cfg.blockDim = dim3(unsigned(shape.threads));
    cfg.dynamicSmemBytes = shape.smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SVX_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace svx
