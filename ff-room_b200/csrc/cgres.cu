// cgres.cu — the reference's unpreconditioned CG with its vectors on chip (sm_100a).
//
// The same solve as k_cg (projection.cu; PoissonSolver::solve, cpp/src/core/
// PoissonSolver.cpp:93-158) for rooms of at most one cell per thread of
// k_cg's grid.  Such a room is bound by latency: an iteration moves a few
// hundred kilobytes and waits twice for every block.  So here
//   - each block owns the same cells for the whole solve; x, r, A d and the
//     stencil row stay in registers, the direction in shared memory together
//     with that of the neighbour cells (its halo);
//   - the halo direction is advanced redundantly, d = r + beta d, so only r
//     crosses blocks, once per iteration, and no barrier but the two
//     reductions is left;
//   - every block adds all partials itself, so nobody waits for a last
//     arriver's broadcast.
// Two forms.  k_cg_cluster: one thread-block cluster of up to 16 blocks, each
// with a run of consecutive cells; r's halo (bulk copies) and the partials
// (st.async) are pushed into the readers' shared memory and counted by an
// mbarrier there.  k_cg_chunks: a cooperative grid; both travel through L2 as
// 8-byte words that carry half a double and a number, so a reader that sees
// the number has the value, and no counter and no fence stands between.
//
// Every sum is formed in k_cg's order (the 256 cells of a partial as its
// blocks add them, the partials as its last arriver adds them), so the
// results are bit-identical to k_cg's.
#include "forms.h"
#include "projection.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace ffr {

// A double as two 8-byte words {number, half} side by side; each word is
// written and read whole.
__device__ __forceinline__ void tagged_store(unsigned long long *at, double v, unsigned tag)
{
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(at), "l"(t | (unsigned)__double2loint(v)),
                 "l"(t | (unsigned)__double2hiint(v))
                 : "memory");
}

__device__ __forceinline__ bool tagged_load(const unsigned long long *at, unsigned tag, double &v)
{
    unsigned long long a, b;
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(at) : "memory");
    v = __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
    return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

// block_sum's combination of eight warp sums (its shuffle tree over lanes 0..7).
__device__ __forceinline__ double tree8(const double (&s)[8])
{
    return ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
}

// block_sum's total of 256 values, by one warp: eight groups of 32 at a
// stride of kPadded.  Four lanes take a group, each every fourth value, so
// the first three steps of its shuffle tree are sums in registers.
__device__ __forceinline__ double sum256(const double *s)
{
    const int lane = threadIdx.x & 31;
    const double *g = s + (lane >> 2) * kPadded + (lane & 3);
    double v[8];
#pragma unroll
    for (int m = 0; m < 8; m++) v[m] = g[4 * m];
    double t = tree8(v);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 16);
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    return t;
}

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned peer_addr(unsigned local, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}

// Stores v into a block's shared memory and counts its 8 bytes on that block's mbarrier.
__device__ __forceinline__ void push(unsigned dst, double v, unsigned bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void bar_expect(unsigned bar, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n.reg .pred p;\n"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}

// The bound of a wait: true once the wait limit has passed (looked at every
// 64 tries) or, in a grid, another block has given up.
struct WaitLimit {
    unsigned spins = 0;
    unsigned long long t0 = 0;
    __device__ __forceinline__ bool over(int *err, unsigned long long at_least = 0)
    {
        if ((++spins & 63u) != 0) return false;
        const unsigned long long now = global_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 <= max(g_wait_limit_ns, at_least) && !(err && *(volatile int *)err)) return false;
        if (err) atomicExch(err, 1);
        return true;
    }
};

__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, unsigned long long at_least = 0)
{
    WaitLimit w;
    while (!bar_try(bar, parity))
        if (w.over(nullptr, at_least)) return false;
    return true;
}

// The stencil row of cell c and its right-hand side.
struct ResRow {
    unsigned code;
    double rhs, diag, w[6];     // w: scale of a neighbour that is an unknown, else 0
    __device__ __forceinline__ ResRow(const CGArgs &A, int c)
    {
        const RoomDev &R = A.R;
        const int nx = R.nx, ny = R.ny, nz = R.nz, plane = ny * nz;
        code = c < R.n ? R.sc[c] : SC_SOLID;
        rhs = 0.0;
        diag = 1.0;
#pragma unroll
        for (int a = 0; a < 6; a++) w[a] = 0.0;
        if (code & SC_SOLID) return;
        int i, j, k;
        decode(c, ny, nz, i, j, k);
        if (A.from_faces) {
            const int v0 = (i * (ny + 1) + j) * nz + k, w0 = (i * ny + j) * (nz + 1) + k;
            const double div = (A.us[c + plane] - A.us[c]) / R.dxv[i] + (A.vs[v0 + nz] - A.vs[v0]) / R.dyv[j] +
                               (A.ws[w0 + 1] - A.ws[w0]) / R.dzv[k];
            rhs = A.rhs_factor * div;
        } else {
            rhs = A.rhs[c];
        }
        const int at[6] = {i, nx + i, 2 * nx + j, 2 * nx + ny + j, 2 * (nx + ny) + k, 2 * (nx + ny) + nz + k};
        double dg = 0.0;
#pragma unroll
        for (int a = 0; a < 6; a++) {
            // the reference's order (PoissonSolver.cpp:61-77)
            const unsigned cls = (code >> (2 * a)) & 3u;
            const double s = R.scale[at[a]];
            if (cls == SC_IN) dg += s;
            else if (cls == SC_DIR) dg += 2.0 * s;
            w[a] = cls == SC_IN ? s : 0.0;
        }
        diag = dg < 1e-30 ? 1.0 : dg;
    }
};

// Above this ||r||^2 the stopping test sqrt(||r||^2) / bnorm < tol fails
// whatever its roundings, so the square root and the division wait until
// the solve is near its end.
__device__ __forceinline__ double not_converged_above(double tol, double bnorm)
{
    const double t = tol * bnorm;
    return 1.000001 * t * t;
}

__device__ __forceinline__ void res_results(const CGArgs &A, double res, int iters, int flags)
{
    if (A.out_res) *A.out_res = res;
    if (A.out_iters) *A.out_iters = iters;
    if (A.out_flags) *A.out_flags = flags;
    if (A.st) {
        A.st->pres = res;
        A.st->iters = iters;
        atomicOr(&A.st->flags, flags);
    }
}

// --------------------------------------------------------- one cluster

// Pushes r of a block's `own` cells (in sr) to the blocks whose halo (srh) holds
// it and counts it on their mbarrier bars[2].  By the last warp.
__device__ __forceinline__ void push_halo(int own, int plane2, const double *sr, const double *srh,
                                          const unsigned long long *bars)
{
    const int lane = threadIdx.x & 31, rank = blockIdx.x, base = rank * own;
    if ((threadIdx.x >> 5) != kResThreads / 32 - 1 || lane >= (int)gridDim.x || lane == rank) return;
    // own cells [lo, hi) that lie in block `lane`'s halo, before or after its cells
    const int b0 = lane * own, b1 = b0 + own;
    const int lo = lane > rank ? max(base, b0 - plane2) : base;
    const int hi = lane > rank ? base + own : min(base + own, b1 + plane2);
    if (lo >= hi) return;
    const int at = lane > rank ? lo - (b0 - plane2) : plane2 + lo - b1;
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     peer_addr(smem_addr(srh + at), lane)),
                 "r"(smem_addr(sr + lo - base)), "r"(8 * (hi - lo)), "r"(peer_addr(smem_addr(bars + 2), lane))
                 : "memory");
}

// After a block of the cluster has given up: waits until every copy between the
// blocks has arrived; true when they have.  A reduction ends once every block
// has pushed, so all blocks are at the last one that any of them began (`seq`
// counts them, `halos` the halos waited for) or the one before it.  Those
// before it push what the others expect (the values no longer matter); then
// all that was pushed is certain to arrive, and each block waits for what is
// addressed to it.  Not inlined: inside the kernel it cost the four-cell form
// 0.8 % (registers of the loop), as a function nothing.
__device__ __noinline__ bool await_copies(int own, int plane2, int halo_bytes, unsigned seq, int halos, const double *sr,
                                          const double *srh, double *parts, unsigned long long *bars, unsigned &s_seq)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, rank = blockIdx.x, blocks = gridDim.x;
    const int V = own / kResGroup;
    auto arrived = [&](unsigned q) {      // reduction q's partials
        return bar_wait(smem_addr(bars + (q & 1)), ((q - 1) >> 1) & 1u, kBarrierTimeoutNs);
    };
    auto halo_arrived = [&](int h) { return bar_wait(smem_addr(bars + 2), (unsigned)h & 1u, kBarrierTimeoutNs); };
    cooperative_groups::this_cluster().sync();
    unsigned last = seq;
    for (int b = 0; b < blocks; b++) {
        unsigned v;
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_addr(smem_addr(&s_seq), b)) : "memory");
        last = max(last, v);
    }
    bool ok = seq == 0 || arrived(seq);
    if (halos > 0) ok = halo_arrived(halos - 1) && ok;
    __syncthreads();
    if (last > seq) {
        if (last & 1) push_halo(own, plane2, sr, srh, bars);
        if (t == 0) bar_expect(smem_addr(bars + (last & 1)), 8 * V * blocks);
        if (warp < V && lane < blocks) {
            const int p = rank * V + warp;
            push(peer_addr(smem_addr(parts + (last & 1) * (8 * kPadded) + (p >> 5) * kPadded + (p & 31)), lane), 0.0,
                 peer_addr(smem_addr(bars + (last & 1)), lane));
        }
        ok = arrived(last) && ok;
    }
    if ((int)(last + 1) / 2 > halos) {
        if (t == 0) bar_expect(smem_addr(bars + 2), halo_bytes);
        ok = halo_arrived(halos) && ok;
    }
    return ok;
}

// Bound by the latency of an iteration's two reductions (about 900 cycles
// each: staged values, one warp's tree per partial, st.async, mbarrier) and,
// from K = 4 on, by shared-memory bandwidth (ten 8-byte accesses per cell).
// Per iteration of a solve (slope over the iteration count), k_cg and this
// kernel: 6 000 cells 11.6 and 1.8 us, 11.6 k 11.1 and 2.4, 25.7 k 11.9 and 3.4,
// 50 k 12.4 and 5.2.
//
// Every wait is bounded.  A block whose wait runs out tells the others when
// the cluster meets at the end, and then every copy still on its way is waited
// for before a block leaves (below); the solve reports FFR_FLAG_TIMEOUT.
//
// ABSENT (self-test): the last block stays away from reduction A.absent_at.
template <int K, bool ABSENT>
__global__ void __launch_bounds__(kResThreads, 1) k_cg_cluster(CGArgs A, int nparts)
{
    constexpr int OWN = K * kResThreads, V = OWN / kResGroup;   // cells and partials of a block
    constexpr int KW = K <= 2 ? K : 1;
    extern __shared__ __align__(16) double res_sm[];
    __shared__ __align__(8) unsigned long long s_bar[3];        // partials (two sets), halo
    __shared__ unsigned s_gave_up, s_seq;
    if (A.st && A.st->halt) return;
    const RoomDev &R = A.R;
    const int nx = R.nx, ny = R.ny, nz = R.nz, n = R.n, plane = ny * nz;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int rank = blockIdx.x, base = rank * OWN, blocks = gridDim.x;
    const ClusterLayout lay(K, nx, ny, nz);
    const int plane2 = lay.plane2;
    double *sd = res_sm + lay.dir, *srh = res_sm + lay.halo, *sr = res_sm + lay.own_r, *stage = res_sm + lay.stage,
           *parts = res_sm + lay.parts, *stab = res_sm + lay.table;
    // cells the other blocks own of this block's two halos
    const int halo_bytes = 8 * (min(plane2, base) + min(plane2, (blocks - 1 - rank) * OWN));

    for (int a = t; a < lay.total; a += kResThreads) res_sm[a] = 0.0;
    if (t == 0) s_gave_up = 0;
    __syncthreads();
    bool even = true;
    if (K > 2) {
        // the scales of an axis agree on an even grid; then three of them are enough
        for (int a = t; a < 2 * (nx + ny + nz); a += kResThreads) {
            const int first = a < 2 * nx ? 0 : (a < 2 * (nx + ny) ? 2 * nx : 2 * (nx + ny));
            stab[a] = R.scale[a];
            even = even && R.scale[a] == R.scale[first];
        }
        even = __syncthreads_and(even);
    }
    if (t < 3) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_bar[t])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cooperative_groups::this_cluster().sync();

    unsigned seq = 0;                // reductions so far; the odd ones push a halo
    int halos = 0;                   // halos received
    bool failed = false;             // a wait ran out

    // Sums what `put` staged (one value per own cell) over all cells;
    // with_halo also pushes r (in sr) to the blocks whose halo holds it.
    auto put = [&](int q, double v) { stage[(q * (kResThreads / 32) + warp) * kPadded + lane] = v; };
    auto reduce = [&](bool with_halo, double &total) -> bool {
        if (ABSENT && rank == blocks - 1 && (int)seq + 1 == A.absent_at) return false;
        seq++;
        if (with_halo) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (with_halo) push_halo(OWN, plane2, sr, srh, s_bar);
        const unsigned bar = smem_addr(&s_bar[seq & 1]);
        double *set = parts + (seq & 1) * (8 * kPadded);
        if (t == 0) bar_expect(bar, 8 * V * blocks);
        if (warp < V) {
            const double s = sum256(stage + warp * 8 * kPadded);
            const int p = rank * V + warp;
            if (lane < blocks)
                push(peer_addr(smem_addr(set + (p >> 5) * kPadded + (p & 31)), lane), s, peer_addr(bar, lane));
        }
        failed = !bar_wait(bar, ((seq - 1) >> 1) & 1u) || failed;
        failed = __syncthreads_or(failed);
        total = nparts <= 32 ? warp_sum(set[lane]) : sum256(set);
        return !failed;
    };

    // set-up: r = rhs (0 in SOLID rows), x = 0, ||r||^2
    // (the direction of the own cells is kept in shared memory only, with
    // many cells per thread r too: registers would spill)
    constexpr bool R_SHARED = K >= 8;
    double x[K], r[R_SHARED ? 1 : K] = {}, ad[K], diag[K], wt[KW][6];
    auto r_of = [&](int q) {
        if constexpr (R_SHARED) return sr[t + q * kResThreads];
        else return r[q];
    };
    unsigned code[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const ResRow row(A, base + t + q * kResThreads);
        code[q] = row.code;
        diag[q] = row.diag;
        if (K <= 2)
#pragma unroll
            for (int a = 0; a < 6; a++) wt[q % KW][a] = row.w[a];
        x[q] = 0.0;
        if constexpr (!R_SHARED) r[q] = row.rhs;
        put(q, row.rhs * row.rhs);
        sr[t + q * kResThreads] = row.rhs;
    }
    const double s3[3] = {K > 2 ? stab[0] : 0.0, K > 2 ? stab[2 * nx] : 0.0, K > 2 ? stab[2 * (nx + ny)] : 0.0};
    double rr = 0.0, bnorm = 0.0, res = 0.0;
    int flags = 0, iters = 0;
    if (!reduce(true, rr)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
    bnorm = sqrt(rr);
    if (bnorm < 1e-15) goto finish;
    {
        double beta = 0.0;
        const double far = not_converged_above(A.tol, bnorm);
        int it = 0;
        for (; it < A.max_iter; it++) {
            // d = r + beta d on the own cells and on the halo
#pragma unroll
            for (int q = 0; q < K; q++) {
                double *s = sd + plane2 + t + q * kResThreads;
                *s = it == 0 ? r_of(q) : fma(beta, *s, r_of(q));
            }
            if (t == 0) bar_expect(smem_addr(&s_bar[2]), halo_bytes);
            failed = !bar_wait(smem_addr(&s_bar[2]), (unsigned)halos & 1u) || failed;
            halos++;
#pragma unroll 4
            for (int h = t; h < 2 * plane2; h += kResThreads) {
                const int a = h < plane2 ? h : h + OWN;
                sd[a] = it == 0 ? srh[h] : fma(beta, sd[a], srh[h]);
            }
            failed = __syncthreads_or(failed);
            if (failed) { flags = FFR_FLAG_TIMEOUT; goto finish; }
            // A d
#pragma unroll
            for (int q = 0; q < K; q++) {
                const double *s = sd + plane2 + t + q * kResThreads;
                const double dn[6] = {s[-plane], s[plane], s[-nz], s[nz], s[-1], s[1]};
                double w[6], o = 0.0;
                if (K <= 2) {
#pragma unroll
                    for (int a = 0; a < 6; a++) w[a] = wt[q % KW][a];
                } else if (even) {
                    // (opaque, or the compiler keeps every cell's weights and spills)
                    asm volatile("" : "+r"(code[q]));
#pragma unroll
                    for (int a = 0; a < 6; a++) w[a] = ((code[q] >> (2 * a)) & 3u) == SC_IN ? s3[a >> 1] : 0.0;
                } else {
                    int i, j, k;
                    decode(min(base + t + q * kResThreads, n - 1), ny, nz, i, j, k);
                    const int at[6] = {i, nx + i, 2 * nx + j, 2 * nx + ny + j, 2 * (nx + ny) + k, 2 * (nx + ny) + nz + k};
#pragma unroll
                    for (int a = 0; a < 6; a++) w[a] = ((code[q] >> (2 * a)) & 3u) == SC_IN ? stab[at[a]] : 0.0;
                }
#pragma unroll
                for (int a = 0; a < 6; a++) o += w[a] * dn[a];
                const double d = *s, v = diag[q] * d - o;
                ad[q] = (code[q] & SC_SOLID) ? d : v;
                put(q, d * ad[q]);
            }
            double dad;
            if (!reduce(false, dad)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
            if (fabs(dad) < 1e-30) {
                flags |= FFR_FLAG_CG_BREAKDOWN;
                break;
            }
            const double alpha = rr / dad;
#pragma unroll
            for (int q = 0; q < K; q++) {
                const double rv = r_of(q) - alpha * ad[q];
                sr[t + q * kResThreads] = rv;
                x[q] = fma(alpha, sd[plane2 + t + q * kResThreads], x[q]);
                if constexpr (!R_SHARED) r[q] = rv;
                put(q, rv * rv);
            }
            double rr1;
            if (!reduce(true, rr1)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
            if (!(rr1 > far)) {
                res = sqrt(rr1) / bnorm;
                if (res < A.tol) {
                    iters = it + 1;
                    break;
                }
            }
            beta = rr1 / rr;
            rr = rr1;
        }
        if (it >= A.max_iter || (flags & FFR_FLAG_CG_BREAKDOWN)) {
            iters = A.max_iter;
            res = sqrt(rr) / bnorm;
            if (!(flags & FFR_FLAG_CG_BREAKDOWN)) flags |= FFR_FLAG_CG_MAXITER;
        }
    }
finish:
#pragma unroll
    for (int q = 0; q < K; q++) {
        const int c = base + t + q * kResThreads;
        if (c < n) A.x[c] = x[q];
    }
    // the halo that the last reduction pushed
    failed = (flags & FFR_FLAG_TIMEOUT) != 0;
    if (!failed && (seq & 1)) {
        if (t == 0) bar_expect(smem_addr(&s_bar[2]), halo_bytes);
        failed = !bar_wait(smem_addr(&s_bar[2]), (unsigned)halos & 1u);
        halos++;
    }
    // no block leaves while another may still write its shared memory, and a
    // block that gave up says so to all
    if (__syncthreads_or(failed) && t < blocks)
        asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(peer_addr(smem_addr(&s_gave_up), t)) : "memory");
    cooperative_groups::this_cluster().sync();
    if (s_gave_up) {
        if (t == 0) s_seq = seq;
        const bool landed = await_copies(OWN, plane2, halo_bytes, seq, halos, sr, srh, parts, s_bar, s_seq);
        if (ABSENT && !__syncthreads_and(landed) && t == 0) atomicExch(A.absent_lost, 1);
        cooperative_groups::this_cluster().sync();
        flags |= FFR_FLAG_TIMEOUT;
    }
    if (rank == 0 && t == 0) res_results(A, res, iters, flags);
}

// ----------------------------------------------------------------- grid

// The partials p, p + 256 and their partners 16 further on meet first in the
// summation tree, so one block takes these four chunks of 256 cells and hands
// out one value: 128 blocks, 128 values.
__device__ __forceinline__ int chunk_of(int block, int v)
{
    return (block >> 4) * 32 + (block & 15) + 16 * (v >> 1) + 256 * (v & 1);
}

// Bound by the two exchanges.  Of 13 k cycles per iteration at 123 k cells
// (block 40, clock reads included) 4.4 k pass waiting for the block sums of
// d.Ad, 4.2 k for those of r.r and the halo's words, 1.3 k go into forming and
// publishing the sums, 0.9 k into the direction with its halo, 0.6 k into A d,
// 0.5 k into the update of x and r, the rest into the final sums.  Fences instead
// of numbered words cost 2-3 k cycles on each side of an exchange.  Per iteration
// of a solve (slope over the iteration count), k_cg and this kernel: 72 k cells
// 12.8 and 6.2 us, 123 k 15.2 and 6.3.
//
// ABSENT (self-test): the last block stays away from reduction A.absent_at.
//
// `words`: the tagged halves of r, {lo, hi} per cell; `slots`: those of the
// block sums, two sets of kMailboxes x 128, then the error word.
template <bool ABSENT>
__global__ void __launch_bounds__(kResThreads, 1)
    k_cg_chunks(CGArgs A, unsigned long long *words, unsigned long long *slots, int nparts)
{
    constexpr int K = 2;                            // cells of a thread: chunk 2 q + (t >> 8)
    extern __shared__ __align__(16) double res_sm[];
    __shared__ double s_part[kChunks], s_fin[8];
    if (A.st && A.st->halt) return;
    const RoomDev &R = A.R;
    const int nz = R.nz, n = R.n, plane = R.ny * nz;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, block = blockIdx.x;
    const ChunkLayout lay(nz);
    double *sd = res_sm + lay.dir, *srh = res_sm + lay.halo, *stage = res_sm + lay.stage;
    int *err = reinterpret_cast<int *>(slots + kSlotWords);
    const int side = 2 * kResGroup + 2 * nz, nhalo = lay.nhalo;
    for (int a = t; a < lay.total; a += kResThreads) res_sm[a] = 0.0;
    // halo element h: its place in the direction windows (-1: no such cell) and its cell
    int2 *at = reinterpret_cast<int2 *>(res_sm + lay.at);
    __syncthreads();
    for (int h = t; h < nhalo; h += kResThreads) {
        const int v = h / side, e = h - v * side, first = chunk_of(block, v) * kResGroup;
        int cell, w = kResGroup + e;
        if (e < nz) { w = e; cell = first - nz + e; }                            // before the chunk
        else if (e < 2 * nz) cell = first + kResGroup + e - nz;                  // after it
        else if (e < 2 * nz + kResGroup) cell = first - plane + e - 2 * nz;      // one plane before
        else cell = first + plane + e - 2 * nz - kResGroup;                      // one plane after
        const bool use = first < n && cell >= 0 && cell < n;
        at[h] = make_int2(use ? v * lay.window + w : -1, use ? cell : -1);
    }
    __syncthreads();

    unsigned seq = 0;
    bool failed = false;
    // Sums val over all cells; with a tag also collects the halo's r
    // published under it, while the block sums travel.
    auto reduce = [&](const double (&val)[K], unsigned tag, double &total) -> bool {
        if (ABSENT && block == kChunkBlocks - 1 && (int)seq + 1 == A.absent_at) return false;
        seq++;
#pragma unroll
        for (int q = 0; q < K; q++) stage[(q * (kResThreads / 32) + warp) * kPadded + lane] = val[q];
        __syncthreads();
        if (warp < kChunks) {
            const double s = sum256(stage + warp * 8 * kPadded);
            if (lane == 0) s_part[warp] = s;
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        unsigned long long *set = slots + (seq & 1) * (kSlotWords / 2);
        if (t < kMailboxes)
            tagged_store(set + 2 * (t * kChunkBlocks + block),
                         (0.0 + s_part[0] + s_part[1]) + (0.0 + s_part[2] + s_part[3]), seq);
        WaitLimit w;
        if (t < kChunkBlocks) {
            double v = 0.0;
            while (!tagged_load(set + 2 * (block % kMailboxes * kChunkBlocks + t), seq, v))
                if (w.over(err)) { failed = true; break; }
            // the rest of the tree: 16 lanes per warp sum, then the eight of them
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if ((lane & 15) == 0) s_fin[t >> 4] = v;
        } else if (tag) {
            constexpr int U = 6, T = kResThreads - kChunkBlocks;
            for (int h0 = t - kChunkBlocks; h0 < nhalo && !failed; h0 += T * U) {
                double v[U];
                int cell[U];
                bool ok;
#pragma unroll
                for (int a = 0; a < U; a++) cell[a] = h0 + T * a < nhalo ? at[h0 + T * a].y : -1;
                do {
                    ok = true;
#pragma unroll
                    for (int a = 0; a < U; a++)
                        if (cell[a] >= 0) ok = tagged_load(words + 2 * (size_t)cell[a], tag, v[a]) && ok;
                    if (!ok && w.over(err)) { failed = true; break; }
                } while (!ok);
#pragma unroll
                for (int a = 0; a < U; a++)
                    if (cell[a] >= 0) srh[h0 + T * a] = v[a];
            }
        }
        failed = __syncthreads_or(failed);
        const double f[8] = {s_fin[0], s_fin[1], s_fin[2], s_fin[3], s_fin[4], s_fin[5], s_fin[6], s_fin[7]};
        total = tree8(f);
        return !failed;
    };

    double x[K], r[K], d[K], ad[K], val[K], diag[K], wt[K][6];
    unsigned code[K];
    int cell[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const int p = chunk_of(block, 2 * q + (t >> 8));
        cell[q] = p < nparts ? p * kResGroup + (t & 255) : n;
        const ResRow row(A, cell[q]);
        code[q] = row.code;
        diag[q] = row.diag;
#pragma unroll
        for (int a = 0; a < 6; a++) wt[q][a] = row.w[a];
        x[q] = 0.0;
        d[q] = 0.0;
        r[q] = row.rhs;
        val[q] = r[q] * r[q];
        // no number of an earlier solve is left where others will look for one
        if (cell[q] < n) tagged_store(words + 2 * (size_t)cell[q], 0.0, 0u);
    }
    double rr = 0.0, bnorm = 0.0, res = 0.0;
    int flags = 0, iters = 0;
    __threadfence();
    if (!reduce(val, 0u, rr)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
    __threadfence();
    bnorm = sqrt(rr);
    if (bnorm < 1e-15) goto finish;
    {
        double beta = 0.0, sum;
        const double far = not_converged_above(A.tol, bnorm);
        int it = 0;
        if (A.max_iter > 0) {
            // the first halo (its reduction's sum is not used)
#pragma unroll
            for (int q = 0; q < K; q++) {
                if (cell[q] < n) tagged_store(words + 2 * (size_t)cell[q], r[q], 1u);
                val[q] = 0.0;
            }
            if (!reduce(val, 1u, sum)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
        }
        for (; it < A.max_iter; it++) {
            // d = r + beta d on the own cells and on the halo
#pragma unroll
            for (int q = 0; q < K; q++) {
                d[q] = it == 0 ? r[q] : fma(beta, d[q], r[q]);
                sd[(2 * q + (t >> 8)) * lay.window + nz + (t & 255)] = d[q];
            }
#pragma unroll 4
            for (int h = t; h < nhalo; h += kResThreads) {
                const int place = at[h].x;
                if (place >= 0) sd[place] = it == 0 ? srh[h] : fma(beta, sd[place], srh[h]);
            }
            __syncthreads();
            // A d
#pragma unroll
            for (int q = 0; q < K; q++) {
                const double *s = sd + (2 * q + (t >> 8)) * lay.window + nz + (t & 255);
                const double *xm = s + kResGroup + nz, *xp = xm + kResGroup;
                const double dn[6] = {*xm, *xp, s[-nz], s[nz], s[-1], s[1]};
                double o = 0.0;
#pragma unroll
                for (int a = 0; a < 6; a++) o += wt[q][a] * dn[a];
                const double v = diag[q] * d[q] - o;
                ad[q] = (code[q] & SC_SOLID) ? d[q] : v;
                val[q] = d[q] * ad[q];
            }
            if (!reduce(val, 0u, sum)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
            if (fabs(sum) < 1e-30) {
                flags |= FFR_FLAG_CG_BREAKDOWN;
                break;
            }
            const double alpha = rr / sum;
#pragma unroll
            for (int q = 0; q < K; q++) {
                const double rv = r[q] - alpha * ad[q];
                if (cell[q] < n) tagged_store(words + 2 * (size_t)cell[q], rv, (unsigned)it + 2u);
                x[q] = fma(alpha, d[q], x[q]);
                r[q] = rv;
                val[q] = rv * rv;
            }
            if (!reduce(val, (unsigned)it + 2u, sum)) { flags = FFR_FLAG_TIMEOUT; goto finish; }
            if (!(sum > far)) {
                res = sqrt(sum) / bnorm;
                if (res < A.tol) {
                    iters = it + 1;
                    break;
                }
            }
            beta = sum / rr;
            rr = sum;
        }
        if (it >= A.max_iter || (flags & FFR_FLAG_CG_BREAKDOWN)) {
            iters = A.max_iter;
            res = sqrt(rr) / bnorm;
            if (!(flags & FFR_FLAG_CG_BREAKDOWN)) flags |= FFR_FLAG_CG_MAXITER;
        }
    }
finish:
#pragma unroll
    for (int q = 0; q < K; q++)
        if (cell[q] < n) A.x[cell[q]] = x[q];
    if (block == 0 && t == 0) res_results(A, res, iters, flags);
}

FFR_DEFINE_WAIT_LIMIT_SETTER(set_wait_limit_cgres)

namespace {

// Shared memory beside the dynamic part (a kernel's static arrays).
constexpr int kResStatic = 256;

struct ResLimits {
    int sms = 0, smem = 0;       // SMs, dynamic shared memory of one block at most
    ResLimits()
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        smem -= kResStatic;
    }
};
const ResLimits &limits()
{
    static const ResLimits l;
    return l;
}

// Lets a kernel take all of the shared memory.  (The limit is one value per
// kernel and process: set to what each room needs, a launch of a smaller room
// in another thread would lower it between a larger one's call and its launch.)
template <class F> int allow_smem(F *fn)
{
    FFR_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limits().smem));
    return FFR_OK;
}

template <class F> int allow_cluster(F *fn)
{
    FFR_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return allow_smem(fn);
}

// Whether the device holds a cluster of `blocks` blocks of this form at once
// (with all of the shared memory, whatever the room needs of it).
template <int K> bool placeable(int blocks)
{
    static ClusterCheck check;
    if (allow_cluster(k_cg_cluster<K, false>)) return false;
    return check((const void *)k_cg_cluster<K, false>, blocks, kResThreads, (size_t)limits().smem);
}

template <int K> int launch_cluster(const CGArgs &a, int nparts, cudaStream_t s)
{
    auto *fn = a.absent_at ? k_cg_cluster<K, true> : k_cg_cluster<K, false>;
    const size_t smem = 8 * (size_t)ClusterLayout(K, a.R.nx, a.R.ny, a.R.nz).total;
    if (int rc = allow_cluster(fn)) return rc;
    const unsigned blocks = (unsigned)cluster_blocks(a.R.n, K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FFR_CUDA(cudaLaunchKernelEx(&cfg, fn, a, nparts));
    count_launch(1);
    return FFR_OK;
}

int launch_chunks(const CGArgs &a, int nparts, cudaStream_t s)
{
    auto *fn = a.absent_at ? k_cg_chunks<true> : k_cg_chunks<false>;
    const size_t smem = 8 * (size_t)ChunkLayout(a.R.nz).total;
    if (int rc = allow_smem(fn)) return rc;
    unsigned long long *words = reinterpret_cast<unsigned long long *>(a.da);
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(a.ad);
    // the block sums' numbers and the error word start at zero
    FFR_CUDA(cudaMemsetAsync(slots, 0, 8 * (kSlotWords + 1), s));
    void *args[] = {(void *)&a, &words, &slots, &nparts};
    FFR_CUDA(cudaLaunchCooperativeKernel((void *)fn, dim3(kChunkBlocks), dim3(kResThreads), args, smem, s));
    count_launch(1);
    return FFR_OK;
}

}  // namespace

int launch_cg_resident(const CGArgs &a, cudaStream_t s, bool *taken)
{
    const RoomDev &R = a.R;
    const int nparts = (int)cdiv(R.n, kResGroup);
    const int form = cg_form(R.nx, R.ny, R.nz, limits().smem, limits().sms, a.db - a.da >= R.n, [](int K, int blocks) {
        return K == 1 ? placeable<1>(blocks)
                      : (K == 2 ? placeable<2>(blocks) : (K == 4 ? placeable<4>(blocks) : placeable<8>(blocks)));
    });
    *taken = form != CG_GRID;
    switch (form) {
    case 1: return launch_cluster<1>(a, nparts, s);
    case 2: return launch_cluster<2>(a, nparts, s);
    case 4: return launch_cluster<4>(a, nparts, s);
    case 8: return launch_cluster<8>(a, nparts, s);
    case CG_CHUNKS: return launch_chunks(a, nparts, s);
    }
    return FFR_OK;
}

}  // namespace ffr
