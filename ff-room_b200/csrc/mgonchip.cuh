// mgonchip.cuh — the V-cycle from level `lo` down inside one thread-block
// cluster, its arrays in shared memory (sm_100a).
//
// Included by mgpcg.cu.  Every cell update is the one smooth_color and
// restrict_level make, operand for operand, so the values do not depend on
// which form ran (the colours are Jacobi sweeps).
//
// What bounds it is the chain of half sweeps (seven per level and V-cycle, and
// thirty-two on the coarsest), each a round of loads and a barrier.  So:
//  - a level is split over the cluster by whole i-planes; the two boundary
//    planes of a colour are stored into the neighbours' halo planes as they are
//    computed, and a half sweep reads its own shared memory only;
//  - levels of at most kOcBlockCells cells stay with block 0 alone, where a
//    half sweep costs a __syncthreads instead of a cluster barrier, and those
//    of at most 32 cell pairs with one of its warps;
//  - red and black cells are kept in arrays of their own, indexed by the pair
//    (k, k+1) that holds one of each: the x and y neighbours of pair q's cell
//    and one of its z neighbours are at q, q +- a row, q +- a plane of the
//    other colour, so neighbouring threads read neighbouring words;
//  - level 0 takes its row from the stencil codes, the others from couplings
//    loaded once per launch;
//  - restriction stores the red cells' residuals (the black ones' are zero)
//    and sums them per coarse cell after a barrier; prolongation adds the
//    correction to the red cells, which only the next black half sweep reads;
//  - the coarsest level stays in the registers of one warp;
//  - one function per kind of pass serves every level, not inlined: with the
//    passes unrolled per level the code (executed once per V-cycle) kept
//    missing the instruction cache, 0.9 k cycles per pass of 0.2 k.
#pragma once

#include <type_traits>

namespace ffr {

extern __shared__ float oc_smem[];

// The arrays of one level, two of each (red, black): x with a halo plane on
// either side, b, the diagonal D, then on level 0 the codes (16 bits), else the
// couplings towards +x, +y, +z with the plane below.  A byte per pair follows.
struct OcLevel {
    int nx, ny, nz, pk, rp;     // pk pairs per row, rp pairs per plane
    int sx, sy, sz;
    int P, p0, np, n;           // planes of a block; this block's first plane, its planes and pairs
    unsigned mag_rp, mag_pk;
    int base, h2, h1, own, flag;   // first word; words of an array with two, one and no halo planes; the bytes
    // pair m of the own planes: m in b, D and code, rp + m in x and t
    __device__ __forceinline__ float *x(int c) const { return oc_smem + base + c * h2; }
    __device__ __forceinline__ float *b(int c) const { return oc_smem + base + 2 * h2 + c * own; }
    __device__ __forceinline__ float *D(int c) const { return oc_smem + base + 2 * (h2 + own) + c * own; }
    __device__ __forceinline__ float *t(int a, int c) const
    {
        return oc_smem + base + 2 * h2 + 4 * own + (2 * a + c) * h1;
    }
    __device__ __forceinline__ unsigned short *code(int c) const
    {
        return reinterpret_cast<unsigned short *>(oc_smem + base + 2 * h2 + 4 * own) + c * own;
    }
    __device__ __forceinline__ unsigned char *flags() const { return reinterpret_cast<unsigned char *>(oc_smem + flag); }
};
// bits of a pair's byte: the red cell is the second one; the red, the black
// cell is an unknown; the pair begins its row
enum : unsigned { OF_PAR = 1, OF_RED = 2, OF_BLACK = 4, OF_FIRST = 8 };

// A launch's levels, in shared memory.
struct OcLevels {
    OcLevel lv[kMaxLevels];
};

__device__ __forceinline__ OcLevel oc_level(const MGDev &M, const OnchipPlan &Q, int l, int rank)
{
    OcLevel L;
    const MGLevel &G = M.lv[l];
    L.nx = G.nx; L.ny = G.ny; L.nz = G.nz;
    L.sx = G.sx; L.sy = G.sy; L.sz = G.sz;
    L.pk = (G.nz + 1) >> 1;
    L.rp = G.ny * L.pk;
    L.P = Q.planes[l];
    L.p0 = l >= Q.fb ? 0 : rank * L.P;
    L.np = l >= Q.fb ? (rank == 0 ? G.nx : 0) : max(0, min(L.P, G.nx - L.p0));
    L.n = L.np * L.rp;
    L.mag_rp = Q.mag_rp[l];
    L.mag_pk = Q.mag_pk[l];
    L.base = Q.off[l];
    L.flag = Q.off_flag[l];
    L.h2 = (L.P + 2) * L.rp;
    L.h1 = (L.P + 1) * L.rp;
    L.own = L.P * L.rp;
    return L;
}

// n / d with mag = floor((2^32 - 1) / d) + 1 (exact while n d < 2^32)
__device__ __forceinline__ int oc_div(int n, int d, unsigned mag) { return d == 1 ? n : (int)__umulhi((unsigned)n, mag); }

// Pair m of a level (from plane p0 + first on): its plane, row and place in the row.
struct OcItem {
    int i, j, p;
    __device__ __forceinline__ OcItem(const OcLevel &L, int m, int first = 0)
    {
        const int slot = oc_div(m, L.rp, L.mag_rp), rem = m - slot * L.rp;
        j = oc_div(rem, L.pk, L.mag_pk);
        p = rem - j * L.pk;
        i = L.p0 + first + slot;
    }
};

// The couplings of one cell in the order x-, x+, y-, y+, z-, z+ (0 where the
// neighbour is no unknown); hi: the cell is its pair's second one.
template <bool FINE>
__device__ __forceinline__ void oc_row(const MGDev &M, const OcLevel &L, int m, int c, unsigned f, float (&t)[6])
{
    const bool hi = (f ^ c) & 1u;
    if constexpr (FINE) {
        const unsigned code = L.code(c)[m];
        if (M.uniform) {
            const float t3[3] = {M.tx, M.ty, M.tz};
#pragma unroll
            for (int a = 0; a < 6; a++) t[a] = ((code >> (2 * a)) & 3u) == SC_IN ? t3[a >> 1] : 0.0f;
        } else {
            const OcItem it(L, m);
            float D;
            fine_coefs(M, code, it.i, it.j, min(2 * it.p + (hi ? 1 : 0), L.nz - 1), t, D);
        }
    } else {
        const int q = L.rp + m, o = c ^ 1;
        t[0] = L.t(0, o)[q - L.rp];
        t[1] = L.t(0, c)[q];
        t[2] = L.t(1, o)[q - L.pk];
        t[3] = L.t(1, c)[q];
        t[4] = !hi && (f & OF_FIRST) ? 0.0f : L.t(2, o)[hi ? q : q - 1];
        t[5] = L.t(2, c)[q];
    }
}

// x of the six neighbours (all of the other colour).
__device__ __forceinline__ void oc_neighbours(const OcLevel &L, int m, int c, unsigned f, float (&v)[6])
{
    const float *o = L.x(c ^ 1) + L.rp + m;
    const int hi = (int)((f ^ c) & 1u);
    v[0] = o[-L.rp];
    v[1] = o[L.rp];
    v[2] = o[-L.pk];
    v[3] = o[L.pk];
    v[4] = o[hi - 1];
    v[5] = o[hi];
}

__device__ __forceinline__ float oc_sum(const float (&t)[6], const float (&v)[6])
{
    // (the choice is made on v: it stays off the chain of sums)
    float s = 0.0f;
#pragma unroll
    for (int a = 0; a < 6; a++) s += t[a] * (t[a] != 0.0f ? v[a] : 0.0f);
    return s;
}

__device__ __forceinline__ void oc_store_peer(const float *local, int rank, float v)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

__device__ __forceinline__ float oc_load_peer(const float *local, int rank)
{
    unsigned a;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// Stores x of pair m's cell of colour c and hands it to the neighbour whose
// halo holds its plane.
__device__ __forceinline__ void oc_set(const OcLevel &L, int m, int c, float val, int rank, bool share)
{
    float *x = L.x(c);
    x[L.rp + m] = val;
    if (share) {
        if (m < L.rp && rank > 0) oc_store_peer(x + (L.P + 1) * L.rp + m, rank - 1, val);
        const int r = m - (L.n - L.rp);
        if (r >= 0 && L.p0 + L.np < L.nx) oc_store_peer(x + r, rank + 1, val);
    }
}

// The threads that work on a level: the cluster's, or the first n of block 0
// (as many warps as the level has pairs for; those of the next coarser level are
// among them).  A barrier of each level, of its own number, holds them together;
// a thread that the next level does not need goes on to wait there.
struct OcTeam {
    int id, n;      // id < 0: the cluster
    __device__ __forceinline__ void sync() const
    {
        // (shared memory only crosses blocks, so no device-wide fence)
        if (id < 0) cooperative_groups::this_cluster().sync();
        else if (n == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
    }
};

// One half sweep over the cells of colour c, by threads t of nt; `share`: the
// boundary planes to the neighbours.
template <bool FINE>
__device__ __noinline__ void oc_sweep(const MGDev &M, const OcLevel &L_, int c, int t, int nt, int rank, bool share)
{
    // (in registers: every field fetched again for a pair is a round trip to
    // shared memory; a half sweep of 1600 pairs per block went from 4.6 k to 3.4 k
    // cycles without them)
    const OcLevel L = L_;
    for (int m = t; m < L.n; m += nt) {
        const unsigned f = L.flags()[m];
        float tt[6], v[6];
        oc_row<FINE>(M, L, m, c, f, tt);
        oc_neighbours(L, m, c, f, v);
        const float b = L.b(c)[m], D = L.D(c)[m];
        if (f & (OF_RED << c)) oc_set(L, m, c, (b + oc_sum(tt, v)) / D, rank, share);
    }
}

// Residuals of the red cells (0 where there is no unknown), pair by pair, to
// res of block `to` (this block's own: to == rank).
template <bool FINE>
__device__ __noinline__ void oc_residual(const MGDev &M, const OcLevel &L_, float *res, int t, int nt, int rank, int to)
{
    const OcLevel L = L_;
    for (int m = t; m < L.n; m += nt) {
        const unsigned f = L.flags()[m];
        float tt[6], v[6];
        oc_row<FINE>(M, L, m, 0, f, tt);
        oc_neighbours(L, m, 0, f, v);
        const float b = L.b(0)[m], D = L.D(0)[m], x = L.x(0)[L.rp + m];
        const float r = f & OF_RED ? b - (D * x - oc_sum(tt, v)) : 0.0f;
        if (to == rank) res[m] = r;
        else oc_store_peer(res + m, to, r);
    }
}

// What a level's smoothing does besides its sweeps.
enum : unsigned { OS_UP = 1,       // after the prolongation (else before the restriction)
                  OS_SHARE = 2,    // boundary planes go to the neighbours
                  OS_TOP = 4 };    // the first level on chip: its last sweep needs no halo

// All half sweeps of one visit of a level of at most one pair per thread (not
// level 0), and on the way down the red residuals (as oc_residual): the pair's
// rows, right-hand sides and place are loaded once and stay in registers, which
// took a half sweep of the lone block from 0.9 k cycles to 0.3 k.  Not for more
// pairs per thread: three in registers measured 10 % slower per iteration than
// oc_sweep (the code grows with them, and every pass of a V-cycle runs once, so
// it is the fetching of instructions that then bounds it).
__device__ __noinline__ void oc_smooth(const MGDev &M, const OcLevel &L_, unsigned what, OcTeam team, int t, int rank,
                                       float *res, int to)
{
    const OcLevel L = L_;
    const int n = L.n, rp = L.rp, pk = L.pk, m = max(0, min(t, n - 1));
    float *const x0 = L.x(0) + rp + m, *const x1 = L.x(1) + rp + m;
    const unsigned f = t < n ? L.flags()[m] : 0u;
    const float b[2] = {L.b(0)[m], L.b(1)[m]}, D[2] = {L.D(0)[m], L.D(1)[m]};
    float row[2][6];
    oc_row<false>(M, L, m, 0, f, row[0]);
    oc_row<false>(M, L, m, 1, f, row[1]);
    const int h = (int)(f & 1u);
    auto sum = [&](int c) {
        const float *o = c ? x0 : x1;
        const int z = h ^ c;
        const float v[6] = {o[-rp], o[rp], o[-pk], o[pk], o[z - 1], o[z]};
        return oc_sum(row[c], v);
    };
    auto half = [&](int c, bool share) {
        const float val = (b[c] + sum(c)) / D[c];
        if (f & (OF_RED << c)) oc_set(L, m, c, val, rank, share && (what & OS_SHARE));
    };
    const bool up = what & OS_UP;
    for (int s = 0; s < kSmoothSweeps; s++) {
        const bool end = s + 1 == kSmoothSweeps, last = up && end && (what & OS_TOP);
        half(1, true);
        team.sync();
        if (!up && end) break;
        half(0, !last);
        if (!(last && (what & OS_SHARE))) team.sync();
    }
    if (up || t >= n) return;
    const float r = f & OF_RED ? b[0] - (D[0] * *x0 - sum(0)) : 0.0f;
    if (to == rank) res[m] = r;
    else oc_store_peer(res + m, to, r);
}

// Right-hand side and first red sweep of level C from the residuals of the
// finer level L's red cells (res: planes i0 on), summed in the order of a
// nested loop over the children.
__device__ __noinline__ void oc_coarse_rhs(const OcLevel &L, int i0, const float *res, const OcLevel &C, int t, int nt,
                                           int rank, bool share)
{
    // (in registers: every field of L that a test below had to fetch again was
    // a round trip to shared memory, 4.8 k cycles for a level of one pair per thread)
    const int nx = L.nx, ny = L.ny, nz = L.nz, sx = L.sx, sy = L.sy, sz = L.sz, pk = L.pk, rp = L.rp;
    const int cnz = C.nz, n = C.n;
    float *const cb[2] = {C.b(0), C.b(1)}, *const cD[2] = {C.D(0), C.D(1)};
    for (int m = t; m < n; m += nt) {
        const OcItem it(C, m);
        const int i = it.i << sx, j = it.j << sy, par = (it.i + it.j) & 1;
        float r[2][8];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int k = (2 * it.p + h) << sz;
            const int at = (i - i0) * rp + j * pk + (k >> 1), up = k & 1;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                // the red children inside the level
                const int a = q >> 2, b = (q >> 1) & 1, e = q & 1;
                const bool use = (a <= sx) & (b <= sy) & (e <= sz) & (i + a < nx) & (j + b < ny) & (k + e < nz) &
                                 (((i + j + k + a + b + e) & 1) == 0);
                r[h][q] = use ? res[at + a * rp + b * pk + ((up + e) >> 1)] : 0.0f;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int c = par ^ h;
            if (2 * it.p + h >= cnz) continue;
            float sum = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; q++) sum += r[h][q];
            const float DP = cD[c][m];
            cb[c][m] = sum;
            oc_set(C, m, c, c == 0 && DP != 0.0f ? sum / DP : 0.0f, rank, share);
        }
    }
}

// Adds the coarse correction to the red cells, halo planes included: the
// black half sweep after it is all that reads them before they are replaced.
// The coarse planes are C's own arrays (copy < 0) or `count` words per colour
// at `copy`, from plane `first` on.
__device__ __noinline__ void oc_prolong(const OcLevel &L, const OcLevel &C, int copy, int first, int count, int t, int nt)
{
    float *const x = L.x(0);
    const unsigned char *const flags = L.flags();
    const int base = copy < 0 ? C.base + (1 - C.p0) * C.rp : copy - first * C.rp, stride = copy < 0 ? C.h2 : count;
    const int n = L.n, rp = L.rp, nx = L.nx, nz = L.nz, sx = L.sx, sy = L.sy, sz = L.sz, crp = C.rp, cpk = C.pk;
    for (int e = t; e < n + 2 * rp && n > 0; e += nt) {
        const OcItem it(L, e, -1);
        const int k = 2 * it.p + ((it.i + it.j) & 1), m = e - rp;
        if ((it.i < 0) | (it.i >= nx) | (k >= nz)) continue;
        if (m >= 0 && m < n && !(flags[m] & OF_RED)) continue;
        const int I = it.i >> sx, J = it.j >> sy, K = k >> sz;
        x[e] += oc_smem[base + ((I + J + K) & 1) * stride + I * crp + J * cpk + (K >> 1)];
    }
}

// The coarsest level (at most 32 pairs): kCoarsestSweeps sweeps, black first,
// by one warp, a pair per lane with x and rows in registers.
__device__ __noinline__ void oc_coarsest(const MGDev &M, const OcLevel &L, int lane)
{
    const int m = min(lane, L.n - 1);
    const unsigned f = L.flags()[m];
    float t0[6], t1[6];
    oc_row<false>(M, L, m, 0, f, t0);
    oc_row<false>(M, L, m, 1, f, t1);
    const float b0 = L.b(0)[m], D0 = L.D(0)[m], b1 = L.b(1)[m], D1 = L.D(1)[m];
    const bool red = f & OF_RED, black = f & OF_BLACK;
    float x0 = L.x(0)[L.rp + m], x1 = L.x(1)[L.rp + m];
    // lanes of the neighbours (any lane where there is none: its weight is 0)
    const int xm = (m - L.rp) & 31, xp = (m + L.rp) & 31, ym = (m - L.pk) & 31, yp = (m + L.pk) & 31;
    const int h0 = f & 1, h1 = h0 ^ 1;
    const int z0m = (m + h0 - 1) & 31, z0p = (m + h0) & 31, z1m = (m + h1 - 1) & 31, z1p = (m + h1) & 31;
    auto from = [](float v, int lane_) { return __shfl_sync(0xffffffffu, v, lane_); };
    for (int sweep = 0; sweep < kCoarsestSweeps; sweep++) {
        const float v1[6] = {from(x0, xm), from(x0, xp), from(x0, ym), from(x0, yp), from(x0, z1m), from(x0, z1p)};
        if (black) x1 = (b1 + oc_sum(t1, v1)) / D1;
        __syncwarp();
        const float v0[6] = {from(x1, xm), from(x1, xp), from(x1, ym), from(x1, yp), from(x1, z0m), from(x1, z0p)};
        if (red) x0 = (b0 + oc_sum(t0, v0)) / D0;
        __syncwarp();
    }
    if (lane < L.n) {
        L.x(0)[L.rp + m] = x0;
        L.x(1)[L.rp + m] = x1;
    }
}

// Loads what a launch keeps: the levels, zeros, the couplings of every level
// on chip and level 0's codes, the pairs' bytes.
__device__ __noinline__ void oc_setup(const PCGArgs &A, const OnchipPlan &Q, int rank, OcLevels &S)
{
    const MGDev &M = A.M;
    const int t = threadIdx.x, nt = blockDim.x;
    for (int a = t; a < Q.floats; a += nt) oc_smem[a] = 0.0f;
    if (t >= Q.lo && t < M.nlev) S.lv[t] = oc_level(M, Q, t, rank);
    __syncthreads();
    for (int l = Q.lo; l < M.nlev; l++) {
        const OcLevel L = S.lv[l];
        if (L.n == 0) continue;
        // one plane below the own ones as well
        const int first = (l == 0 || L.p0 == 0) ? 0 : -1, count = L.n - first * L.rp;
        const float4 *const coef = M.lv[l].coef;
        constexpr int U = 4;      // pairs in flight
        for (int e0 = t; e0 < count; e0 += U * nt) {
            float4 cf[U][2];
            unsigned code[U][2];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const OcItem it(L, min(e0 + u * nt, count - 1), first);
                const int cell = (it.i * L.ny + it.j) * L.nz + 2 * it.p, two = 2 * it.p + 1 < L.nz;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (l == 0) code[u][h] = A.R.sc[cell + h * two];
                    else cf[u][h] = coef[cell + h * two];
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int e = e0 + u * nt, m = e + first * L.rp;
                if (e >= count) break;
                const OcItem it(L, e, first);
                const int par = (it.i + it.j) & 1;
                unsigned f = (par ? OF_PAR : 0u) | (it.p == 0 ? OF_FIRST : 0u);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int k = 2 * it.p + h, c = par ^ h;      // colour of cell k
                    if (k >= L.nz) continue;
                    if (l == 0) {
                        float tt[6], D;
                        fine_coefs(M, code[u][h], it.i, it.j, k, tt, D);
                        L.code(c)[m] = (unsigned short)code[u][h];
                        L.D(c)[m] = D;
                        if (active_code(code[u][h])) f |= OF_RED << c;
                    } else {
                        if (cf[u][h].w != 0.0f) f |= OF_RED << c;
                        L.t(0, c)[L.rp + m] = cf[u][h].x;
                        L.t(1, c)[L.rp + m] = cf[u][h].y;
                        L.t(2, c)[L.rp + m] = cf[u][h].z;
                        if (m >= 0) L.D(c)[m] = cf[u][h].w;
                    }
                }
                if (m >= 0) L.flags()[m] = (unsigned char)f;
            }
        }
    }
    __syncthreads();
}

// The V-cycle of levels lo .. nlev-1: level lo's right-hand side and first red
// sweep in global memory (M.lv[lo].b, .x), its x back there.  On level 0 the
// last red half sweep is left to the r.z pass.  Every block of the cluster
// calls it; global data is visible to the cluster before and must be made so
// by the caller afterwards.  FINE: lo may be 0.
template <bool FINE>
__device__ __noinline__ void oc_vcycle(const PCGArgs &A, const OnchipPlan &Q, int rank, const OcLevels &S)
{
    const MGDev &M = A.M;
    const int t = threadIdx.x, nt = blockDim.x, last = M.nlev - 1;
    const bool lone = Q.blocks == 1 || Q.fb == Q.lo;
    float *red = oc_smem + Q.off_red, *res0 = oc_smem + Q.off_res;
    auto sweep = [&](int l, int c, int n, bool share) {
        if (FINE && l == 0) oc_sweep<true>(M, S.lv[l], c, t, n, rank, share);
        else oc_sweep<false>(M, S.lv[l], c, t, n, rank, share);
    };
    auto residual = [&](int l, float *res, int n, int to) {
        if (FINE && l == 0) oc_residual<true>(M, S.lv[l], res, t, n, rank, to);
        else oc_residual<false>(M, S.lv[l], res, t, n, rank, to);
    };
    const OcTeam all{lone ? 0 : -1, nt};
    auto team_of = [&](int l) {
        return l < Q.fb ? all : OcTeam{1 + l - Q.fb, min(nt, (S.lv[l].nx * S.lv[l].rp + 31) & ~31)};
    };
    // one visit of a level: its half sweeps, on the way down the residuals too
    auto smooth = [&](int l, const OcTeam &T, bool up, float *res, int to) {
        const OcLevel &L = S.lv[l];
        const bool split = l < Q.fb, top = l == Q.lo;
        if (l > 0 && L.own <= T.n) {
            const unsigned what = (up ? OS_UP : 0u) | (split ? OS_SHARE : 0u) | (top ? OS_TOP : 0u);
            return oc_smooth(M, L, what, T, t, rank, res, to);
        }
        // (level 0 leaves its last red half sweep to the r.z pass)
        for (int sw = 0; sw < level_sweeps(l); sw++) {
            const bool end = sw + 1 == level_sweeps(l), stop = up && end && l == 0, out = up && end && top;
            sweep(l, 1, T.n, split && !stop);
            if (stop) return;
            T.sync();
            if (!up && end) break;
            sweep(l, 0, T.n, split && !out);
            if (!(out && split)) T.sync();
        }
        if (!up) residual(l, res, T.n, to);
    };
    {
        const OcLevel &L = S.lv[Q.lo];
        const float *gx = M.lv[Q.lo].x, *gb = M.lv[Q.lo].b;
        const int n = L.n, rp = L.rp, all_ = n > 0 ? n + 2 * rp : 0, nx = L.nx, ny = L.ny, nz = L.nz;
        float *const xs[2] = {L.x(0), L.x(1)}, *const bs[2] = {L.b(0), L.b(1)};
        constexpr int U = 4;      // pairs in flight
        for (int e0 = t; e0 < all_; e0 += U * nt) {
            float xv[U][2], bv[U][2];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const OcItem it(L, min(e0 + u * nt, all_ - 1), -1);
                const int i = max(0, min(it.i, nx - 1)), cell = (i * ny + it.j) * nz + 2 * it.p, two = 2 * it.p + 1 < nz;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    xv[u][h] = __ldcg(gx + cell + h * two);
                    bv[u][h] = __ldcg(gb + cell + h * two);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int e = e0 + u * nt, m = e - rp;
                if (e >= all_) break;
                const OcItem it(L, e, -1);
                if (it.i < 0 || it.i >= nx) continue;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int c = ((it.i + it.j) & 1) ^ h;
                    if (2 * it.p + h >= nz) continue;
                    xs[c][e] = xv[u][h];
                    if (m >= 0 && m < n) bs[c][m] = bv[u][h];
                }
            }
        }
        all.sync();        // a neighbour's first push must find its halo loaded
    }
    // down: the split levels by the cluster, the others by block 0
    for (int l = Q.lo; l < last; l++) {
        const bool split = l < Q.fb;
        const OcTeam T = team_of(l);
        if (!split && (rank != 0 || t >= T.n)) break;
        if (split && l + 1 == Q.fb) {
            smooth(l, T, false, res0 + S.lv[l].p0 * S.lv[l].rp, 0);
            T.sync();
            if (rank != 0) break;
            oc_coarse_rhs(S.lv[l], 0, res0, S.lv[l + 1], t, nt, 0, false);
            __syncthreads();
        } else {
            // (a split level's coarse planes have their children in the same block)
            smooth(l, T, false, red, rank);
            if (split) __syncthreads();
            else T.sync();
            oc_coarse_rhs(S.lv[l], S.lv[l].p0, red, S.lv[l + 1], t, T.n, rank, split);
            T.sync();
        }
    }
    const int coarsest = S.lv[last].nx * S.lv[last].rp;
    if (rank == 0) {
        if (coarsest <= 32) {
            if (t < 32) oc_coarsest(M, S.lv[last], t);
        } else if (t < team_of(last).n) {
            const OcTeam T = team_of(last);
            for (int sw = 0; sw < kCoarsestSweeps; sw++)
                for (int c = 1; c >= 0; c--) {
                    sweep(last, c, T.n, false);
                    T.sync();
                }
        }
    }
    // up
    for (int l = last - 1; l >= Q.lo; l--) {
        const bool split = l < Q.fb;
        const OcTeam T = team_of(l);
        if (!split && (rank != 0 || t >= T.n)) continue;
        // the coarser level's results to all who need them
        if (!split || l + 1 == Q.fb) T.sync();
        if (split && l + 1 == Q.fb) {
            // from block 0, through a copy of the planes around this block's parents
            const OcLevel &L = S.lv[l], &B = S.lv[Q.fb];
            const int first = max(0, (L.p0 - 1) >> L.sx), end = min(B.nx, ((L.p0 + L.np) >> L.sx) + 1);
            float *copy = oc_smem + Q.off_par;
            const int count = L.n > 0 ? (end - first) * B.rp : 0;
            for (int e = t; e < count; e += nt) {
                copy[e] = oc_load_peer(B.x(0) + (first + 1) * B.rp + e, 0);
                copy[count + e] = oc_load_peer(B.x(1) + (first + 1) * B.rp + e, 0);
            }
            __syncthreads();
            oc_prolong(L, B, Q.off_par, first, count, t, nt);
        } else {
            oc_prolong(S.lv[l], S.lv[l + 1], -1, 0, 0, t, T.n);
        }
        // (a neighbour stores into the red halo, prolonged here, after the next
        // cluster barrier only)
        if (split) __syncthreads();
        else T.sync();
        smooth(l, T, true, nullptr, rank);
    }
    __syncthreads();
    {
        const OcLevel &L = S.lv[Q.lo];
        float *gx = M.lv[Q.lo].x;
        for (int m = t; m < L.n; m += nt) {
            const OcItem it(L, m);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int k = 2 * it.p + h, c = ((it.i + it.j) & 1) ^ h;
                if (k < L.nz) gx[(it.i * L.ny + it.j) * L.nz + k] = L.x(c)[L.rp + m];
            }
        }
    }
}

}  // namespace ffr
