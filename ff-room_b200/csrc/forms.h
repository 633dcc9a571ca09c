// forms.h — which form of a solve a room and a device take.  Plain C++: sizes
// and rules only, `placeable` asks the device (a part of a GPU may not hold a
// cluster that the whole one holds, and a launch that cannot be placed fails).
#pragma once

#include <initializer_list>

#ifdef __CUDACC__
#define FFR_HD __host__ __device__
#else
#define FFR_HD
#endif

namespace ffr {

// ------------------------------------------ plain CG on chip (cgres.cu)

constexpr int kResThreads = 512;
constexpr int kResGroup = 256;               // cells of one partial (a k_cg block)
constexpr int kResClusterCtas = 16;
constexpr int kPadded = 36;                  // 32 values and 4 of padding (bank offset between groups)

FFR_HD constexpr int even_up(int v) { return (v + 1) & ~1; }

// Shared memory of one block of the cluster form, in doubles.  Halos are
// padded to an even number of cells at their outer end: a bulk copy moves
// 16-byte units.
struct ClusterLayout {
    int plane2;                              // cells of one halo side, padded
    int dir, halo, own_r, stage, parts, table, total;
    FFR_HD ClusterLayout(int K, int nx, int ny, int nz)
    {
        const int own = K * kResThreads;
        plane2 = even_up(ny * nz);
        dir = 0;                                        // direction: halo, own cells, halo
        halo = dir + own + 2 * plane2;                  // r of the two halos
        own_r = halo + 2 * plane2;                      // r of the own cells
        stage = own_r + own;                            // one value per own cell
        parts = stage + own / 32 * kPadded;             // two sets of 256 partials
        table = parts + 2 * 8 * kPadded;
        total = table + (K > 2 ? 2 * (nx + ny + nz) : 0);   // stencil scales (else in registers)
    }
};

// The grid form: blocks, and chunks of kResGroup cells per block.
constexpr int kChunks = 4, kChunkBlocks = 128;
constexpr int kChunkMaxParts = 512;

// Shared memory of one block of the grid form, in doubles.  Each chunk keeps
// the direction on three windows: its cells with nz more on either side, and
// the 256 cells one plane before and one after.
struct ChunkLayout {
    int window, nhalo, dir, halo, at, stage, total;
    FFR_HD ChunkLayout(int nz)
    {
        window = 3 * kResGroup + 2 * nz;
        nhalo = kChunks * (2 * kResGroup + 2 * nz);
        dir = 0;
        halo = dir + kChunks * window;              // r of the halo cells, in window order
        at = halo + nhalo;                          // their places in the windows and their cells
        stage = at + nhalo;
        total = stage + kChunks * 8 * kPadded;
    }
};

// The block sums are handed out in kMailboxes copies: 128 blocks polling one
// copy delay the stores to it (7.3k cycles per exchange; 2.9k with 16).
constexpr int kMailboxes = 16;
constexpr int kSlotWords = 2 * kMailboxes * 2 * kChunkBlocks;

// A form of the solve: cells per thread in a cluster, or one of these.
enum : int { CG_CHUNKS = 0, CG_GRID = -1 };

// Blocks of the cluster form.
FFR_HD constexpr int cluster_blocks(int n, int K) { return (n + K * kResThreads - 1) / (K * kResThreads); }

// smem: bytes of shared memory a block may have; pair: a direction array
// follows the other in memory; placeable(K, blocks): the device holds a
// cluster of `blocks` blocks of the form with K cells per thread.
//
// The smallest number of cells per thread that fits a cluster.  Per iteration
// with 1, 2, 4 and 8 cells per thread: 6 000 cells 1.8, 2.0, 2.7, 4.1 us;
// 11.6 k -, 2.3, 3.0, 4.4; 25.7 k -, -, 3.2, 4.5; 50 k 5.0 with 8.  The grid form
// takes 5.9 to 6.3 us at any size on 128 SMs instead of 16, k_cg 11 to 15 us.
template <class Place>
int cg_form(int nx, int ny, int nz, int smem, int sms, bool pair, Place placeable)
{
    const int n = nx * ny * nz;
    for (int K : {1, 2, 4, 8}) {
        const int blocks = cluster_blocks(n, K);
        if (blocks <= kResClusterCtas && (long long)ny * nz < smem &&
            8ll * ClusterLayout(K, nx, ny, nz).total <= smem && placeable(K, blocks))
            return K;
    }
    // r's words (16 bytes per cell) take both direction arrays, the slots A.ad
    if ((n + kResGroup - 1) / kResGroup <= kChunkMaxParts && sms >= kChunkBlocks && pair && n > kSlotWords &&
        nz < smem / 128 && 8 * ChunkLayout(nz).total <= smem)
        return CG_CHUNKS;
    return CG_GRID;
}

// ------------------------- coarse levels of the split solve (mgpcg.cu)

// One cluster: the largest of 16 and 8 blocks (16 needs the non-portable
// cluster size) that the device can place; onchip: also with the levels in its
// shared memory.  placeable(onchip, ctas) asks for either kernel.
struct MidForm {
    int ctas;
    bool onchip;
};
template <class Place> MidForm mid_form(Place placeable)
{
    for (int ctas : {16, 8})
        if (placeable(false, ctas)) return {ctas, placeable(true, ctas)};
    return {1, placeable(true, 1)};
}

}  // namespace ffr
