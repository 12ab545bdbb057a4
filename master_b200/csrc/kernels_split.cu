// Split-precision instantiation of the DSMC kernels: int voxel index + fp32
// in-voxel offset, fp32 velocities, fp64 cell bookkeeping and tallies.
#define DSMC_PREC Split32
#define DSMC_PREC_NS split32
#include <algorithm>
#include "kernels_impl.cuh"

#include "split_pass.cuh"

namespace dsmc {
namespace split32 {

// Cells per chunk for a persistent grid of `warps` warps taking chunks at a
// fixed stride: 32 (one table row or lane per cell) gives some warps one chunk
// more than the rest, and none to most of them when there are few cells, so
// the chunk is cut until every warp has the same number of them.  us per step
// at 32 and as cut, collide / move / place / sample: 64^3 (2.2e4 cells, chunks
// of 7 to 10) 18.8 / 28.8 / 12.7 -> 18.5 / 16.9 / 10.9; 128^3 (1.8e5) 51 / 101
// / 33 / 166 -> 50 / 83 / 31 / 122; at 256^3 every warp has ten or more chunks
// of 32 and it changes nothing.
static PassParams with_chunk(const PassParams &P, long long warps) {
    PassParams Q = P;
    const long long C = P.cells.num_cells;
    const long long rounds = std::max(1ll, (C + 32 * warps - 1) / (32 * warps));
    Q.chunk = (int)std::max(1ll, (C + rounds * warps - 1) / (rounds * warps));
    return Q;
}

// The production pass (split_pass.cuh): collide_cells, move_cells with the
// smallest ring that holds the largest cell, place_movers, and place_walls
// where place_movers lists its wall flights.
template <int R> static cudaError_t launch_move_ring(const PassParams &P, int grid, cudaStream_t st) {
    pass3::move_cells_kernel<R><<<grid, 32 * pass3::M_WARPS, pass3::move_smem_bytes<R>(), st>>>(
        with_chunk(P, (long long)grid * pass3::M_WARPS));
    return cudaGetLastError();
}
template <int R> static int move_ring_blocks() {
    const size_t smem = pass3::move_smem_bytes<R>();
    // the opt-in limit is a property of the function, shared by every
    // context: raise it to the device maximum, never lower it
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, pass3::move_cells_kernel<R>) != cudaSuccess) return 0;
    if (smem + fa.sharedSizeBytes > (size_t)optin) return 0;
    if (cudaFuncSetAttribute(pass3::move_cells_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - (int)fa.sharedSizeBytes) != cudaSuccess)
        return 0;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, pass3::move_cells_kernel<R>, 32 * pass3::M_WARPS,
                                                      smem) != cudaSuccess)
        return 0;
    return nb;
}
template <class K> static int static_blocks(K kernel, int threads) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, 0) != cudaSuccess) return 0;
    return nb;
}

// Records of the groups that move_cells' warps stage, for cells of at most
// `smem_cap` slots (128 at least)
// (0: no ring is large enough, or a cell could exceed the collide batch).
int fused_capacity(int smem_cap) {
    static const int rings[] = {128, 160, 192, 224, 256, 320, 384, 448, 512};
    if (smem_cap > pass3::PCAP) return 0;
    for (int r : rings)
        if (smem_cap <= r) return r;
    return 0;
}

int ring_for(int smem_cap, int ring) {
    static const int rings[] = {128, 160, 192, 224, 256, 320, 384, 448, 512};
    const int need = fused_capacity(smem_cap);
    if (need <= 0) return 0;
    const int want = std::max(need, ring);
    for (int r : rings)
        if (want <= r) return r;
    return 0;
}

int max_ring() { return 512; }

int fused_block() { return 32 * pass3::M_WARPS; }

#define DSMC_MOVE_RINGS(X) X(128) X(160) X(192) X(224) X(256) X(320) X(384) X(448) X(512)

int fused_grids(int smem_cap, int num_sms, int grids[5], int ring, int max_bps[5]) {
    int bm = 0;
    switch (ring_for(smem_cap, ring)) {
#define X(r) \
    case r: bm = move_ring_blocks<r>(); break;
        DSMC_MOVE_RINGS(X)
#undef X
    }
    const int bc = std::min(static_blocks(pass3::collide_cells_kernel<false>, 32 * pass3::C_WARPS),
                            static_blocks(pass3::collide_cells_kernel<true>, 32 * pass3::C_WARPS));
    const int bp = static_blocks(pass3::place_movers_kernel<false>, 32 * pass3::P_WARPS);
    const int bw = static_blocks(pass3::place_walls_kernel, 32 * pass3::W_WARPS);
    const int bs = static_blocks(pass3::sample_cells_kernel, 32 * pass3::C_WARPS);
    if (bm <= 0 || bc <= 0 || bp <= 0 || bw <= 0 || bs <= 0) return 0;
    grids[0] = bc * num_sms;
    grids[1] = bm * num_sms;
    grids[2] = bp * num_sms;
    grids[3] = bw * num_sms;
    grids[4] = bs * num_sms;
    if (max_bps) {
        max_bps[0] = bc;
        max_bps[1] = bm;
        max_bps[2] = bp;
        max_bps[3] = bw;
        max_bps[4] = bs;
    }
    return 1;
}

// collide_cells with the chunk counter when each warp has many chunks
static void launch_collide_cells(const PassParams &P0, int grid, cudaStream_t st) {
    PassParams P = with_chunk(P0, (long long)grid * pass3::C_WARPS);
    const long long nchunks = (P.cells.num_cells + 31) / 32;
    const bool counter = P.claim == 2 ||
                         (P.claim == 0 && nchunks >= (long long)pass3::CLAIM_MIN_CHUNKS_PER_WARP * grid * pass3::C_WARPS);
    if (counter) P.chunk = 32;
    if (counter)
        pass3::collide_cells_kernel<true><<<grid, 32 * pass3::C_WARPS, 0, st>>>(P);
    else
        pass3::collide_cells_kernel<false><<<grid, 32 * pass3::C_WARPS, 0, st>>>(P);
}

// place_movers' blocks when its warps move their own wall flights: half the
// blocks of the listing kernel fit
static int own_walls_grid(const int grids[5]) { return std::max(1, grids[2] / 2); }

// They do up to four chunks of 32 cells per warp (place_movers_kernel's comment).
bool own_walls(int num_cells, int any_cl, const int grids[5]) {
    return !any_cl && num_cells <= 4ll * 32 * own_walls_grid(grids) * pass3::P_WARPS;
}

cudaError_t launch_fused(const PassParams &P, const int grids[5], cudaStream_t st, cudaEvent_t *ev) {
    if (ev) cudaEventRecord(ev[0], st);
    if (P.do_collide || P.do_sample) {
        launch_collide_cells(P, grids[0], st);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (P.do_sample) {  // sampled steps only: the host knows the cadence
            pass3::sample_cells_kernel<<<grids[4], 32 * pass3::C_WARPS, 0, st>>>(
                with_chunk(P, (long long)grids[4] * pass3::C_WARPS));
            e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
    }
    if (ev) cudaEventRecord(ev[1], st);
    cudaError_t e = cudaErrorInvalidValue;
    switch (ring_for(P.smem_cap, P.ring)) {
#define X(r) \
    case r: e = launch_move_ring<r>(P, grids[1], st); break;
        DSMC_MOVE_RINGS(X)
#undef X
    }
    if (e != cudaSuccess) return e;
    if (ev) cudaEventRecord(ev[2], st);
    if (own_walls(P.cells.num_cells, P.any_cl, grids)) {
        const int own_grid = own_walls_grid(grids);
        pass3::place_movers_kernel<true><<<own_grid, 32 * pass3::P_WARPS, 0, st>>>(
            with_chunk(P, (long long)own_grid * pass3::P_WARPS));
        e = cudaGetLastError();
        if (ev) cudaEventRecord(ev[3], st);
    } else {
        pass3::place_movers_kernel<false><<<grids[2], 32 * pass3::P_WARPS, 0, st>>>(
            with_chunk(P, (long long)grids[2] * pass3::P_WARPS));
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (ev) cudaEventRecord(ev[3], st);
        pass3::place_walls_kernel<<<grids[3], 32 * pass3::W_WARPS, 0, st>>>(P);
        e = cudaGetLastError();
    }
    if (ev) cudaEventRecord(ev[4], st);
    return e;
}

cudaError_t launch_collide(const PassParams &P, const int grids[5], cudaStream_t st) {
    launch_collide_cells(P, grids[0], st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (P.do_sample) {
        pass3::sample_cells_kernel<<<grids[4], 32 * pass3::C_WARPS, 0, st>>>(
                with_chunk(P, (long long)grids[4] * pass3::C_WARPS));
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    // place_walls, whose last block zeroes collide_cells' chunk counter at the
    // end of a full pass, does not run here
    return cudaMemsetAsync(&P.status->collide_taken, 0, sizeof(unsigned), st);
}

cudaError_t launch_put(const SysDev *sys, int s, const CellArrays &cells, const ParticleArrays &parts, int cur, int cin,
                       long long n, const uint4 *rec, Status *status, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int grid = (int)std::min<long long>((n + 255) / 256, 148LL * 8);
    pass3::put_records_kernel<<<grid, 256, 0, st>>>(sys, s, cells, parts, cur, cin, n, rec, status);
    return cudaGetLastError();
}

}  // namespace split32
}  // namespace dsmc
