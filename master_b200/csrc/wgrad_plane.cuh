// Weight gradient of the 3x3x3 periodic convolution for edges of 8 and more,
// on tcgen05.mma with the planes of both operands staged once per tile: the
// tiles, the staging and the roles of conv_plane.cuh.
//
// Measured (batch 8, back to back), wgrad_kernel of surrogate.cu before and
// this kernel: 64^3 48 -> 16 channels 1154 -> 181 us (42 us for its bytes),
// 64^3 16 -> 16 615 -> 77 us (21 us), 32^3 96 -> 32 270 -> 66 us, 16^3
// 64 -> 64 106 -> 20 us.  Before, every voxel of dY was read from L2 once per
// tap; now shared memory feeding the MMAs bounds it (46 cycles for M = 128 and
// N = 48, 30 for M = 64, of which 24 would be the tensor pipe's at full rate).
#pragma once
#include "conv_plane.cuh"

namespace sg {

struct PlaneWgradArgs {
    const bf16 *dy;
    int dy_cs, dy_coff;  // (coff: of the call's first channel)
    const bf16 *x;
    int x_cs, x_coff;
    float *dw;           // [cout][27][cin], accumulated
    int cin;             // row length of dw
    int ci0;             // first input channel of this launch
    int ciblocks;        // blocks of CIB input channels of this launch
    int cob;             // output channels per CTA: 16, 32 or 48
    int coblocks;        // cout / cob
    int S, lg, lgL;
    int items;
    int flush;           // planes between two flushes of the accumulators
    int batch;
};

// PAIR (edge 8): a tile is the whole planes of two samples, the second one's
// lines behind the first's. wgrad_kernel and this kernel, us: 1 sample of 16 -> 16
// channels 11.6 -> 6.2, 64 -> 64 17.9 -> 8.8; 16 of 96 -> 32 23 -> 9.7; 64 of 64 -> 64
// 104 -> 20.5, 96 -> 96 123 -> 32.
template <int CIB, bool PAIR> struct PlaneWgradShape {
    static constexpr int kHLines = PAIR ? 20 : kLines + 2;
    static constexpr int kHalo = kHLines * kHRow;
    static constexpr int kCpt = CIB / 8;
    static constexpr int kLine = kCpt * kHRow * 16;   // staged bytes of a line of X: [chunk][10 voxels]
    static constexpr int kX = kHLines * kLine;
    static constexpr int kPad = 2048;                 // the last lines' unused row groups read past X
    static constexpr int kXLoads = (kHalo * kCpt + 32 * kLoadWarps - 1) / (32 * kLoadWarps);
    static constexpr int kSlots = CIB == 16 ? 12 : 8; // planes in flight
    static constexpr int kPairs = kSlots / 2;         // two planes share a barrier (see PlaneShape::kGroup)
    static constexpr int kBars = 2 * kPairs + 4;
    static constexpr int kM = CIB == 16 ? 64 : 128;   // rows: 3 x CIB and unused ones
    static constexpr int smem(int cob) { return kSlots * (kX + kLines * cob * 16) + kPad + kBars * 8 + 16; }
};

// dW[co][t][ci] = sum_v dY[v][co] X[v + off(t)][ci]: the voxels of a plane of
// the tile are K (8 steps of two lines), both operands MN-major.  A's rows
// are (axis-1 tap, input channel): a line of X is staged [chunk][voxel], so
// the next tap's chunks follow at the same distance and M = 64 (CIB = 16) or
// 128 holds the 3 x CIB of them (the rest is not used); B's columns are three planes of dY (the
// axis-0 taps) x cob; the axis-2 taps are three start addresses of A with an
// accumulator each.  The accumulators are added to dW every `flush` planes.
template <int CIB, bool PAIR>
__global__ void __launch_bounds__(kPlaneThreads, 1) wgrad_plane_kernel(const __grid_constant__ PlaneWgradArgs a) {
    using Sh = PlaneWgradShape<CIB, PAIR>;
    constexpr int kHalo = Sh::kHalo;
    extern __shared__ __align__(128) unsigned char smem[];
    const int cob = a.cob, cpy = cob >> 3;
    const int ystep = cpy * 128;              // bytes of one slot in a line of dY: [slot][chunk][8 voxels]
    const int yline = Sh::kSlots * ystep;
    unsigned char *Ys = smem + Sh::kSlots * Sh::kX + Sh::kPad;
    uint64_t *full = reinterpret_cast<uint64_t *>(Ys + kLines * yline);
    uint64_t *empty = full + Sh::kPairs;
    uint64_t *accfull = empty + Sh::kPairs;   // [2]
    uint64_t *accfree = accfull + 2;          // [2]
    uint32_t *tslot = reinterpret_cast<uint32_t *>(accfree + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int groups = a.ciblocks * a.coblocks;
    const int group = (int)blockIdx.x % groups;
    const int first = (int)blockIdx.x / groups, stride = (int)gridDim.x / groups;
    const int ci0 = a.ci0 + (group % a.ciblocks) * CIB, co0 = (group / a.ciblocks) * cob;
    const int lg = a.lg, lg2 = 2 * lg, lg3 = 3 * lg, msk = a.S - 1;
    const int L = 1 << a.lgL;
    const int ncol = 9 * cob;                 // accumulator columns of an item
    const int nacc = 2 * ncol <= (int)kTmemCols ? 2 : 1;

    if (warp == kEpiWarps + kLoadWarps) {
        tc05::tmem_alloc(tslot, kTmemCols);
        tc05::tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < Sh::kPairs; ++s) {
            tc05::mbar_init(&full[s], 32 * kLoadWarps);
            tc05::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            tc05::mbar_init(&accfull[s], 1);
            tc05::mbar_init(&accfree[s], kEpiWarps);
        }
        tc05::mbar_fence_init();
    }
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    const uint32_t tmem = *tslot;

    if (warp >= kEpiWarps && warp < kEpiWarps + kLoadWarps) {
        const int lt = tid - 32 * kEpiWarps;
        int s = 0, n = 0;
        uint32_t ph = 0;
        bool ok = true;
        const int ym = lt >> 3, yx = lt & 7;  // this thread's voxel of dY
        for (int item = first; item < a.items; item += stride) {
            const PlaneItem p = PAIR ? pair_item(item, lg, a.lgL) : plane_item(item, lg, a.lgL);
            // PAIR: an odd batch's last tile has one sample, its other lines are zero
            const bool two = !PAIR || p.b + 1 < a.batch;
            int off[Sh::kXLoads];
#pragma unroll
            for (int i = 0; i < Sh::kXLoads; ++i) {
                const int idx = lt + 32 * kLoadWarps * i;
                const int r = idx / Sh::kCpt, c = idx - r * Sh::kCpt;
                const int line = r / kHRow, x = r - line * kHRow;
                const int second = PAIR && two && line >= 10 ? 1 << lg3 : 0;
                const int l1 = PAIR && line >= 10 ? line - 10 : line;
                off[i] = (second + (((p.x1 - 1 + l1) & msk) << lg) + ((p.x2 - 1 + x) & msk)) * a.x_cs + a.x_coff + ci0 + c * 8;
            }
            const int yv = PAIR ? (two ? (ym >> 3) << lg3 : 0) + ((ym & 7) << lg) + yx : ((p.x1 + ym) << lg) + p.x2 + yx;
            const int yoff = yv * a.dy_cs + a.dy_coff + co0;
            const uint32_t ybytes = two || ym < 8 ? 16u : 0u;
            for (int u = 0; u < L + 2; ++u) {  // unit u: planes z0 - 1 + u of dY and, inside the item, of X
                if (!(u & 1) && n >= Sh::kSlots) ok &= tc05::mbar_wait(&empty[s >> 1], ph ^ 1u);
                const long long plane = ((long long)p.b << lg3) + ((long long)((p.z0 - 1 + u) & msk) << lg2);
                const bf16 *py = a.dy + plane * a.dy_cs + yoff;
                unsigned char *yd = Ys + ym * yline + s * ystep + yx * 16;
                for (int c = 0; c < cpy; ++c) {
                    if (PAIR) tc05::cp_async16_zfill(yd + c * 128, py + c * 8, ybytes);
                    else tc05::cp_async16(yd + c * 128, py + c * 8);
                }
                if (u >= 1 && u <= L) {
                    const bf16 *px = a.x + plane * a.x_cs;
                    unsigned char *xd = smem + s * Sh::kX;
#pragma unroll
                    for (int i = 0; i < Sh::kXLoads; ++i) {
                        const int idx = lt + 32 * kLoadWarps * i;
                        if (idx < kHalo * Sh::kCpt) {
                            const int r = idx / Sh::kCpt, c = idx - r * Sh::kCpt;
                            const int line = r / kHRow, x = r - line * kHRow;
                            unsigned char *to = xd + line * Sh::kLine + c * (kHRow * 16) + x * 16;
                            if (PAIR) tc05::cp_async16_zfill(to, px + off[i], two || line < 10 ? 16u : 0u);
                            else tc05::cp_async16(to, px + off[i]);
                        }
                    }
                }
                if (u & 1) tc05::cp_async_arrive(&full[s >> 1]);
                ++n;
                if (++s == Sh::kSlots) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        tc05::cp_async_wait_all();
        if (!ok) atomicOr(&g_error, 2u);
    } else if (warp == kEpiWarps + kLoadWarps) {
        const uint32_t lead = tc05::elect_one();
        const uint64_t adesc = tc05::desc_noswizzle(tc05::smem_u32(smem), Sh::kLine, kHRow * 16);
        const uint64_t bdesc = tc05::desc_noswizzle(tc05::smem_u32(Ys), yline, 128);
        const uint32_t ahi = (uint32_t)(adesc >> 32), bhi = (uint32_t)(bdesc >> 32);
        const uint32_t alo0 = (uint32_t)adesc, blo0 = (uint32_t)bdesc;
        auto idesc = [&](int planes) { return tc05::idesc_bf16_f32(Sh::kM, planes * cob, 1, 1); };
        int s = 0;          // slot of the newest plane waited for
        uint32_t ph = 0;
        int acc = 0, flushes = 0, since = 0;  // accumulator; flushes so far; planes since the last
        uint32_t aph = 0;
        bool ok = true;
        auto prev = [&](int q, int d) { return q >= d ? q - d : q - d + Sh::kSlots; };
        for (int item = first; item < a.items; item += stride) {
            for (int u = 0; u < L + 2; ++u) {
                if (!(u & 1)) {
                    ok &= tc05::mbar_wait(&full[s >> 1], ph);
                    tc05::fence_proxy_async_smem();
                    tc05::fence_after_sync();
                }
                if (u >= 2) {
                    // plane u - 1 of X against planes u - 2 .. u of dY
                    const bool start = since == 0;
                    const bool last = ++since == a.flush || (u == L + 1 && item + stride >= a.items);
                    if (start && flushes >= nacc) ok &= tc05::mbar_wait(&accfree[acc], aph ^ 1u);
                    tc05::fence_after_sync();
                    const int y0 = prev(s, 2), xs = prev(s, 1);
                    const int n0 = min(3, Sh::kSlots - y0), n1 = 3 - n0;
                    const uint32_t i0 = idesc(n0), i1 = idesc(n1);
                    const uint32_t col = tmem + acc * ncol;
                    const uint32_t alo = alo0 + (uint32_t)((xs * Sh::kX) >> 4);
                    const uint32_t blo = blo0 + (uint32_t)((y0 * ystep) >> 4);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {
                        const uint32_t ys = (uint32_t)((2 * kk * yline) >> 4);
                        const uint32_t add = kk > 0 || !start ? 1u : 0u;
#pragma unroll
                        for (int t2 = 0; t2 < 3; ++t2) {
                            const uint32_t ad = alo + (uint32_t)(((2 * kk + (PAIR && kk >= 4 ? 2 : 0)) * Sh::kLine) >> 4) + (uint32_t)t2;
                            tc05::mma_bf16_warp(lead, col + t2 * 3 * cob, ad, ahi, blo + ys, bhi, i0, add);
                            if (n1 > 0)
                                tc05::mma_bf16_warp(lead, col + (t2 * 3 + n0) * cob, ad, ahi, blo0 + ys, bhi, i1, add);
                        }
                    }
                    // (L is even: planes go in pairs) the pair u - 3, u - 2 has served its last step
                    if (u & 1) tc05::mma_commit_warp(lead, &empty[prev(s, 3) >> 1]);
                    if (u == L + 1) tc05::mma_commit_warp(lead, &empty[s >> 1]);
                    if (last) {
                        tc05::mma_commit_warp(lead, &accfull[acc]);
                        since = 0;
                        ++flushes;
                        if (++acc == nacc) {
                            acc = 0;
                            aph ^= 1u;
                        }
                    }
                }
                if (++s == Sh::kSlots) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        if (!ok && lead) atomicOr(&g_error, 2u);
    } else {
        // ---- flush: row m = (axis-1 tap, input channel), 32 lanes 32 of them
        const int quarter = warp & 3, half = warp >> 2;
        // (M = 64 fills lanes 0-15 of each quarter)
        const int m = Sh::kM == 64 ? quarter * 16 + (lane & 15) : quarter * 32 + lane;
        const bool row = Sh::kM == 128 || lane < 16;
        const int g = m >> 3, t1 = g / Sh::kCpt, ci = (g - t1 * Sh::kCpt) * 8 + (m & 7);
        int acc = 0;
        uint32_t aph = 0;
        bool ok = true;
        // this CTA's planes, `flush` at a time
        for (long long planes = (long long)((a.items - first + stride - 1) / stride) << a.lgL; planes > 0; planes -= a.flush) {
            ok &= tc05::mbar_wait(&accfull[acc], aph);
            tc05::fence_after_sync();
            const uint32_t col = tmem + ((uint32_t)(quarter * 32) << 16) + acc * ncol;
            for (int c0 = 16 * half; c0 < ncol; c0 += 32) {
                float v[16];
                tc05::tmem_ld16(col + c0, v);
                // column = (axis-2 tap, plane of dY, output channel): 16 columns share their taps
                const int t2 = c0 / (3 * cob), j = (c0 / cob) % 3, co = co0 + c0 % cob;
                if (row && t1 < 3) {
                    float *d = a.dw + ((long long)co * 27 + (2 - j) * 9 + t1 * 3 + t2) * a.cin + ci0 + ci;
#pragma unroll
                    for (int i = 0; i < 16; ++i) atomicAdd(d + (long long)i * 27 * a.cin, v[i]);
                }
            }
            tc05::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc05::mbar_arrive(&accfree[acc]);
            if (++acc == nacc) {
                acc = 0;
                aph ^= 1u;
            }
        }
        if (!ok) atomicOr(&g_error, 2u);
    }
    __syncwarp();
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    if (warp == kEpiWarps + kLoadWarps) tc05::tmem_dealloc(tmem, kTmemCols);
}

}  // namespace sg
