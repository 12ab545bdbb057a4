// 3x3x3 periodic convolution for edges of 8 and more, on tcgen05.mma with
// each input plane staged once per tile.
//
// A CTA walks tiles of 16 x 8 voxels (axes 1 and 2: the 128 rows of an MMA)
// along axis 0.  A plane of the tile with its one-voxel halo, 18 x 10 voxels,
// is staged in the no-swizzle layout, whose rows are 16 bytes apart: the
// operand of each of the nine in-plane taps is then the same plane from
// another start address (the groups of 8 rows are the tile's lines, one staged
// line apart), so a voxel is read from L2 1.4 times per tile and not once per
// tap.
//
// The three taps along axis 0 are the N dimension: plane z adds to output
// planes z - 1, z and z + 1, which lie side by side in tensor memory
// (N = 3 x output channels).  The bound is shared memory feeding the MMAs: one
// of M = 128 and K = 16 takes 34 + N / 4 cycles here (measured for N <= 128;
// 4 KB of A and 32 N bytes of B at 128 bytes a cycle), so at 16 output
// channels one of N = 48 does in 46 cycles what three of N = 16 do in 114.
//
// Measured (batch 8, back to back), conv3_kernel of surrogate.cu before and
// this kernel: 64^3 48 -> 16 channels 2479 -> 127 us (0.69 PFLOP/s; 53 us at
// the measured cuBLAS rate, 42 us for its bytes), 64^3 16 -> 16 860 -> 64 us
// (21 us for its bytes), 32^3 96 -> 32 653 -> 62 us, 16^3 64 -> 64 78 -> 19
// us.  The one-tap-at-a-time gather was bound by its 27 reads of every voxel
// from L2.  Timed without its loads and its epilogue the 64^3 16 -> 16 kernel
// still takes 57 of 64 us, without the MMAs 33: in the kernel an MMA of N = 48
// takes about 60 cycles.  Two CTAs per SM (half the TMEM columns and epilogue warps
// each) ran that forward in 58 us but its gradient in 79 for 74, 64^3 48 -> 16 in 135
// for 127 and 32^3 32 -> 32 in 30 for 24.
//
// Per output value the taps and channels are accumulated in the order tap
// 0..26, channels within a tap, as conv3_kernel (surrogate.cu) does: the two
// kernels give the same bits.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "tc05.cuh"

namespace sg {

using bf16 = __nv_bfloat16;

constexpr int kLines = 16, kRow = 8;             // voxels of a tile along axes 1 and 2
constexpr int kHLines = kLines + 2, kHRow = kRow + 2;
constexpr int kHalo = kHLines * kHRow;           // staged rows of a plane of a tile
constexpr int kEpiWarps = 8, kLoadWarps = 4;     // two warps per TMEM lane quarter; then the loaders, then the issuer
constexpr int kPlaneThreads = 32 * (kEpiWarps + kLoadWarps + 1);
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxSlots = 32;

// A tile of the walk: sample, tile origin in the plane, first plane.
struct PlaneItem {
    int b, x1, x2, z0;
};
__device__ __forceinline__ PlaneItem plane_item(int item, int lg, int lgL) {
    PlaneItem p;
    const int n2 = lg - 3, n1 = lg - 4, nz = lg - lgL;  // log2 of the tiles per axis
    p.x2 = (item & ((1 << n2) - 1)) << 3;
    item >>= n2;
    p.x1 = (item & ((1 << n1) - 1)) << 4;
    item >>= n1;
    p.z0 = (item & ((1 << nz) - 1)) << lgL;
    p.b = item >> nz;
    return p;
}

// The same for pairs of samples (edge 8).
__device__ __forceinline__ PlaneItem pair_item(int item, int lg, int lgL) {
    const int nz = lg - lgL;
    return PlaneItem{(item >> nz) << 1, 0, 0, (item & ((1 << nz) - 1)) << lgL};
}

// ---- forward (and input gradient) --------------------------------------------

struct PlaneArgs {
    const bf16 *in;
    int in_cs, in_coff;
    const bf16 *w;      // [cout][27][CIN]
    const float *bias;  // [cout] or null
    bf16 *out;
    int out_cs, out_coff;
    const bf16 *mask;   // multiply by (mask > 0), or null
    int mask_cs, mask_coff;
    int relu;
    int S, lg, lgL;     // edge, log2(edge), log2(planes per item)
    int nb;             // output channels per CTA
    int nsplit;         // CTAs per item: cout / nb
    int items;          // tiles x plane segments
    int batch;
};

// PAIR (edge 8): a tile is the whole planes of two samples, their lines
// interleaved (the second sample's a line after the first's, so the groups of 8
// rows stay one staged line apart and a tap along axis 1 is two lines). conv3_kernel
// and this kernel, us, forward: 1 sample of 16 -> 16 channels 9.9 -> 5.7, 64 -> 64 38
// -> 10; 16 of 96 -> 32 49 -> 14.5; 64 of 64 -> 64 77 -> 19.5, 96 -> 96 124 -> 37.
template <int CIN, bool PAIR> struct PlaneShape {
    static constexpr int kLineStep = PAIR ? 2 : 1;
    static constexpr int kHalo = (kLines + 2 * kLineStep) * kHRow;  // staged rows of a plane
    static constexpr int kCpt = CIN / 8;                        // 16-byte channel chunks
    static constexpr int kChunk = kHalo * 16 + 16;              // bytes between chunks (odd in 16 bytes: no bank conflicts)
    static constexpr int kPlane = kCpt * kChunk;
    // planes per barrier: a wait costs the issuer about 100 cycles of the
    // tensor pipe (nothing is queued behind an MMA that could start), as much
    // as two or three MMAs, so planes of few MMAs share one
    static constexpr int kGroup = CIN <= 32 ? 3 : CIN == 48 ? 2 : 1;
    static constexpr int kGroups = CIN == 16 ? 4 : CIN <= 48 || (CIN == 96 && PAIR) ? 3 : 4;
    static constexpr int kStages = kGroup * kGroups;            // planes in flight
    static constexpr int kLoads = (kHalo * kCpt + 32 * kLoadWarps - 1) / (32 * kLoadWarps);
    static constexpr int kBars = 2 * kGroups + kMaxSlots + 2;
    // the largest nb whose weights fit beside the planes
    static constexpr int kMaxNb = CIN <= 32 ? 48 : CIN <= 64 ? 32 : 16;
    static constexpr int smem(int nb) { return kStages * kPlane + 27 * CIN * nb * 2 + kBars * 8 + 48 * 4 + 16; }
};

// Roles: warps 0-7 epilogue, 8-11 load planes, 12 issues the MMAs.  Every
// wait is bounded (a wait that runs out sets bit 0 of the error flags).
template <int CIN, bool PAIR>
__global__ void __launch_bounds__(kPlaneThreads, 1) conv_plane_kernel(const __grid_constant__ PlaneArgs a) {
    using Sh = PlaneShape<CIN, PAIR>;
    constexpr int kHalo = Sh::kHalo;
    extern __shared__ __align__(128) unsigned char smem[];
    const int nb = a.nb, nb3 = 3 * nb;
    unsigned char *Ws = smem + Sh::kStages * Sh::kPlane;
    uint64_t *full = reinterpret_cast<uint64_t *>(Ws + 27 * CIN * nb * 2);
    uint64_t *empty = full + Sh::kGroups;
    uint64_t *accfull = empty + Sh::kGroups;  // per accumulator plane
    uint64_t *accfree = accfull + kMaxSlots;  // per half of them
    float *bias = reinterpret_cast<float *>(accfree + 2);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bias + 48);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = (int)blockIdx.x % a.nsplit;
    const int first = (int)blockIdx.x / a.nsplit, stride = (int)gridDim.x / a.nsplit;
    const int co0 = split * nb;
    const int lg = a.lg, lg2 = 2 * lg, lg3 = 3 * lg, msk = a.S - 1;
    const int L = 1 << a.lgL;
    const int R = (int)kTmemCols / nb, H = R / 2;  // accumulator planes (32, 16 or 10) and half of them

    if (warp == kEpiWarps + kLoadWarps) {
        tc05::tmem_alloc(tslot, kTmemCols);
        tc05::tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < Sh::kGroups; ++s) {
            tc05::mbar_init(&full[s], 32 * kLoadWarps);
            tc05::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < kMaxSlots; ++s) tc05::mbar_init(&accfull[s], 1);
        for (int s = 0; s < 2; ++s) tc05::mbar_init(&accfree[s], 4 * H);
        tc05::mbar_fence_init();
    }
    if (tid < nb) bias[tid] = a.bias ? a.bias[co0 + tid] : 0.0f;
    // weights, K-major: row j * nb + co holds tap plane 2 - j (the block of
    // output plane z - 1 + j), 16-byte K chunks nb3 rows apart
    for (int i = tid; i < 9 * Sh::kCpt * nb3; i += kPlaneThreads) {
        const int c = i % Sh::kCpt, r = i / Sh::kCpt;
        const int t12 = r % 9, n = r / 9;
        const int j = n / nb, co = n - j * nb;
        const bf16 *src = a.w + ((long long)(co0 + co) * 27 + (2 - j) * 9 + t12) * CIN + c * 8;
        tc05::cp_async16(Ws + ((t12 * Sh::kCpt + c) * nb3 + n) * 16, src);
    }
    tc05::cp_async_commit();
    tc05::cp_async_wait<0>();
    tc05::fence_proxy_async_smem();
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    const uint32_t tmem = *tslot;

    if (warp >= kEpiWarps && warp < kEpiWarps + kLoadWarps) {
        // ---- loaders: one 16-byte copy per thread, row and chunk
        const int lt = tid - 32 * kEpiWarps;
        int s = 0, in_g = 0;  // group; plane in it
        uint32_t ph = 0;      // parity of the group's round
        bool lapped = false;  // every group has been filled once
        bool ok = true;
        for (int item = first; item < a.items; item += stride) {
            const PlaneItem p = PAIR ? pair_item(item, lg, a.lgL) : plane_item(item, lg, a.lgL);
            int off[Sh::kLoads];
#pragma unroll
            for (int i = 0; i < Sh::kLoads; ++i) {
                const int idx = lt + 32 * kLoadWarps * i;
                const int r = idx / Sh::kCpt, c = idx - r * Sh::kCpt;
                const int line = r / kHRow, x = r - line * kHRow;
                // (the last sample of an odd batch is its own pair)
                const int second = PAIR && p.b + 1 < a.batch ? (line & 1) << lg3 : 0;
                const int l1 = PAIR ? (line >> 1) - 1 : p.x1 - 1 + line;
                off[i] = (second + ((l1 & msk) << lg) + ((p.x2 - 1 + x) & msk)) * a.in_cs + a.in_coff + c * 8;
            }
            for (int z = p.z0 - 1; z <= p.z0 + L; ++z) {
                if (in_g == 0 && lapped) ok &= tc05::mbar_wait(&empty[s], ph ^ 1u);
                const bf16 *pl = a.in + (((long long)p.b << lg3) + ((long long)(z & msk) << lg2)) * a.in_cs;
                unsigned char *st = smem + (s * Sh::kGroup + in_g) * Sh::kPlane;
#pragma unroll
                for (int i = 0; i < Sh::kLoads; ++i) {
                    const int idx = lt + 32 * kLoadWarps * i;
                    if (idx < kHalo * Sh::kCpt) {
                        const int r = idx / Sh::kCpt, c = idx - r * Sh::kCpt;
                        tc05::cp_async16(st + c * Sh::kChunk + r * 16, pl + off[i]);
                    }
                }
                if (++in_g == Sh::kGroup || z == p.z0 + L) {
                    tc05::cp_async_arrive(&full[s]);
                    in_g = 0;
                    if (++s == Sh::kGroups) {
                        s = 0;
                        ph ^= 1u;
                        lapped = true;
                    }
                }
            }
        }
        tc05::cp_async_wait_all();
        if (!ok) atomicOr(&g_error, 1u);
    } else if (warp == kEpiWarps + kLoadWarps) {
        // ---- the issuer: the whole warp in step, one lane's MMAs
        const uint32_t lead = tc05::elect_one();
        const uint64_t adesc = tc05::desc_noswizzle(tc05::smem_u32(smem), Sh::kChunk, kHRow * 16);
        const uint64_t bdesc = tc05::desc_noswizzle(tc05::smem_u32(Ws), nb3 * 16, 128);
        const uint32_t ahi = (uint32_t)(adesc >> 32), bhi = (uint32_t)(bdesc >> 32);
        const uint32_t alo0 = (uint32_t)adesc, blo0 = (uint32_t)bdesc;
        auto idesc = [&](int blocks) { return tc05::idesc_bf16_f32(128, blocks * nb, 0, 0); };
        int s = 0, in_g = 0;    // group and plane in it
        int slot0 = 0;          // slot of the item's first output plane
        uint32_t ph = 0;        // parity of `full`
        uint32_t use = 0;       // parity of the slots' current use, toggled at each wrap
        bool lapped = false;    // the slots have been used before
        bool ok = true;
        for (int item = first; item < a.items; item += stride) {
            int slot = slot0;   // slot of output plane `zi` (the newest block)
            for (int zi = 0; zi < L + 2; ++zi) {
                const int jb = zi < 2 ? 2 - zi : 0, je = zi < L ? 3 : L + 2 - zi;
                const bool fresh = je == 3;  // the plane's newest block starts an accumulator
                if (fresh && lapped && (slot == 0 || slot == H)) {
                    ok &= tc05::mbar_wait(&accfree[slot ? 1 : 0], use ^ 1u);
                    tc05::fence_after_sync();  // the epilogue's reads, before the MMAs that start these slots again
                }
                if (in_g == 0) {
                    ok &= tc05::mbar_wait(&full[s], ph);
                    tc05::fence_proxy_async_smem();  // the loaders' copies, for the MMAs' reads
                    tc05::fence_after_sync();
                }
                // block j accumulates in slot + j - 2, modulo R: up to two runs
                int c0 = slot + jb - 2;
                if (c0 < 0) c0 += R;
                const int n0 = min(je - jb, R - c0), n1 = je - jb - n0;
                const uint32_t d0 = tmem + c0 * nb;
                const uint32_t i0 = idesc(n0);
                const uint32_t alo = alo0 + (uint32_t)(((s * Sh::kGroup + in_g) * Sh::kPlane) >> 4);
                const uint32_t blo = blo0 + (uint32_t)(jb * nb);
                if (fresh) {  // the first MMA: the older blocks add, the newest starts
                    const int old = 2 - jb, o0 = min(old, R - c0);
                    if (old > 0) tc05::mma_bf16_warp(lead, d0, alo, ahi, blo, bhi, idesc(o0), 1u);
                    if (old > o0) tc05::mma_bf16_warp(lead, tmem, alo, ahi, blo + (uint32_t)(o0 * nb), bhi, idesc(old - o0), 1u);
                    tc05::mma_bf16_warp(lead, tmem + slot * nb, alo, ahi, blo + (uint32_t)(old * nb), bhi, idesc(1), 0u);
                }
                const int k0 = fresh ? 1 : 0;
                if (n1 == 0) {
#pragma unroll
                    for (int k = 0; k < 9 * (CIN / 16); ++k) {
                        const int t = k / (CIN / 16), c = k % (CIN / 16);
                        if (k >= k0)
                            tc05::mma_bf16_warp(lead, d0, alo + (uint32_t)((t / 3) * Sh::kLineStep * kHRow + t % 3 + ((2 * c * Sh::kChunk) >> 4)),
                                                ahi, blo + (uint32_t)((t * Sh::kCpt + 2 * c) * nb3), bhi, i0, 1u);
                    }
                } else {
                    const uint32_t i1 = idesc(n1);
                    for (int k = k0; k < 9 * (CIN / 16); ++k) {
                        const int t = k / (CIN / 16), c = k % (CIN / 16);
                        const uint32_t ad = alo + (uint32_t)((t / 3) * Sh::kLineStep * kHRow + t % 3 + ((2 * c * Sh::kChunk) >> 4));
                        const uint32_t bd = blo + (uint32_t)((t * Sh::kCpt + 2 * c) * nb3);
                        tc05::mma_bf16_warp(lead, d0, ad, ahi, bd, bhi, i0, 1u);
                        tc05::mma_bf16_warp(lead, tmem, ad, ahi, bd + (uint32_t)(n0 * nb), bhi, i1, 1u);
                    }
                }
                if (zi >= 2) {
                    int done = slot - 2;
                    if (done < 0) done += R;
                    tc05::mma_commit_warp(lead, &accfull[done]);
                }
                if (++in_g == Sh::kGroup || zi == L + 1) {
                    tc05::mma_commit_warp(lead, &empty[s]);
                    in_g = 0;
                    if (++s == Sh::kGroups) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                // (past the item's last output plane the counter runs on for
                // the older blocks; the next item goes on from its own planes)
                if (++slot == R) {
                    slot = 0;
                    if (zi < L) {
                        use ^= 1u;
                        lapped = true;
                    }
                }
            }
            slot0 += L % R;
            if (slot0 >= R) slot0 -= R;
        }
        if (!ok && lead) atomicOr(&g_error, 1u);
    } else {
        // ---- epilogue: warps 0-3 take the even output planes, 4-7 the odd ones
        const int quarter = warp & 3;
        const int m = quarter * 32 + lane, line = m >> 3, x = m & 7;
        int slot = 0, k = 0;  // of output plane k of this CTA
        uint32_t use = 0;
        bool ok = true;
        for (int item = first; item < a.items; item += stride) {
            const PlaneItem p = PAIR ? pair_item(item, lg, a.lgL) : plane_item(item, lg, a.lgL);
            const int b = PAIR ? p.b + (line & 1) : p.b, x1 = PAIR ? line >> 1 : p.x1 + line;
            const bool here = !PAIR || b < a.batch;
            const long long row0 = here ? ((long long)b << lg3) + ((long long)p.z0 << lg2) + ((long long)x1 << lg) + p.x2 + x : 0;
            for (int rel = 0; rel < L; ++rel, ++k) {
                if ((k & 1) == (warp >> 2)) {
                    const long long row = row0 + ((long long)rel << lg2);
                    bf16 *dst = a.out + row * a.out_cs + a.out_coff + co0;
                    const bf16 *mk = a.mask ? a.mask + row * a.mask_cs + a.mask_coff + co0 : nullptr;  // (row 0's where not here)
                    uint4 mw[Sh::kMaxNb / 8];  // the mask's row, in flight during the wait
                    if (mk) {
#pragma unroll
                        for (int i = 0; i < Sh::kMaxNb / 8; ++i)
                            if (8 * i < nb) mw[i] = __ldg(reinterpret_cast<const uint4 *>(mk + 8 * i));
                    }
                    ok &= tc05::mbar_wait(&accfull[slot], use);
                    tc05::fence_after_sync();
                    const uint32_t col = tmem + ((uint32_t)(quarter * 32) << 16) + slot * nb;
#pragma unroll
                    for (int c0 = 0; c0 < Sh::kMaxNb; c0 += 16) {
                        if (c0 >= nb) break;
                        float v[16];
                        tc05::tmem_ld16(col + c0, v);
                        if (a.bias) {
#pragma unroll
                            for (int i = 0; i < 16; ++i) v[i] += bias[c0 + i];
                        }
                        if (a.relu) {
#pragma unroll
                            for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.0f);
                        }
                        if (mk) {
                            const bf16 *mb0 = reinterpret_cast<const bf16 *>(&mw[c0 / 8]);
                            const bf16 *mb1 = reinterpret_cast<const bf16 *>(&mw[c0 / 8 + 1]);
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                if (!(__bfloat162float(mb0[i]) > 0.0f)) v[i] = 0.0f;
                                if (!(__bfloat162float(mb1[i]) > 0.0f)) v[8 + i] = 0.0f;
                            }
                        }
                        uint4 o0, o1;
                        __nv_bfloat162 *h0 = reinterpret_cast<__nv_bfloat162 *>(&o0);
                        __nv_bfloat162 *h1 = reinterpret_cast<__nv_bfloat162 *>(&o1);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            h0[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                            h1[i] = __floats2bfloat162_rn(v[8 + 2 * i], v[8 + 2 * i + 1]);
                        }
                        if (here) {
                            *reinterpret_cast<uint4 *>(dst + c0) = o0;
                            *reinterpret_cast<uint4 *>(dst + c0 + 8) = o1;
                        }
                    }
                    tc05::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc05::mbar_arrive(&accfree[slot >= H]);
                }
                if (++slot == R) {
                    slot = 0;
                    use ^= 1u;
                }
            }
        }
        if (!ok) atomicOr(&g_error, 1u);
    }
    __syncwarp();
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    if (warp == kEpiWarps + kLoadWarps) tc05::tmem_dealloc(tmem, kTmemCols);
}

}  // namespace sg
