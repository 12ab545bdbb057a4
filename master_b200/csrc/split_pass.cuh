// The production timestep pass for split-precision state: three or four
// kernels per step (one more on sampled steps) over the active cells, which the previous pass
// left sorted by cell (bottom segment + top segment of each cell's slots,
// counts in the `cin` occupancy set).
//
//   collide_cells  Cell::prepare + Cell::collide (dsmc/cell.cpp:42-111) of
//                  every cell.
//                  Per chunk of (up to 32) consecutive cells lane i selects for cell
//                  i and runs its candidate loop; the members' order is the
//                  id order (the reference's).
//                  Velocities are updated in place in the input buffer.
//   sample_cells   On sampled steps only (the reference's cadence,
//                  dsmc/statisticssampler.cpp:45-66): every cell's fp64
//                  moments and the y-binned profiles.
//   move_cells     System::accelerate + the mover's first flight
//                  (dsmc/system.cpp:133-144, dsmc/moleculemover.cpp:50-126)
//                  for every particle.  A particle that stays inside its
//                  empty voxel goes, moved, to the bottom segment of its cell
//                  in the output buffer; the rest ("movers"), accelerated but
//                  not moved, go to the gap just above: slots
//                  [base + stayers, base + n_in) hold exactly the cell's
//                  movers.  Particle records stream through a per-warp
//                  shared-memory ring with bulk copies, a group of cells
//                  ahead of the one in work.
//   place_movers   A mover whose flight ends in an empty voxel completes it
//                  and takes a top slot of its new cell (warp-aggregated
//                  atomics; the spill list when the cell is full).  Flights
//                  that meet a wall go through the general mover
//                  (bisection, facet, wall model) and the same placement: by
//                  the warp that found them (few cells), or from a list of
//                  (slot, source cell) pairs by
//   place_walls    where there are many.  The last block of the last kernel
//                  ends the pass (step counter, halting).
//
// Top slots are taken from the top of the cell down and never below
// base + n_in(cell), so they cannot meet the bottom segment or the gap.
//
// Member order: move_cells writes each cell's stayers in id order, so a
// bottom segment is normally sorted by id and only the few arrivals of the
// top segment are out of order.  The id rank of a member (the reference's
// cell-list order) is then its bottom position plus the arrivals below it:
// move_cells computes it with one shuffle and ballot per arrival, collide_cells
// turns a picked rank into its member by the bottom ids next to it.  A cell whose bottom segment is not sorted (after a repack or the
// stand-alone stage kernels) is ranked in full and leaves move_cells sorted.
#pragma once
#include "engine.cuh"

namespace dsmc {
namespace pass3 {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bulk copies global -> shared of this block (addresses and size multiples of
// 16 bytes), completing on an mbarrier.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Waits for the phase of the given parity; false when the (far too long)
// limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    for (unsigned i = 0; i < (1u << 22); ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// A particle record {A, B} of slot s in one 32-byte access.  (With A and B in
// arrays of their own a mover took four sectors, each half used, and
// place_movers 174 us at 256^3; now 108.)
__device__ __forceinline__ void load_record(const void *A, long long s, uint4 &a, float4 &b) {
    uint32_t r[8];
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(reinterpret_cast<const uint4 *>(A) + rec_at(s))
                 : "memory");
    a = make_uint4(r[0], r[1], r[2], r[3]);
    b = make_float4(__uint_as_float(r[4]), __uint_as_float(r[5]), __uint_as_float(r[6]), __uint_as_float(r[7]));
}
__device__ __forceinline__ void store_record(void *A, long long s, const uint4 &a, const float4 &b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(reinterpret_cast<uint4 *>(A) + rec_at(s)),
                 "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(__float_as_uint(b.x)), "r"(__float_as_uint(b.y)),
                 "r"(__float_as_uint(b.z)), "r"(__float_as_uint(b.w))
                 : "memory");
}

// Input occupancy of active cell a (clamped to its capacity).
__device__ __forceinline__ void input_counts(const PassParams &P, int a, const int4 &m, unsigned &nb, unsigned &nt) {
    nb = min(P.cells.bot[P.cin][a], (unsigned)m.y);
    nt = min(P.cells.top[P.cin][a], (unsigned)m.y - nb);
}
// Slot of member q of a cell: bottom segment, then top segment.
__device__ __forceinline__ int member_slot(int base, int cap, int nb, int nt, int q) {
    return q < nb ? base + q : base + cap - nt + (q - nb);
}

__device__ __forceinline__ unsigned warp_sum(unsigned x) { return __reduce_add_sync(0xffffffffu, x); }
__device__ __forceinline__ int warp_sum(int x) { return __reduce_add_sync(0xffffffffu, x); }

// The system shared by the valid lanes of a warp, or -2 when they differ
// (-1 when no lane is valid).  All lanes call.
__device__ __forceinline__ int common_system(bool valid, int sys) {
    const unsigned vm = __ballot_sync(0xffffffffu, valid);
    if (!vm) return -1;
    const int s0 = __shfl_sync(0xffffffffu, sys, __ffs(vm) - 1);
    return __all_sync(0xffffffffu, !valid || sys == s0) ? s0 : -2;
}

// collide_cells' chunks of 32 cells beyond each warp's first go to warps from
// a pass-wide counter when there are many per warp, so that a warp that
// finishes early takes more (a chunk's cost varies with its cells'
// collisions); place_walls' last block zeroes the counter for the next pass.
// Four chunks per warp or more take the counter.  (move_cells, place_movers
// and sample_cells keep a fixed stride: a counter made them no faster or
// slower.)  claim_issue starts a claim (lane 0), claim_take hands its chunk
// to every lane: issued a chunk ahead, the atomic's latency is hidden.
constexpr int CLAIM_MIN_CHUNKS_PER_WARP = 4;
__device__ __forceinline__ unsigned claim_issue(unsigned *counter, int lane) {
    return lane == 0 ? atomicAdd(counter, 1u) : 0u;
}
__device__ __forceinline__ int claim_take(unsigned claimed) { return (int)__shfl_sync(0xffffffffu, claimed, 0); }

// ---- collide_cells ----------------------------------------------------------

constexpr int C_WARPS = 4;
constexpr int PCAP = 512;    // members per warp and batch (>= the largest cell)
constexpr int NTMAX = 8;     // arrivals a lane merges on its own (sorted bottom segments)

struct CollideSmem {
    uint32_t ids[PCAP];  // batch members: ids and slots, cell by cell
    int slot[PCAP];
    int perm[PCAP];      // batch members by id rank within each cell (warp-ranked cells)
    uint32_t aid[32 * (NTMAX + 1)];  // lane i: its cell's arrivals in id order: id
    int aslot[32 * (NTMAX + 1)];     //   and slot (rows of NTMAX + 1: no bank conflicts)
};

// Velocities of one cell's members in the input buffer, by id rank.
struct RankVel {
    float4 *b;
    const int *perm;
    __device__ __forceinline__ void get(int r, float &x, float &y, float &z) const {
        const float4 v = b[rec_at(perm[r])];
        x = v.x;
        y = v.y;
        z = v.z;
    }
    __device__ __forceinline__ void set(int r, float x, float y, float z) const {
        float *q = reinterpret_cast<float *>(b + rec_at(perm[r]));
        q[0] = x;
        q[1] = y;
        q[2] = z;
    }
};
struct IdentityPerm {
    __device__ __forceinline__ void pick(int r0, int r1, int &s0, int &s1) const {
        s0 = r0;
        s1 = r1;
    }
};
// Velocities of a cell's members by slot.
struct SlotVel {
    float4 *b;
    __device__ __forceinline__ void get(int s, float &x, float &y, float &z) const {
        const float4 v = b[rec_at(s)];
        x = v.x;
        y = v.y;
        z = v.z;
    }
    __device__ __forceinline__ void set(int s, float x, float y, float z) const {
        float *q = reinterpret_cast<float *>(b + rec_at(s));
        q[0] = x;
        q[1] = y;
        q[2] = z;
    }
};
// Slots of the members of two id ranks in a cell whose bottom segment is
// sorted.  With the bottom ids b[k] (nothing below 0, everything at nb and
// above) and the arrivals' ids t[j] in order, arrival j has rank p_j =
// #{b < t[j]} + j, so p_j < r exactly if b[r - j - 1] > t[j], and p_j <= r if
// b[r - j] > t[j]: rank r is settled by the nt + 1 bottom members up to
// position r, without the other members' ids.
struct PickPerm {
    const float4 *B;
    const uint32_t *aid;
    const int *aslot;
    int nt, nb, base;
    __device__ __forceinline__ uint32_t bottom(int k) const {
        return k < 0 ? 0u : k >= nb ? 0xffffffffu : __float_as_uint(B[rec_at(base + k)].w);
    }
    __device__ __forceinline__ int resolve(int r, uint32_t b0, uint32_t b1, uint32_t b2) const {
        uint32_t at = b0, below = b1;  // b[r - j], b[r - j - 1]
        int j = 0;
        for (; j < nt; ++j) {
            const uint32_t t = aid[j];
            if (!(below > t)) return at > t ? aslot[j] : base + (r - j);
            at = below;
            below = j == 0 ? b2 : bottom(r - j - 2);
        }
        return base + (r - j);
    }
    __device__ __forceinline__ void pick(int r0, int r1, int &s0, int &s1) const {
        // both ranks' first three bottom ids in flight together (two arrivals)
        uint32_t x0 = 0, x1 = 0, x2 = 0, y0 = 0, y1 = 0, y2 = 0;
        if (nt > 0) {
            x0 = bottom(r0);
            x1 = bottom(r0 - 1);
            y0 = bottom(r1);
            y1 = bottom(r1 - 1);
        }
        if (nt > 1) {
            x2 = bottom(r0 - 2);
            y2 = bottom(r1 - 2);
        }
        s0 = resolve(r0, x0, x1, x2);
        s1 = resolve(r1, y0, y1, y2);
    }
};

__device__ __forceinline__ void publish_collide(const PassParams &P, int sys, unsigned col, unsigned cand,
                                                bool per_lane) {
    if (per_lane) {
        if (sys >= 0) {
            if (col) atomicAdd(&P.tally[sys].collisions, (unsigned long long)col);
            if (cand) atomicAdd(&P.tally[sys].candidates, (unsigned long long)cand);
        }
        return;
    }
    const unsigned c = warp_sum(col), d = warp_sum(cand);
    if ((threadIdx.x & 31) == 0 && sys >= 0) {
        if (c) atomicAdd(&P.tally[sys].collisions, (unsigned long long)c);
        if (d) atomicAdd(&P.tally[sys].candidates, (unsigned long long)d);
    }
}

// Bound by the latency of a lane's chain: header, arrivals' ids, the picks'
// bottom ids and velocities per candidate.  us per step, with every member's id
// of a colliding cell loaded and ranked, and so: 64^3 18.0 -> 17.1, 128^3 58 ->
// 35, 256^3 267 -> 153.  Five blocks per SM (96 registers): six spill (80
// registers; 172 us at 256^3), four have too few warps (179 us).
// CLAIM: chunks beyond each warp's first come from the counter (chosen by
// the launcher when there are many chunks per warp; a fixed stride measured
// faster with few: packed_64 and packed_128).
template <bool CLAIM>
__global__ void __launch_bounds__(32 * C_WARPS, 5) collide_cells_kernel(const __grid_constant__ PassParams P) {
    __shared__ CollideSmem smem[C_WARPS];
    const int lane = threadIdx.x & 31;
    const volatile Status *vs = P.status;
    if (vs->halted) return;
    const uint32_t step = vs->step;
    CollideSmem &W = smem[threadIdx.x >> 5];
    float4 *Bin = reinterpret_cast<float4 *>(P.parts.B[P.cur]);

    const int C = P.cells.num_cells, CH = P.chunk;
    const int nchunks = (C + CH - 1) / CH;
    unsigned col = 0, cand = 0;  // this lane's counts for system tsys
    int tsys = -1;

    // A warp's first chunk is its index; with CLAIM the later ones come from
    // the counter, each claimed while the chunk before is in work.
    const int nw = gridDim.x * C_WARPS;
    unsigned nxt = 0;
    for (int ch = blockIdx.x * C_WARPS + (threadIdx.x >> 5); ch < nchunks;
         ch = CLAIM ? nw + claim_take(nxt) : ch + nw) {
        if (CLAIM) nxt = claim_issue(&P.status->collide_taken, lane);  // the next chunk, in flight meanwhile
        const int first = ch * CH;
        const bool mine = lane < min(CH, C - first);
        const int a = first + lane;
        int4 m = make_int4(0, 0, 0, -1);
        unsigned nb = 0, nt = 0;
        double vr = 0, rest = 0;
        int pairs = 0;
        if (mine) {
            m = P.cells.meta[a];
            input_counts(P, a, m, nb, nt);
            const double4 st = P.cells.state[a];
            vr = st.x;
            rest = st.y;
            if (P.do_collide) {
                pairs = ntc_select(st.z, (int)(nb + nt), vr, rest);
                if (nb + nt < 2) pairs = 0;
                if (nb + nt > (unsigned)PCAP) {  // the host keeps every cap below PCAP
                    atomicOr(&P.status->error, DSMC_EBIT_SMEM);
                    pairs = 0;
                }
            }
        }
        const int n = (int)(nb + nt);
        const int sys = m.w;
        const int csys = common_system(mine, sys);
        if (csys != tsys) {
            publish_collide(P, tsys, col, cand, false);
            col = cand = 0;
            tsys = csys;
        }

        // Cells with a sorted bottom and few arrivals, as nearly all: each lane
        // sorts its cell's arrivals by id and runs its candidate loop.
        const bool lp = pairs > 0 && P.sorted_in && (int)nt <= NTMAX;
        if (lp) {
            uint32_t *aid = W.aid + lane * (NTMAX + 1);
            int *as = W.aslot + lane * (NTMAX + 1);
            const int t0 = m.x + m.y - (int)nt;
            for (int j = 0; j < (int)nt; ++j) aid[j] = __float_as_uint(Bin[rec_at(t0 + j)].w);
            for (int j = 0; j < (int)nt; ++j) {
                const uint32_t id = aid[j];
                int i = j - 1;
                while (i >= 0 && aid[i] > id) {
                    aid[i + 1] = aid[i];
                    as[i + 1] = as[i];
                    --i;
                }
                aid[i + 1] = id;
                as[i + 1] = t0 + j;
            }
            DrawStream rs;
            rs.init(P.sys[sys].seed, (uint32_t)m.z, step, DSMC_TAG_COLLIDE);
            unsigned long long c_ = 0;
            SlotVel vel;
            vel.b = Bin;
            PickPerm pick;
            pick.B = Bin;
            pick.aid = aid;
            pick.aslot = as;
            pick.nt = (int)nt;
            pick.nb = (int)nb;
            pick.base = m.x;
            ntc_loop<float>(rs, n, pairs, vr, vel, pick, c_);
            col += (unsigned)c_;
            cand += (unsigned)pairs;
        }
        // The others (unsorted bottoms after a repack or the stage kernels,
        // many arrivals): rank their members by id, a batch at a time, and run
        // the batch's candidate loops one cell per lane.
        unsigned todo = __ballot_sync(0xffffffffu, pairs > 0 && !lp);
        while (todo) {
            // the batch: colliding cells, in order, whose members fit PCAP
            unsigned ready = 0;
            {
                int off = 0;
                for (unsigned t2 = todo; t2;) {
                    const int c = __ffs(t2) - 1;
                    const int nc = __shfl_sync(0xffffffffu, n, c);
                    if (off + nc > PCAP) break;  // off > 0 here: nc <= PCAP
                    off += nc;
                    ready |= 1u << c;
                    t2 &= t2 - 1u;
                }
            }
            todo &= ~ready;
            // offsets of the batch cells' members: exclusive prefix over lanes
            const bool rb = (ready >> lane) & 1u;
            const int nr = rb ? n : 0;
            int incl = nr;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int start = incl - nr;
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            // ids and slots of every batch member: independent loads
            for (int f0 = 0; f0 < total; f0 += 32) {
                const int f = f0 + lane;
                int c = 0;  // the last lane whose start is <= f: a batch cell holding member f
#pragma unroll
                for (int st = 16; st > 0; st >>= 1) {
                    const int sc = __shfl_sync(0xffffffffu, start, c + st);
                    if (sc <= f) c += st;
                }
                const int k = f - __shfl_sync(0xffffffffu, start, c);
                const int cb = __shfl_sync(0xffffffffu, m.x, c), cc = __shfl_sync(0xffffffffu, m.y, c);
                const int cnb = (int)__shfl_sync(0xffffffffu, nb, c), cnt = __shfl_sync(0xffffffffu, n, c) - cnb;
                if (f < total) W.slot[f] = member_slot(cb, cc, cnb, cnt, k);
            }
            __syncwarp();
            // the members' ids, four loads in flight per lane
            for (int f0 = lane; f0 < total; f0 += 128) {
                uint32_t v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int f = f0 + 32 * u;
                    v[u] = f < total ? __float_as_uint(Bin[rec_at(W.slot[f])].w) : 0u;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (f0 + 32 * u < total) W.ids[f0 + 32 * u] = v[u];
            }
            __syncwarp();
            // id ranks by the warp, cell by cell
            for (unsigned t2 = ready; t2; t2 &= t2 - 1u) {
                const int c = __ffs(t2) - 1;
                const int off = __shfl_sync(0xffffffffu, start, c);
                const int nc = __shfl_sync(0xffffffffu, n, c);
                const int nbc = (int)__shfl_sync(0xffffffffu, nb, c);
                const int ntc = nc - nbc;
                if (nc <= 32) {
                    const uint32_t id = lane < nc ? W.ids[off + lane] : 0xffffffffu;
                    const uint32_t nxt = __shfl_down_sync(0xffffffffu, id, 1);
                    const bool sorted = !__any_sync(0xffffffffu, lane + 1 < nbc && !(id < nxt));
                    int rank = 0;
                    if (sorted) {
                        // bottom position (or the bottom members below an
                        // arrival) plus the arrivals below
                        const unsigned bmask = nbc >= 32 ? 0xffffffffu : (1u << nbc) - 1u;
                        unsigned add = 0, pb = 0;
                        for (int i = 0; i < ntc; ++i) {
                            const uint32_t t = __shfl_sync(0xffffffffu, id, nbc + i);
                            add += t < id;
                            const unsigned bl = __popc(bmask & __ballot_sync(0xffffffffu, id < t));
                            if (lane == nbc + i) pb = bl;
                        }
                        rank = (lane < nbc ? lane : (int)pb) + (int)add;
                    } else {
#pragma unroll
                        for (int r = 0; r < 32; ++r) rank += __shfl_sync(0xffffffffu, id, r) < id;
                    }
                    if (lane < nc) W.perm[off + rank] = W.slot[off + lane];
                } else {
                    const uint32_t *ids = W.ids + off;
                    bool viol = false;
                    for (int q = lane; q + 1 < nbc; q += 32) viol |= !(ids[q] < ids[q + 1]);
                    const bool sorted = !__any_sync(0xffffffffu, viol);
                    for (int q = lane; q < nc; q += 32) {
                        const uint32_t id = ids[q];
                        int rank = 0;
                        if (sorted) {
                            if (q < nbc) {
                                rank = q;
                            } else {  // bottom members below: binary search
                                int lo = 0, hi = nbc;
                                while (lo < hi) {
                                    const int mid = (lo + hi) >> 1;
                                    if (ids[mid] < id) lo = mid + 1;
                                    else hi = mid;
                                }
                                rank = lo;
                            }
                            for (int i = nbc; i < nc; ++i) rank += ids[i] < id;
                        } else {
                            for (int r = 0; r < nc; ++r) rank += ids[r] < id;
                        }
                        W.perm[off + rank] = W.slot[off + q];
                    }
                }
            }
            __syncwarp();
            if (rb) {
                const SysDev &g = P.sys[sys];
                DrawStream rs;
                rs.init(g.seed, (uint32_t)m.z, step, DSMC_TAG_COLLIDE);
                unsigned long long c_ = 0;
                RankVel vel;
                vel.b = Bin;
                vel.perm = W.perm + start;
                ntc_loop<float>(rs, n, pairs, vr, vel, IdentityPerm(), c_);
                col += (unsigned)c_;
                cand += (unsigned)pairs;
            }
            __syncwarp();
        }
        if (mine && P.do_collide)
            *reinterpret_cast<double2 *>(&P.cells.state[a]) = make_double2(vr, rest);

        if (tsys == -2) {  // a chunk that spans systems: per-lane counts
            publish_collide(P, sys, col, cand, true);
            col = cand = 0;
        }
    }
    publish_collide(P, tsys, col, cand, false);
}

// ---- sample_cells -----------------------------------------------------------

constexpr int SHIST = 1024;  // v_x histogram bins a warp counts in shared memory

// Eight per-lane values summed over the warp, transposed: lane l returns the
// sum of slot l >> 2 (lanes 4j..4j+3 hold the sum of slot j).  Each exchange
// halves the slots a lane carries (4, 2, 1, then two plain steps): 9 fp64
// shuffles where eight separate reductions take 40.  All lanes call.
__device__ __forceinline__ double warp_transpose_sum8(const double (&v)[8], int lane) {
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    double w[4], u[2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = (b4 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, b4 ? v[i] : v[i + 4], 16);
#pragma unroll
    for (int i = 0; i < 2; ++i)
        u[i] = (b3 ? w[i + 2] : w[i]) + __shfl_xor_sync(0xffffffffu, b3 ? w[i] : w[i + 2], 8);
    double t = (b2 ? u[1] : u[0]) + __shfl_xor_sync(0xffffffffu, b2 ? u[0] : u[1], 4);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    return t;
}

// The sampler on the reference's cadence (StatisticsSampler::sample,
// dsmc/statisticssampler.cpp:45-66), after collide_cells on sampled steps
// only: every cell's fp64 moments and the y-binned profiles.  A warp takes a
// chunk of 32 cells, their headers one per lane, then each sampled cell with
// its members over the lanes.  Per cell one transposing butterfly sums the
// six velocity moments and the cell's profile sums {v_z, 1/2 m v_z^2} in the
// bin of its first member (members in another bin, rare when the bins are
// no finer than the cells, add their own); lanes 4j then add slot j to the
// cell's moment row or the profile.  Each warp counts the v_x histogram in
// shared memory and adds it to its copy of the sums once per system (every
// particle lands in one of a few bins: one global atomic per particle queued
// on those addresses).
__global__ void __launch_bounds__(32 * C_WARPS) sample_cells_kernel(const __grid_constant__ PassParams P) {
    __shared__ unsigned hist[C_WARPS][SHIST];
    const int lane = threadIdx.x & 31;
    const volatile Status *vs = P.status;
    if (vs->halted) return;
    const uint32_t step = vs->step;
    unsigned *H = hist[threadIdx.x >> 5];
    for (int b = lane; b < SHIST; b += 32) H[b] = 0;
    __syncwarp();
    int hsys = -1;  // the system whose histogram H holds
    auto flush = [&]() {
        if (hsys >= 0) {
            const SysDev &gh = P.sys[hsys];
            double *pr = profile_copy(gh) + 3 * (size_t)gh.prof_bins;
            for (int b = lane; b < gh.prof_bins; b += 32)
                if (H[b]) {
                    atomicAdd(pr + b, (double)H[b]);
                    H[b] = 0;
                }
            __syncwarp();
        }
    };
    // moment row entry this lane adds: slot j of the butterfly to M[1 + j]
    // (j < 6), lane 1 the count to M[0]; lane 12 also M[7] = the three sums
    // of squares
    const int slot = lane >> 2;
    const int mcol = (lane & 3) == 0 && slot < 6 ? 1 + slot : lane == 1 ? 0 : -1;
    const int C = P.cells.num_cells, CH = P.chunk;
    const int nchunks = (C + CH - 1) / CH;
    const int nwarps = gridDim.x * C_WARPS;
    for (int ch = blockIdx.x * C_WARPS + (threadIdx.x >> 5); ch < nchunks; ch += nwarps) {
        const int a = ch * CH + lane;
        int4 m = make_int4(0, 0, 0, -1);
        unsigned nb = 0, nt = 0;
        bool smp = false;
        if (lane < CH && a < C) {
            m = P.cells.meta[a];
            input_counts(P, a, m, nb, nt);
            const SysDev &g = P.sys[m.w];
            smp = g.sample_interval > 0 && step > 0 && (step % (uint32_t)g.sample_interval) == 0 &&
                  step >= (uint32_t)g.sample_begin;
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, smp); todo; todo &= todo - 1u) {
            const int c = __ffs(todo) - 1;
            const int ac = ch * CH + c;
            const int sys = __shfl_sync(0xffffffffu, m.w, c);
            const int cb = __shfl_sync(0xffffffffu, m.x, c), cc = __shfl_sync(0xffffffffu, m.y, c);
            const int cnb = (int)__shfl_sync(0xffffffffu, nb, c), cnt = (int)__shfl_sync(0xffffffffu, nt, c);
            const int n = cnb + cnt;
            const SysDev &g = P.sys[sys];
            double *M = P.cells.mom + 8 * (size_t)ac;
            const double mold = mcol >= 0 ? M[mcol] : 0.0;  // in flight with the members' loads
            const double m7 = lane == 12 ? M[7] : 0.0;
            const bool local = g.prof_bins <= SHIST;
            if (local && sys != hsys) {
                flush();
                hsys = sys;
            }
            // Σv_x Σv_y Σv_z Σv_x² Σv_y² Σv_z², then Σv_z and Σ 1/2 m v_z² in bin b0
            double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            int b0 = 0;
            unsigned in0 = 0;  // members in bin b0
            for (int q0 = 0; q0 < n; q0 += 32) {
                const int q = q0 + lane;
                const bool ok = q < n;
                int bin = 0;
                double x = 0, y = 0, z = 0;
                if (ok) {
                    const int sl = member_slot(cb, cc, cnb, cnt, q);
                    uint4 ra;
                    float4 b;
                    load_record(P.parts.A[P.cur], sl, ra, b);
                    x = b.x;
                    y = b.y;
                    z = b.z;
                    bin = profile_bin(g, Split32::y_of(g, ra));
                    v[0] += x;
                    v[1] += y;
                    v[2] += z;
                    v[3] += x * x;
                    v[4] += y * y;
                    v[5] += z * z;
                }
                if (q0 == 0) b0 = __shfl_sync(0xffffffffu, bin, 0);
                const bool here = ok && bin == b0;
                const double e = 0.5 * g.mass * z * z;
                if (here) {
                    v[6] += z;
                    v[7] += e;
                }
                in0 += (unsigned)__popc(__ballot_sync(0xffffffffu, here));
                profile_add_warp(g, ok && !here, bin, 1.0, z, e);
                if (ok) {
                    if (local) {
                        const int hb = profile_vx_bin(g, x);
                        if (hb >= 0) atomicAdd(&H[hb], 1u);
                    } else {
                        profile_vx(g, x);
                    }
                }
            }
            const double t = warp_transpose_sum8(v, lane);
            const double sq = __shfl_sync(0xffffffffu, t, 12) + __shfl_sync(0xffffffffu, t, 16) +
                              __shfl_sync(0xffffffffu, t, 20);
            if (mcol >= 0) M[mcol] = mold + (mcol == 0 ? (double)n : t);
            if (lane == 12) M[7] = m7 + sq;
            if (in0) {
                double *pr = profile_copy(g) + 3 * b0;
                if (lane == 2) atomicAdd(pr, (double)in0);
                if (lane == 24) atomicAdd(pr + 1, t);
                if (lane == 28) atomicAdd(pr + 2, t);
            }
            if (lane == 0 && ac == g.active_begin) atomicAdd(&P.tally[sys].samples, 1ull);
        }
    }
    flush();
}

// ---- move_cells -------------------------------------------------------------

constexpr int M_WARPS = 4;

struct MoveTab {
    int4 t[32];  // {first slot, slots, bottom | top << 16 occupancy, system}: one load per cell
    int first, ncell;
    __device__ __forceinline__ static int nb(const int4 &c) { return c.z & 0xffff; }
    __device__ __forceinline__ static int nt(const int4 &c) { return (int)((unsigned)c.z >> 16); }
};
template <int R> struct MoveSmem {
    static constexpr int H = R < 256 ? R : 256;  // records of a staged group
    static constexpr int T = 2 * H;              // two groups
    uint4 rec[2 * T];  // records of 32 bytes
    __device__ __forceinline__ uint4 a(int r) const { return rec[2 * r]; }
    __device__ __forceinline__ float4 b(int r) const { return *reinterpret_cast<const float4 *>(&rec[2 * r + 1]); }
    __device__ __forceinline__ uint32_t id(int r) const { return rec[2 * r + 1].w; }
    __device__ __forceinline__ void set(int r, const uint4 &ra, const float4 &rb) {
        rec[2 * r] = ra;
        *reinterpret_cast<float4 *>(&rec[2 * r + 1]) = rb;
    }
    uint64_t bar[2];   // a half's copies
    MoveTab tab[2];
    uint16_t pref[R + 2];  // two-pass placement: stayers before each member
};

// accelerate, then the first flight when it stays inside the particle's empty
// voxel (the reference's outcome: r += v dt lands in an empty voxel,
// dsmc/moleculemover.cpp:74-77); false leaves the particle accelerated.
//
// A system's constants of the first flight, held in registers.
struct FlightConst {
    float inv_vox[3], dt, accel[3];  // accel: the flow axis's accel_dt_f, 0 on the others
};
__device__ __forceinline__ FlightConst flight_const(const SysDev &g) {
    FlightConst k;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        k.inv_vox[d] = g.inv_vox_f[d];
        k.accel[d] = g.flow_dir == d ? g.accel_dt_f : 0.0f;
    }
    k.dt = g.dt_f;
    return k;
}
// first_flight on the packed record itself: the voxel index is never
// unpacked (a stayer changes only its offsets, a mover only its velocity).
// The values that unpack + first_flight + pack give.  [0, 1) is tested on the
// bits: of the floats, exactly those from 0 to below 1 are below 0x3f800000 as
// unsigned numbers (negative ones and NaNs are above).
__device__ __forceinline__ bool first_flight_raw(const FlightConst &k, uint4 &a, float4 &b) {
    b.x += k.accel[0];
    b.y += k.accel[1];
    b.z += k.accel[2];
    const uint32_t x0 = __float_as_uint(fmaf(b.x * k.inv_vox[0], k.dt, __uint_as_float(a.y)));
    const uint32_t x1 = __float_as_uint(fmaf(b.y * k.inv_vox[1], k.dt, __uint_as_float(a.z)));
    const uint32_t x2 = __float_as_uint(fmaf(b.z * k.inv_vox[2], k.dt, __uint_as_float(a.w)));
    // (the flag of a particle whose voxel is not empty, the general mover's, is a.y's sign bit)
    const bool stay = (max(max(x0, x1), x2) < 0x3f800000u) & ((int)a.y >= 0);
    if (stay) {
        a.y = x0;
        a.z = x1;
        a.w = x2;
    }
    return stay;
}

// One cell of at most 32 * NR members whose bottom segment is sorted by id,
// held in registers (member q = 32 k + lane in ra[k], rb[k]): flight of every
// member, then stayers to the bottom segment in id order and movers to the
// gap.  Returns the number of stayers.  All lanes call.
template <int NR>
__device__ __forceinline__ unsigned place_sorted(const FlightConst &fc, uint4 (&ra)[NR], float4 (&rb)[NR], int base, int n,
                                                 int nb, void *out, int lane) {
    const unsigned below = (1u << lane) - 1u;
    bool stay[NR];
    uint32_t id[NR];
    unsigned fast[NR], slow[NR], bm[NR], add[NR], pb[NR];
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        const bool valid = 32 * k + lane < n;
        stay[k] = first_flight_raw(fc, ra[k], rb[k]);
        id[k] = valid ? __float_as_uint(rb[k].w) : 0xffffffffu;
        fast[k] = __ballot_sync(0xffffffffu, valid && stay[k]);
        slow[k] = __ballot_sync(0xffffffffu, valid && !stay[k]);
        const int nbk = nb - 32 * k;  // bottom members of chunk k
        bm[k] = nbk >= 32 ? 0xffffffffu : nbk <= 0 ? 0u : (1u << nbk) - 1u;
        add[k] = pb[k] = 0;
    }
    // each arrival i: staying arrivals below every member, bottom stayers
    // below the arrival
    for (int i = nb; i < n; ++i) {
        const int li = i & 31, ki = i >> 5;
        uint32_t src = id[0];
        unsigned fk = fast[0];
#pragma unroll
        for (int k = 1; k < NR; ++k) {
            src = ki == k ? id[k] : src;
            fk = ki == k ? fast[k] : fk;
        }
        const uint32_t t = __shfl_sync(0xffffffffu, src, li);
        const unsigned ts = (fk >> li) & 1u;
        unsigned bl = 0;
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            add[k] += ts && t < id[k];
            bl += (unsigned)__popc(fast[k] & bm[k] & __ballot_sync(0xffffffffu, id[k] < t));
        }
#pragma unroll
        for (int k = 0; k < NR; ++k)
            if (lane == li && ki == k) pb[k] = bl;
    }
    unsigned fs_before = 0, mv_before = 0, nfs = 0;  // bottom stayers and movers of the earlier chunks; stayers
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        const int q = 32 * k + lane;
        if (q < n) {
            const unsigned dst =
                stay[k] ? (unsigned)base + (q < nb ? fs_before + (unsigned)__popc(fast[k] & bm[k] & below) : pb[k]) + add[k]
                        : (unsigned)(base + n) - 1u - mv_before - (unsigned)__popc(slow[k] & below);
            store_record(out, dst, ra[k], rb[k]);
        }
        fs_before += (unsigned)__popc(fast[k] & bm[k]);
        mv_before += (unsigned)__popc(slow[k]);
        nfs += (unsigned)__popc(fast[k]);
    }
    return nfs;
}

// Two cells of at most 32 members each with sorted bottom segments and one
// system: place_sorted<1> for both, written as one straight-line body so that
// the two cells' dependency chains interleave.  nfs[k]: stayers of cell k.
// All lanes call.
__device__ __forceinline__ void place_pair(const FlightConst &fc, uint4 (&ra)[2], float4 (&rb)[2], const int base[2],
                                          const int n[2], const int nb[2], void *out, int lane, unsigned nfs[2]) {
    const unsigned below = (1u << lane) - 1u;
    bool stay[2];
    uint32_t id[2];
    unsigned fast[2], slow[2], bm[2], add[2], pb[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const bool valid = lane < n[k];
        stay[k] = first_flight_raw(fc, ra[k], rb[k]);
        id[k] = valid ? __float_as_uint(rb[k].w) : 0xffffffffu;
        fast[k] = __ballot_sync(0xffffffffu, valid && stay[k]);
        slow[k] = __ballot_sync(0xffffffffu, valid && !stay[k]);
        bm[k] = nb[k] >= 32 ? 0xffffffffu : (1u << nb[k]) - 1u;
        add[k] = pb[k] = 0;
    }
    // arrival j of each cell: staying arrivals below every member, bottom
    // stayers below the arrival (both cells in every iteration)
    const int nt0 = n[0] - nb[0], nt1 = n[1] - nb[1];
    const int ntmax = max(nt0, nt1);
    for (int j = 0; j < ntmax; ++j) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool has = j < (k ? nt1 : nt0);
            const int li = (nb[k] + j) & 31;
            const uint32_t t = __shfl_sync(0xffffffffu, id[k], li);
            const unsigned ts = has ? (fast[k] >> li) & 1u : 0u;
            add[k] += ts && t < id[k];
            const unsigned bl = (unsigned)__popc(fast[k] & bm[k] & __ballot_sync(0xffffffffu, id[k] < t));
            if (has && lane == li) pb[k] = bl;
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (lane < n[k]) {
            const unsigned dst =
                stay[k] ? (unsigned)base[k] + (lane < nb[k] ? (unsigned)__popc(fast[k] & bm[k] & below) : pb[k]) + add[k]
                        : (unsigned)(base[k] + n[k]) - 1u - (unsigned)__popc(slow[k] & below);
            store_record(out, dst, ra[k], rb[k]);
        }
        nfs[k] = (unsigned)__popc(fast[k]);
    }
}

// A cell whose n records are staged at record r0: any size, any order of the
// bottom segment, in two passes.  Returns the number of stayers.  All lanes
// call.
template <int R>
__device__ __noinline__ unsigned place_staged(int sorted_in, FlightConst fc, MoveSmem<R> &W, int r0, int base, int n, int nb,
                                              void *out, int lane) {
    auto rid = [&](int q) { return W.id(r0 + q); };
    bool viol = false;
    if (!sorted_in)
        for (int q = lane; q + 1 < nb; q += 32) viol |= !(rid(q) < rid(q + 1));
    const bool sorted = !__any_sync(0xffffffffu, viol);
    if (sorted && n <= 128) {
        uint4 ra[4];
        float4 rb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = r0 + max(min(32 * k + lane, n - 1), 0);
            ra[k] = W.a(r);
            rb[k] = W.b(r);
        }
        return place_sorted<4>(fc, ra, rb, base, n, nb, out, lane);
    }
    const unsigned below = (1u << lane) - 1u;
    // pass 1: every member's flight; the record goes back and pref[q] counts
    // the stayers before member q
    unsigned S = 0;
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int q = c0 + lane;
        const bool valid = q < n;
        bool stay = false;
        if (valid) {
            uint4 ra = W.a(r0 + q);
            float4 rb = W.b(r0 + q);
            stay = first_flight_raw(fc, ra, rb);
            W.set(r0 + q, ra, rb);
        }
        const unsigned fast = __ballot_sync(0xffffffffu, valid && stay);
        if (valid) W.pref[q] = (uint16_t)(S + (unsigned)__popc(fast & below));
        S += (unsigned)__popc(fast);
    }
    if (lane == 0) W.pref[n] = (uint16_t)S;
    __syncwarp();
    // pass 2: stayers in id order, movers below the top of the gap
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int q = c0 + lane;
        if (q < n) {
            const uint32_t id = rid(q);
            unsigned dst;
            if (W.pref[q + 1] > W.pref[q]) {
                unsigned pos;
                if (sorted) {
                    int lb = q;  // bottom members below this id
                    if (q >= nb) {
                        int lo = 0, hi = nb;
                        while (lo < hi) {
                            const int mid = (lo + hi) >> 1;
                            if (rid(mid) < id) lo = mid + 1;
                            else hi = mid;
                        }
                        lb = lo;
                    }
                    pos = W.pref[lb];
                    for (int i = nb; i < n; ++i) pos += (W.pref[i + 1] > W.pref[i]) && rid(i) < id;
                } else {
                    pos = 0;
                    for (int i = 0; i < n; ++i) pos += (W.pref[i + 1] > W.pref[i]) && rid(i) < id;
                }
                dst = (unsigned)base + pos;
            } else {
                dst = (unsigned)(base + n) - 1u - ((unsigned)q - W.pref[q]);
            }
            store_record(out, dst, W.a(r0 + q), W.b(r0 + q));
        }
    }
    return S;
}

// Cells staged together: cells [ci, ci + cnt) of their chunk, at most H
// records, or one cell larger than that (`big`: staged when its turn comes).
struct MoveGroup {
    int ci, cnt;  // cnt 0: none left
    bool big, last;  // last: of its chunk
};

// Each lane stages its own cell: a bulk copy of the bottom segment and one of
// the top, tracked by an mbarrier per half of the staging memory; a group is in
// flight while the one before is worked on.  With 16-byte copies per lane, cell by
// cell, the staging took a quarter of the instructions.  us per step at 64^3 /
// 128^3 / 256^3: so staged 16.9 / 83 / 549; in groups of up to 80 records 16.4 /
// 72 / 470, of 128 15.0 / 65 / 418 (4.8 TB/s, 0.75 of the copy rate), of 160
// 14.6 / 63 / 430, of 192 14.6 / 62 / 448.  Loaded straight into registers a pair of cells
// ahead, with fewer instructions still, 14.5 / 84 / 590: too few bytes in flight.
template <int R>
__global__ void __launch_bounds__(32 * M_WARPS, 4) move_cells_kernel(const __grid_constant__ PassParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int H = MoveSmem<R>::H, T2 = MoveSmem<R>::T;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const volatile Status *vs = P.status;
    if (vs->halted) return;

    MoveSmem<R> &W = reinterpret_cast<MoveSmem<R> *>(smem_raw)[wib];
    const uint4 *in = reinterpret_cast<const uint4 *>(P.parts.A[P.cur]);
    void *out = P.parts.A[P.cur ^ 1];

    const int C = P.cells.num_cells, CH = P.chunk;
    const int nchunks = (C + CH - 1) / CH;
    const int wstride = gridDim.x * M_WARPS;
    const int chunk0 = blockIdx.x * M_WARPS + wib;

    auto load_tab = [&](int b, int ch) {
        MoveTab &T = W.tab[b];
        const int first = ch * CH;
        const int ncell = ch < nchunks ? min(CH, C - first) : 0;
        if (lane == 0) {
            T.first = first;
            T.ncell = ncell;
        }
        int4 row = make_int4(0, 0, 0, 0);
        if (lane < ncell) {
            const int a = first + lane;
            const int4 m = P.cells.meta[a];
            unsigned nb, nt;
            input_counts(P, a, m, nb, nt);
            if (nb + nt > (unsigned)R) {  // the host sizes R above every cap
                atomicOr(&P.status->error, DSMC_EBIT_SMEM);
                nb = nt = 0;
            }
            // top slots free for arrivals this pass: above the input occupancy
            P.cells.room[a] = make_int2(m.x + m.y, m.y - (int)(nb + nt));
            row = make_int4(m.x, m.y, (int)(nb | nt << 16), m.w);  // (cells hold at most R <= 512)
        }
        T.t[lane] = row;
    };
    // Lane i publishes cell i's bottom occupancy and clears the set the next
    // pass writes.
    auto write_tab = [&](int b, unsigned nfs) {
        const MoveTab &T = W.tab[b];
        if (lane < T.ncell) {
            const int a = T.first + lane;
            P.cells.bot[P.cout][a] = nfs;
            P.cells.bot[P.cclear][a] = 0;
            P.cells.top[P.cclear][a] = 0;
        }
    };

    if (lane == 0) {
        mbar_init(&W.bar[0], 1);
        mbar_init(&W.bar[1], 1);
        mbar_fence_init();
    }
    load_tab(0, chunk0);
    load_tab(1, chunk0 + wstride);
    __syncwarp();

    int gt = 0, gi = 0;     // the next group: chunk ordinal, first cell
    uint32_t parity = 0;    // bit h: phase of half h's barrier
    bool ok = true;
    // The next group; its copies start, into half h, unless it is big.
    auto next_group = [&](MoveGroup &g, int h) {
        const MoveTab &T = W.tab[gt & 1];
        const int nc = T.ncell;
        g.cnt = 0;
        if (gi >= nc) return;  // past the warp's last cell
        const int4 c = T.t[lane];  // (rows past the chunk's cells are empty)
        const int nb = MoveTab::nb(c), nt = MoveTab::nt(c), n = lane >= gi ? nb + nt : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const bool fits = lane >= gi && lane < nc && incl <= H;
        g.ci = gi;
        g.cnt = __popc(__ballot_sync(0xffffffffu, fits));
        g.big = g.cnt == 0;
        if (g.big) {
            g.cnt = 1;
        } else {
            const int total = __shfl_sync(0xffffffffu, incl, gi + g.cnt - 1);
            if (lane == 0) mbar_expect(&W.bar[h], 32u * (unsigned)total);
            __syncwarp();
            if (fits) {
                uint4 *dst = &W.rec[2 * (h * H + incl - n)];
                if (nb) bulk_load(dst, in + rec_at(c.x), 32u * (unsigned)nb, &W.bar[h]);
                if (nt) bulk_load(dst + 2 * nb, in + rec_at(c.x + c.y - nt), 32u * (unsigned)nt, &W.bar[h]);
            }
        }
        gi += g.cnt;
        g.last = gi == nc;
        if (gi == CH) {
            ++gt;
            gi = 0;
        }
    };

    int ct = 0;             // chunk in work
    unsigned nfs_mine = 0;  // lane i: bottom occupancy of cell i of the chunk in work
    unsigned moved = 0;     // particles moved, system tsys (warp-uniform)
    int tsys = -1;
    FlightConst fc = {};    // constants of system tsys
    MoveGroup cur, nxt;
    int half = 0;
    next_group(cur, 0);
    while (cur.cnt) {
        const MoveTab &T = W.tab[ct & 1];
        int r = half * H;   // record of the cell in work
        if (cur.big) {
            // (nothing else is staged: the whole ring is free)
            const int4 c = T.t[cur.ci];
            const int nb = MoveTab::nb(c), nt = MoveTab::nt(c);
            if (lane == 0) {
                mbar_expect(&W.bar[half], 32u * (unsigned)(nb + nt));
                if (nb) bulk_load(W.rec, in + rec_at(c.x), 32u * (unsigned)nb, &W.bar[half]);
                if (nt) bulk_load(W.rec + 2 * nb, in + rec_at(c.x + c.y - nt), 32u * (unsigned)nt, &W.bar[half]);
            }
            __syncwarp();
            r = 0;
        } else {
            next_group(nxt, half ^ 1);
        }
        ok &= mbar_wait(&W.bar[half], (parity >> half) & 1u);
        parity ^= 1u << half;
        const int end = cur.ci + cur.cnt;
        for (int i = cur.ci; i < end;) {
            const int4 c0 = T.t[i], c1 = T.t[min(i + 1, 31)];
            if (c0.w != tsys) {
                if (lane == 0 && tsys >= 0 && moved) atomicAdd(&P.tally[tsys].particle_steps, (unsigned long long)moved);
                moved = 0;
                tsys = c0.w;
                fc = flight_const(P.sys[tsys]);
            }
            const int nb[2] = {MoveTab::nb(c0), MoveTab::nb(c1)};
            int n[2] = {nb[0] + MoveTab::nt(c0), nb[1] + MoveTab::nt(c1)};
            if (P.sorted_in && n[0] <= 32) {
                // two small cells of one system go together
                const bool two = i + 1 < end && n[1] <= 32 && c1.w == c0.w;
                n[1] = two ? n[1] : 0;
                const int base[2] = {c0.x, c1.x};
                const int q[2] = {r + lane, r + n[0] + lane};
                uint4 ra[2];
                float4 rb[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int at = min(q[k], T2 - 1);  // (lanes past the members read some record)
                    ra[k] = W.a(at);
                    rb[k] = W.b(at);
                }
                unsigned nfs[2];
                place_pair(fc, ra, rb, base, n, nb, out, lane, nfs);
                if (lane == i) nfs_mine = nfs[0];
                if (two && lane == i + 1) nfs_mine = nfs[1];
                r += n[0] + n[1];
                moved += (unsigned)(n[0] + n[1]);
                i += two ? 2 : 1;
                continue;
            }
            unsigned nfs;
            if (P.sorted_in && n[0] <= 64) {
                uint4 ra[2];
                float4 rb[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int at = min(r + 32 * k + lane, T2 - 1);
                    ra[k] = W.a(at);
                    rb[k] = W.b(at);
                }
                nfs = place_sorted<2>(fc, ra, rb, c0.x, n[0], nb[0], out, lane);
            } else {
                nfs = place_staged<R>(P.sorted_in, fc, W, r, c0.x, n[0], nb[0], out, lane);
                proxy_fence();  // its writes to the ring, before the next copies there
            }
            if (lane == i) nfs_mine = nfs;
            r += n[0];
            moved += (unsigned)n[0];
            ++i;
        }
        __syncwarp();  // every lane is done with the group's records
        if (cur.last) {
            write_tab(ct & 1, nfs_mine);
            __syncwarp();
            load_tab(ct & 1, chunk0 + (ct + 2) * wstride);
            __syncwarp();
            ++ct;
        }
        if (cur.big) {
            half ^= 1;
            next_group(cur, half);
        } else {
            half ^= 1;
            cur = nxt;
        }
    }
    if (!ok) atomicOr(&P.status->error, DSMC_EBIT_SMEM);
    if (lane == 0 && tsys >= 0 && moved) atomicAdd(&P.tally[tsys].particle_steps, (unsigned long long)moved);
}

template <int R> constexpr size_t move_smem_bytes() { return sizeof(MoveSmem<R>) * M_WARPS; }

// ---- place_movers -----------------------------------------------------------

constexpr int P_WARPS = 4;
constexpr int W_WARPS = 4;
constexpr int WQ = 64;  // wall flights a warp collects: 31 left over and a turn's 32 fit

struct PlaceSmem {
    int2 q[WQ];  // {output slot, source cell}
    int qn;
};

struct MoveCounts {
    unsigned wall, reseed, stranded, err;
    int cross[3];
};
__device__ __forceinline__ void counts_reset(MoveCounts &c) {
    c.wall = c.reseed = c.stranded = c.err = 0;
    c.cross[0] = c.cross[1] = c.cross[2] = 0;
}
__device__ __forceinline__ void counts_add(MoveCounts &c, const MoveTally &t) {
    c.wall += (unsigned)t.wall_hits;
    c.reseed += (unsigned)t.reseeds;
    c.err |= t.err;
#pragma unroll
    for (int d = 0; d < 3; ++d) c.cross[d] += t.cross[d];
}
// Publishes the counts for system sys: the warp's sum (all lanes call) or,
// per_lane, each lane's own.
__device__ void counts_publish(const PassParams &P, int sys, MoveCounts &c, bool per_lane) {
    unsigned w = c.wall, r = c.reseed, s = c.stranded, e = c.err;
    int x[3] = {c.cross[0], c.cross[1], c.cross[2]};
    if (!per_lane) {
        w = warp_sum(w);
        r = warp_sum(r);
        s = warp_sum(s);
        e = __reduce_or_sync(0xffffffffu, e);
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = warp_sum(x[d]);
    }
    if ((per_lane || (threadIdx.x & 31) == 0) && sys >= 0) {
        SysTally &T = P.tally[sys];
        if (w) atomicAdd(&T.wall_hits, (unsigned long long)w);
        if (r) atomicAdd(&T.reseeds, (unsigned long long)r);
        if (s) atomicAdd(&T.stranded, (unsigned long long)s);
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (x[d]) atomicAdd((unsigned long long *)&T.count_periodic[d], (unsigned long long)(long long)x[d]);
    }
    if ((per_lane || (threadIdx.x & 31) == 0) && e) atomicOr(&P.status->error, e);
    counts_reset(c);
}

// Places one particle per valid lane into a top slot of cell `key`
// (warp-aggregated atomics).  A slot at or below the cell's input occupancy
// could meet its bottom segment or gap: that particle spills instead, and its
// slot is given back so the counter ends at the number placed.
__device__ __forceinline__ void insert_top(const PassParams &P, const Split32::Particle &p, bool valid,
                                           unsigned key, unsigned &err) {
    const int lane = threadIdx.x & 31;
    unsigned *top_out = P.cells.top[P.cout];
    const int2 rt = valid ? P.cells.room[key] : make_int2(0, 0);  // {first slot past the cell, room}
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? key : 0xffffffffu);
    const int leader = __ffs(peers) - 1;
    unsigned slot0 = 0;
    if (valid && lane == leader) slot0 = atomicAdd(&top_out[key], (unsigned)__popc(peers));
    slot0 = __shfl_sync(0xffffffffu, slot0, leader);
    bool spilled = false;
    if (valid) {
        const unsigned j = slot0 + (unsigned)__popc(peers & ((1u << lane) - 1u));
        uint4 ra;
        float4 rb;
        Split32::pack(p, ra, rb);
        if (j < (unsigned)rt.y) {
            const unsigned dst = (unsigned)rt.x - 1u - j;
            store_record(P.parts.A[P.cur ^ 1], dst, ra, rb);
        } else {
            spilled = true;
            const unsigned si = atomicAdd(&P.status->spill, 1u);
            if (si < P.parts.spill_cap) {
                SpillRec &sr = P.parts.spill[si];
                sr.a = ra;
                sr.b = *reinterpret_cast<const uint4 *>(&rb);
                sr.cell = (int)key;
            } else {
                err |= DSMC_EBIT_SPILL_FULL;
            }
        }
    }
    const unsigned over = __ballot_sync(0xffffffffu, spilled) & peers;
    if (valid && lane == leader && over) atomicSub(&top_out[key], (unsigned)__popc(over));
}

// Where a particle that completed its flight goes: its new active cell; or,
// when it ended inside solid whose cell has no free volume, its source cell
// (the reference aborts there, dsmc/system.h:134-142; the particle's next
// move re-seeds it, dsmc/moleculemover.cpp:57-60); or, in another slab's
// cell, the outgoing list (`leave`).  False only for the outgoing list.
__device__ __forceinline__ bool new_cell(const SysDev &g, const Split32::Particle &p, int src, unsigned &key,
                                         bool &leave, MoveCounts &cnt, unsigned &err) {
    const int ac = __ldg(g.cell_map + Split32::cell_global(g, p));
    leave = ac == DSMC_CELL_FOREIGN;
    if (ac >= 0) {
        key = (unsigned)ac;
    } else if (!leave) {
        err |= DSMC_EBIT_STRANDED;
        ++cnt.stranded;
        key = (unsigned)src;
    }
    return !leave;
}

// Appends the particles of the valid lanes to the outgoing list (one atomic
// per warp).  All lanes call.
__device__ __forceinline__ void leave_slab(const PassParams &P, const Split32::Particle &p, bool valid, unsigned &err) {
    const int lane = threadIdx.x & 31;
    const unsigned vm = __ballot_sync(0xffffffffu, valid);
    if (!vm) return;
    unsigned at = 0;
    if (lane == __ffs(vm) - 1) at = atomicAdd(&P.status->nout, (unsigned)__popc(vm));
    at = __shfl_sync(0xffffffffu, at, __ffs(vm) - 1) + (unsigned)__popc(vm & ((1u << lane) - 1u));
    if (valid) {
        if (at < P.parts.out_cap) {
            uint4 ra;
            float4 rb;
            Split32::pack(p, ra, rb);
            P.parts.out[2 * (size_t)at] = ra;
            P.parts.out[2 * (size_t)at + 1] = *reinterpret_cast<const uint4 *>(&rb);
        } else {
            err |= DSMC_EBIT_SPILL_FULL;
        }
    }
}

// Takes up to 32 of the warp's collected wall flights, one per lane (true in
// the lanes that got one).  All lanes call.
__device__ __forceinline__ bool pop_walls(PlaceSmem &W, int2 &e) {
    const int lane = threadIdx.x & 31;
    const int qn = W.qn, n = min(qn, 32);
    e = lane < n ? W.q[qn - n + lane] : make_int2(0, -1);
    __syncwarp();
    if (lane == 0) W.qn = qn - n;
    __syncwarp();
    return lane < n;
}

// Appends the valid lanes' wall flights to the list (one atomic).  All lanes call.
__device__ __forceinline__ void list_walls(const PassParams &P, int2 e, bool valid) {
    const int lane = threadIdx.x & 31;
    const int n = __popc(__ballot_sync(0xffffffffu, valid));  // the first n lanes
    unsigned at = 0;
    if (lane == 0 && n) at = atomicAdd(&P.status->walls, (unsigned)n);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (valid) {
        if (at + lane < P.parts.walls_cap) P.parts.walls[at + lane] = e;
        else atomicOr(&P.status->error, DSMC_EBIT_SPILL_FULL);  // cannot happen: one entry per slot at most
    }
}

// The general mover for the listed wall flights of the valid lanes, {output
// slot, source cell} each, then their placement.  All lanes call; tsys as
// counts_publish's.  CL: some system may have Cercignani-Lampis walls.
template <bool CL>
__device__ __forceinline__ void wall_flights(const PassParams &P, uint32_t move_step, int2 e, bool valid,
                                             MoveCounts &cnt, int &tsys) {
    const int esys = valid ? P.cells.meta[e.y].w : -1;
    const int csys = common_system(valid, esys);
    if (csys != tsys) {
        counts_publish(P, tsys, cnt, false);
        tsys = csys;
    }
    Split32::Particle p;
    MoveTally mt;
    mt.wall_hits = mt.reseeds = 0;
    mt.cross[0] = mt.cross[1] = mt.cross[2] = 0;
    mt.err = 0;
    unsigned key = 0;
    bool place = false, leave = false;
    if (valid) {
        uint4 ra;
        float4 rb;
        load_record(P.parts.A[P.cur ^ 1], e.x, ra, rb);
        Split32::unpack(ra, rb, p);
    }
    // the lanes of a warp share their system unless it is mixed; a mixed
    // warp moves its lanes one system at a time
    for (unsigned todo = __ballot_sync(0xffffffffu, valid); todo;) {
        const int sys = __shfl_sync(0xffffffffu, esys, __ffs(todo) - 1);
        const bool mine = valid && esys == sys;
        const SysDev &g = P.sys[sys];
        if (CL && g.wall_model == DSMC_WALL_CL)
            Split32::move_general_warp(g, p, move_step, mt, mine);
        else if (mine)
            Split32::move_general(g, p, move_step, mt);
        __syncwarp();
        todo &= ~__ballot_sync(0xffffffffu, mine);
    }
    if (valid) place = new_cell(P.sys[esys], p, e.y, key, leave, cnt, mt.err);
    insert_top(P, p, place, key, mt.err);
    leave_slab(P, p, leave, mt.err);
    counts_add(cnt, mt);
    if (tsys == -2) counts_publish(P, esys, cnt, true);
}

// The last block ends the pass: it advances the step and halts the pipeline
// if anything spilled or failed.
__device__ __forceinline__ void end_split_pass(const PassParams &P) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned done = atomicAdd(&P.status->blocks_done, 1u);
        if (done == gridDim.x - 1) {
            __threadfence();
            if (P.advance_step) atomicAdd(&P.status->step, 1u);
            if (atomicAdd(&P.status->spill, 0u) != 0u || (atomicAdd(&P.status->error, 0u) & DSMC_EBIT_FATAL) != 0u)
                atomicExch(&P.status->halted, 1u);
            atomicExch(&P.status->walls, 0u);
            atomicExch(&P.status->walls_taken, 0u);
            atomicExch(&P.status->collide_taken, 0u);
            atomicExch(&P.status->blocks_done, 0u);
        }
    }
}

// Bound by the latency of a mover's chain (record, voxel type, cell map, room,
// counter, store) over as many warps as fit: at 256^3 108, 103 and 99 us with
// five, seven and eight blocks per SM (77, 70 and 64 registers).
//
// OWN: a warp moves its own wall flights, 32 at a time and the rest at its end,
// and the kernel ends the pass; otherwise they go to place_walls' list.  The
// general mover takes 123 registers (four blocks per SM; held to 102 and 85,
// 45.2 and 46.8 us per step against 44.9 at 64^3), which costs the placing of
// many movers more than a launch and the list's turn-around: us per step, both
// kernels, list -> own: 64^3 (2e4 cells) 39 -> 28, 128^3 (2e5) 60 -> 49, 160^3
// (3.5e5) 76 -> 68 in all 226 -> 223, 192^3 (6e5) 92 -> 99, 256^3 162 -> 193. The
// rule (four chunks per warp, 3.0e5 cells on 148 SMs) lies below that crossing:
// 160^3 is listed.
// Cercignani-Lampis flights are always listed: their warps share the rejection
// trials, so equal claims matter more (64^3 69 -> 182, 128^3 119 -> 393).
template <bool OWN>
__global__ void __launch_bounds__(32 * P_WARPS, OWN ? 4 : 8) place_movers_kernel(const __grid_constant__ PassParams P) {
    __shared__ PlaceSmem smem[P_WARPS];
    const int lane = threadIdx.x & 31;
    const volatile Status *vs = P.status;
    if (vs->halted) return;
    const uint32_t move_step = vs->step + 1;
    PlaceSmem &W = smem[threadIdx.x >> 5];
    if (lane == 0) W.qn = 0;
    __syncwarp();
    const void *out = P.parts.A[P.cur ^ 1];

    MoveCounts cnt;
    counts_reset(cnt);
    int tsys = -1;

    // the flights collected so far: moved here (OWN), or appended to the list
    auto walls = [&]() {
        int2 e;
        const bool valid = pop_walls(W, e);
        if (OWN) wall_flights<false>(P, move_step, e, valid, cnt, tsys);
        else list_walls(P, e, valid);
    };
    const int C = P.cells.num_cells, CH = P.chunk;
    const int nchunks = (C + CH - 1) / CH;
    for (int ch = blockIdx.x * P_WARPS + (threadIdx.x >> 5); ch < nchunks; ch += gridDim.x * P_WARPS) {
        const int first = ch * CH;
        const bool mine = lane < min(CH, C - first);
        // lane i: the movers of cell i sit in output slots [gap, gap + cnt)
        int gap = 0, mv = 0, sys = -1;
        if (mine) {
            const int a = first + lane;
            const int4 m = P.cells.meta[a];
            unsigned nb, nt;
            input_counts(P, a, m, nb, nt);
            const unsigned nfs = min(P.cells.bot[P.cout][a], nb + nt);
            gap = m.x + (int)nfs;
            mv = (int)(nb + nt - nfs);
            sys = m.w;
        }
        // exclusive prefix of the mover counts over the chunk's cells
        int incl = mv;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const int pre = mine ? incl - mv : 0x7fffffff;
        for (int f0 = 0; f0 < total; f0 += 32) {
            const int f = f0 + lane;
            const bool valid = f < total;
            // cell of mover f: the last cell whose prefix is <= f
            int c = 0;
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                const int pc = __shfl_sync(0xffffffffu, pre, (c + s) & 31);
                if (c + s < 32 && pc <= f) c += s;
            }
            const int slot = __shfl_sync(0xffffffffu, gap, c) + (f - __shfl_sync(0xffffffffu, pre, c));
            const int psys = __shfl_sync(0xffffffffu, sys, c);
            const int src = first + c;  // the mover's cell
            const int csys = common_system(valid, psys);
            if (csys != tsys) {
                counts_publish(P, tsys, cnt, false);
                tsys = csys;
            }
            Split32::Particle p;
            MoveTally mt;
            mt.wall_hits = mt.reseeds = 0;
            mt.cross[0] = mt.cross[1] = mt.cross[2] = 0;
            mt.err = 0;
            bool done = false, place = false, leave = false;
            unsigned key = 0;
            if (valid) {
                uint4 ra;
                float4 rb;
                load_record(out, slot, ra, rb);
                Split32::unpack(ra, rb, p);
                const SysDev &g = P.sys[psys];
                done = Split32::move_open(g, p, mt);
                if (done) place = new_cell(g, p, src, key, leave, cnt, mt.err);
            }
            // flights that meet a wall stay in their slot for place_walls
            const unsigned wall = __ballot_sync(0xffffffffu, valid && !done);
            if (wall) {
                if (valid && !done) W.q[W.qn + __popc(wall & ((1u << lane) - 1u))] = make_int2(slot, src);
                __syncwarp();
                if (lane == 0) W.qn += __popc(wall);
                __syncwarp();
            }
            insert_top(P, p, place, key, mt.err);
            leave_slab(P, p, leave, mt.err);
            counts_add(cnt, mt);
            if (tsys == -2) counts_publish(P, psys, cnt, true);
            if (W.qn >= 32) walls();
        }
    }
    if (W.qn) walls();
    counts_publish(P, tsys, cnt, false);
    if (OWN) end_split_pass(P);
}

// The general mover for every listed wall flight, one per lane, then the
// placement.  Bound by the longest flight's serial chain (ten reflections of
// about 2 us each) and, with many flights, by the divergence of a warp's.
// Measured, us per step at 64^3 (2e3 flights) / 128^3 (1.8e4) / 256^3 (1.5e5):
// a warp-wide state machine with claims of 32 42 / 61 / 93; claims sized to the
// grid, draws and frames overlapped 35 / 47 / 78; each flight on its own lane,
// without the machine, 27 / 35 / 65.  With Cercignani-Lampis walls (128^3,
// alpha_n = 0.8) 524, with the trials shared by the warp 91.  Held to fewer
// registers (128, 102, 85 for 4, 5, 6 blocks per SM) the machine spilled: 37, 40
// and 44 us at 64^3.
__global__ void __launch_bounds__(32 * W_WARPS) place_walls_kernel(const __grid_constant__ PassParams P) {
    const int lane = threadIdx.x & 31;
    const volatile Status *vs = P.status;
    if (vs->halted) return;
    const uint32_t move_step = vs->step + 1;
    const unsigned nwalls = min(vs->walls, P.parts.walls_cap);
    MoveCounts cnt;
    counts_reset(cnt);
    int tsys = -1;
    // Warps claim entries from a counter: flights differ widely in length, so
    // a warp that finishes early takes more.  A claim is 32 entries, or fewer
    // when the list would not fill the grid's warps: a warp's lanes wait for one
    // another where their flights part (and, with Cercignani-Lampis walls, take turns
    // in the state machine), so a warp of few lanes finishes its flights sooner.
    const unsigned nw = gridDim.x * W_WARPS;
    const unsigned claim = min(32u, max(1u, (nwalls + nw - 1u) / nw));
    for (;;) {
        unsigned i0 = 0;
        if (lane == 0) i0 = atomicAdd(&P.status->walls_taken, claim);
        i0 = __shfl_sync(0xffffffffu, i0, 0);
        if (i0 >= nwalls) break;
        const unsigned i = i0 + lane;
        const bool valid = (unsigned)lane < claim && i < nwalls;
        const int2 e = valid ? P.parts.walls[i] : make_int2(0, -1);  // {slot, source cell}
        wall_flights<true>(P, move_step, e, valid, cnt, tsys);
    }
    counts_publish(P, tsys, cnt, false);
    end_split_pass(P);
}

// ---- slab exchange ----------------------------------------------------------

// Records that arrive from another slab (the receiving side of the
// reference's mpi_move, dsmc/system.cpp:49-105): each goes into the top
// segment of its cell, above the bottom segment, or into the overflow list
// (the host then repacks).  A record outside this system's cells is an error.
__global__ void put_records_kernel(const SysDev *sys, int s, const CellArrays cells, const ParticleArrays parts,
                                   int cur, int cin, long long n, const uint4 *rec, Status *status) {
    const SysDev &g = sys[s];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const uint4 ra = rec[2 * i];
        const uint4 rbits = rec[2 * i + 1];
        const float4 rb = *reinterpret_cast<const float4 *>(&rbits);
        Split32::Particle p;
        Split32::unpack(ra, rb, p);
        if (p.c[0] < 0 || p.c[0] >= g.n[0] || p.c[1] >= g.n[1] || p.c[2] >= g.n[2]) {
            atomicOr(&status->error, DSMC_EBIT_CELL);
            continue;
        }
        const int ac = __ldg(g.cell_map + Split32::cell_global(g, p));
        if (ac < 0) {
            atomicOr(&status->error, DSMC_EBIT_CELL);
            continue;
        }
        const int4 m = cells.meta[ac];
        const unsigned nb = min(cells.bot[cin][ac], (unsigned)m.y);
        const unsigned j = atomicAdd(&cells.top[cin][ac], 1u);
        if (nb + j < (unsigned)m.y) {
            const unsigned dst = (unsigned)(m.x + m.y) - 1u - j;
            store_record(parts.A[cur], dst, ra, rb);
        } else {
            atomicSub(&cells.top[cin][ac], 1u);
            const unsigned si = atomicAdd(&status->spill, 1u);
            if (si < parts.spill_cap) {
                SpillRec &sr = parts.spill[si];
                sr.a = ra;
                sr.b = rbits;
                sr.cell = ac;
            } else {
                atomicOr(&status->error, DSMC_EBIT_SPILL_FULL);
            }
        }
    }
}

}  // namespace pass3
}  // namespace dsmc
