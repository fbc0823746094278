// Spatial sort, cell binning and neighbour-list build (the GPU replacement of
// the reference's Voronoi tessellation + k-d tree + Morton reorder:
// src/voronoi.h:143-237, src/kdtree.h:117-285, src/reorder_morton.h:44-122,
// src/reorder.h:33-149), plus state conversion between the caller's AoS
// double arrays and the device layout.
//
// Rebuild chain (runs only when a particle moved more than skin/2 since the
// last build, or on demand):
//   k_rebin          re-express each position in the cell that now holds it,
//                    clear the old cell ranges, count cells and tiles
//   k_tile_scan      prefix of the particles per tile of 64 cells
//   k_tile_cells     [begin, end) of each occupied cell
//   k_place, k_rank  slots by cell, in the order of their old slots
//   k_gather         the physical reorder of all per-particle arrays (bond /
//                    face partners remapped)
//   k_nlist          full neighbour list per particle from the 27 cells
//                    around its own; the last block flips buffer parities
#include "orbc_device.cuh"

#include <algorithm>
#include <cstdio>
#include <type_traits>

namespace orbc {

namespace {

__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }


__device__ __forceinline__ int gate_closed(const int *gate) { return gate && !__ldcg(gate); }

}  // namespace

/* ------------------------------------------------------------------------- */
/* LSD radix sort of (uint32 key, int value) pairs, 8-bit digits, stable.     */
/* One 4096-key tile per block: histogram -> per-digit scan over tiles ->    */
/* stable in-tile ranking (warp match + per-warp digit counts) and scatter.  */
/* ------------------------------------------------------------------------- */
__global__ void __launch_bounds__(256) k_rs_hist(const uint32_t *keys, int64_t n, int shift, int *counts,
                                                  int ntiles) {
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = int64_t(blockIdx.x) * SORT_TILE;
#pragma unroll 4
    for (int k = 0; k < SORT_TILE / 256; ++k) {
        const int64_t idx = base + k * 256 + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 255u], 1);
    }
    __syncthreads();
    counts[int64_t(threadIdx.x) * ntiles + blockIdx.x] = h[threadIdx.x];
}

__global__ void __launch_bounds__(1024) k_rs_scan(int *counts, int ntiles, int *digit_total) {
    __shared__ int wsum[32];
    __shared__ int carry;
    int *row = counts + int64_t(blockIdx.x) * ntiles;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < ntiles; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < ntiles ? row[i] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int s = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            wsum[lane] = s;
        }
        __syncthreads();
        const int incl = x + (warp > 0 ? wsum[warp - 1] : 0);
        const int c0 = carry;
        if (i < ntiles) row[i] = c0 + incl - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry = c0 + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) digit_total[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(256) k_rs_scatter(const uint32_t *kin, const int *vin, uint32_t *kout, int *vout,
                                                     int64_t n, int shift, const int *counts, int ntiles,
                                                     const int *digit_total) {
    __shared__ int base_s[256];
    __shared__ int run[256];
    __shared__ int wcnt[8][256];
    __shared__ int wsum[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // exclusive scan of the digit totals -> global digit base
    {
        const int v = digit_total[t];
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        int off = 0;
        for (int w = 0; w < warp; ++w) off += wsum[w];
        base_s[t] = off + x - v + counts[int64_t(t) * ntiles + blockIdx.x];
        run[t] = 0;
    }
    const unsigned lt = (1u << lane) - 1u;
    const int64_t tb = int64_t(blockIdx.x) * SORT_TILE;
    for (int r = 0; r < SORT_TILE / 256; ++r) {
#pragma unroll
        for (int k = 0; k < 8; ++k) wcnt[k][t] = 0;
        __syncthreads();
        const int64_t idx = tb + r * 256 + t;
        const bool valid = idx < n;
        const uint32_t key = valid ? kin[idx] : 0u;
        const int val = valid ? vin[idx] : 0;
        const int dg = valid ? int((key >> shift) & 255u) : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, dg);
        const int rank = __popc(peers & lt);
        if (valid && lane == __ffs(peers) - 1) wcnt[warp][dg] = __popc(peers);
        __syncthreads();
        {
            int acc = run[t];
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const int c = wcnt[w][t];
                wcnt[w][t] = acc;
                acc += c;
            }
            run[t] = acc;
        }
        __syncthreads();
        if (valid) {
            const int pos = base_s[dg] + wcnt[warp][dg] + rank;
            kout[pos] = key;
            vout[pos] = val;
        }
        __syncthreads();
    }
}

int sort_tiles(int64_t n) { return int((n + SORT_TILE - 1) / SORT_TILE); }

int radix_sort_pairs(uint32_t *keys[2], int *vals[2], int *counts, int *digit_total, int64_t n, int passes, int ntiles,
                     cudaStream_t st) {
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        k_rs_hist<<<ntiles, 256, 0, st>>>(keys[cur], n, shift, counts, ntiles);
        k_rs_scan<<<256, 1024, 0, st>>>(counts, ntiles, digit_total);
        k_rs_scatter<<<ntiles, 256, 0, st>>>(keys[cur], vals[cur], keys[1 - cur], vals[1 - cur], n, shift, counts,
                                             ntiles, digit_total);
        cur = 1 - cur;
    }
    return cur;
}

/* ------------------------------------------------------------------------- */
/* Rebuild chain                                                             */
/* ------------------------------------------------------------------------- */
/* The particles are ordered by (cell id, old slot) without sorting keys: cells
 * are counted, tiles of 64 cells are scanned, and the handful of particles of a
 * cell are ranked by their old slot.  An LSD radix sort of the ids (three or
 * four passes of three kernels) took 58 us for 33 thousand particles and 190 us for
 * 4.0M, most of it launches and serial scans. */
template<class R> __global__ void __launch_bounds__(256) k_rebin(KArgs<R> a, int gated) {
    using T4 = typename Vec<R>::T4;
    if (gated && !__ldcg(&a.S->rebuild)) return;
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.S->max_nnb = 0;
        a.S->out_of_grid = 0;
    }
    int out = 0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // npad is a multiple of the block size
    const int s = a.blk_sys[i / SYS_PAD];
    const SysDev &sd = a.sys[s];
    T4 p = a.pos[cur][i];
    const bool real = w_type(wbits(p.w)) != GHOST;
    uint32_t key = 0xffffffffu;
    if (real) {
        const int c = a.cell[lp][i];
        int cc[3] = {cx_of(c), cy_of(c), cz_of(c)};
        a.ranges[sd.cell_base + cell_code(sd, cc[0], cc[1], cc[2])] = make_int2(0, 0);
        R o[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const R L = lc_of<R>(sd, d);
            const R invL = inv_lc_of<R>(sd, d);
            const int k = int(floor(add_rn(mul_rn(o[d], invL), R(0.5))));
            int nc = cc[d] + k;
            if (sd.per[d]) {
                o[d] = sub_rn(o[d], mul_rn(R(k), L));
                nc %= sd.nc[d];
                if (nc < 0) nc += sd.nc[d];
            } else {
                const int cl = min(max(nc, 0), sd.nc[d] - 1);
                if (cl != nc) out = 1;
                o[d] = sub_rn(o[d], mul_rn(R(cl - cc[d]), L));
                nc = cl;
            }
            cc[d] = nc;
        }
        p.x = o[0];
        p.y = o[1];
        p.z = o[2];
        a.pos[cur][i] = p;  // the gather that follows sets the displacement reference
        a.cell[lp][i] = cpack(cc[0], cc[1], cc[2]);
        key = sd.cell_base + cell_code(sd, cc[0], cc[1], cc[2]);
    }
    a.skey[0][i] = key;
    // one atomic per cell and per tile of the warp (its particles sit in a few
    // cells); ghosts take the places behind the system's particles
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(int(peers)) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(real ? a.ccnt + key : a.gcnt + s, __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    a.sval[1][i] = base + __popc(peers & ((1u << lane) - 1u));
    const unsigned tpeers = __match_any_sync(0xffffffffu, key >> 6);
    if (real && lane == __ffs(int(tpeers)) - 1) atomicAdd(a.tcnt + (key >> 6), __popc(tpeers));
    if (out) {
        atomicOr(&a.S->error, ERRB_GRID);
        atomicAdd(&a.S->out_of_grid, 1);
    }
}

constexpr int SCAN_GRID = NUM_SM * 2;  // resident blocks of the tile scan
/* Exclusive prefix of the tiles' particle counts inside each block of
 * SCAN_TILES; the last block to finish turns the block totals into prefixes.
 * The grid is bounded (SCAN_GRID), as an open system with a stray particle may have
 * 10^9 cells, almost all of them empty: 1.7e9 cells, 2,000 particles, rebuild 187 ->
 * 102 us, and the launches of a chain that finds the gate closed 230 -> 44. */
__global__ void __launch_bounds__(1024) k_tile_scan(const int *tcnt, int *tstart, int *bsum, int nscan,
                                                    unsigned int *counter, const int *gate) {
    if (gate_closed(gate)) return;
    __shared__ int wsum[32];
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // inclusive prefix of v over the block; total in wsum[31]
    auto scan = [&](int v) {
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int w = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        return x + (warp > 0 ? wsum[warp - 1] : 0);
    };
    auto load = [&](int b) {
        return b < nscan ? reinterpret_cast<const int4 *>(tcnt)[int64_t(b) * (SCAN_TILES / 4) + t] : make_int4(0, 0, 0, 0);
    };
    int4 c = load(blockIdx.x);
    for (int b = blockIdx.x; b < nscan; b += gridDim.x) {
        const int4 next = load(b + gridDim.x);
        const int sum = c.x + c.y + c.z + c.w;
        int total = 0;
        if (__syncthreads_or(sum)) {  // the prefixes of empty tiles are not read
            const int e = scan(sum) - sum;
            reinterpret_cast<int4 *>(tstart)[int64_t(b) * (SCAN_TILES / 4) + t] =
                make_int4(e, e + c.x, e + c.x + c.y, e + c.x + c.y + c.z);
            total = wsum[31];
        }
        if (t == 0) bsum[b] = total;
        c = next;
    }
    if (t == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int carry = 0;
    for (int b0 = 0; b0 < nscan; b0 += 1024) {
        const int v = b0 + t < nscan ? __ldcg(bsum + b0 + t) : 0;
        const int x = scan(v);
        if (b0 + t < nscan) bsum[b0 + t] = carry + x - v;
        carry += wsum[31];
        __syncthreads();  // wsum is read by all before the next scan
    }
    if (t == 0) *counter = 0;
}

/* Ranges of the occupied cells, one warp per 32 tiles; the counts go back to
 * zero. */
template<class R> __global__ void __launch_bounds__(256) k_tile_cells(KArgs<R> a, int gated) {
    if (gated && !__ldcg(&a.S->rebuild)) return;
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0)
        for (int s = threadIdx.x; s < a.nsys; s += blockDim.x) a.gcnt[s] = 0;
    const int stride = int(gridDim.x) * 256;
    for (int t0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 32; t0 < a.nctile; t0 += stride) {
        if (stride < a.nctile) {  // scan blocks without particles are passed over
            const int b = t0 / SCAN_TILES;
            if (b + 1 < a.nscan && a.bsum[b] == a.bsum[b + 1]) continue;
        }
        const int n = a.tcnt[t0 + lane];  // nctile is a multiple of 32
        const int start = n ? a.tstart[t0 + lane] + a.bsum[(t0 + lane) / SCAN_TILES] : 0;
        if (n) a.tcnt[t0 + lane] = 0;
        for (unsigned m = __ballot_sync(0xffffffffu, n != 0); m; m &= m - 1u) {
            const int l = __ffs(int(m)) - 1;
            const int64_t id0 = int64_t(t0 + l) * 64;
            int lo = 0, hi = a.nsys - 1;  // the system whose ids these are
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (int64_t(a.sys[mid].cell_base) <= id0)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const int base = __shfl_sync(0xffffffffu, start, l) + a.sys[lo].slot_shift;
            const int c0 = a.ccnt[id0 + 2 * lane], c1 = a.ccnt[id0 + 2 * lane + 1];
            int x = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            const int b = base + x - c0 - c1;
            if (c0) {
                a.ranges[id0 + 2 * lane] = make_int2(b, b + c0);
                a.ccnt[id0 + 2 * lane] = 0;
            }
            if (c1) {
                a.ranges[id0 + 2 * lane + 1] = make_int2(b + c0, b + c0 + c1);
                a.ccnt[id0 + 2 * lane + 1] = 0;
            }
        }
    }
}

/* Slots by cell in arrival order, then each slot's place by its rank among
 * the old slots of its cell. */
template<class R> __global__ void __launch_bounds__(256) k_place(KArgs<R> a, int gated) {
    if (gated && !__ldcg(&a.S->rebuild)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t key = a.skey[0][i];
    if (key != 0xffffffffu) a.skey[1][a.ranges[key].x + a.sval[1][i]] = uint32_t(i);
}
template<class R> __global__ void __launch_bounds__(256) k_rank(KArgs<R> a, int gated) {
    if (gated && !__ldcg(&a.S->rebuild)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t key = a.skey[0][i];
    int p;
    if (key == 0xffffffffu) {
        const SysDev &sd = a.sys[a.blk_sys[i / SYS_PAD]];
        p = sd.off + sd.nreal + a.sval[1][i];
    } else {
        const int2 rg = a.ranges[key];
        p = rg.x;
        for (int q = rg.x; q < rg.y; ++q) p += a.skey[1][q] < uint32_t(i) ? 1 : 0;
    }
    a.sval[0][p] = i;
    a.inv[i] = p;
}

template<class R> __global__ void __launch_bounds__(256) k_gather(KArgs<R> a, int gated) {
    if (gated && !__ldcg(&a.S->rebuild)) return;
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    const int nc = 1 - cur, nl = 1 - lp;
    const int *sv = a.sval[0];
    const int n = a.npad;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        // every load of the slot before its first store: the stores may alias
        // the loads as far as the compiler knows, and would serialise them
        const int src = sv[p];
        const auto ps = a.pos[cur][src];
        const auto ns = a.nrm[cur][src];
        const auto vs = a.vel[lp][src];
        const auto os = a.omg[lp][src];
        const int cs = a.cell[lp][src], ts = a.tag[lp][src], h = a.home[lp][src];
        if (a.carry_forces) {  // Nose-Hoover carries f and t from one half-step to the next
            const auto fs = a.frc[lp][src], qs = a.trq[lp][src];
            a.frc[nl][p] = fs;
            a.trq[nl][p] = qs;
        }
        a.pos[nc][p] = ps;
        a.nrm[nc][p] = ns;
        a.vel[nl][p] = vs;
        a.omg[nl][p] = os;
        a.xref[nl][p] = ps;  // the list about to be built is referenced to these positions
        a.cell[nl][p] = cs;
        a.tag[nl][p] = ts;
        a.home[nl][p] = h;
        if (h >= 0) a.slot_of_home[h] = p;
        const int w = wbits(ps.w);
        const int bd = w_bdeg(w), fd = w_fdeg(w);
        for (int b = 0; b < bd; ++b) {
            BondSlot s = a.bond[lp][int64_t(b) * n + src];
            s.partner = a.inv[s.partner];
            a.bond[nl][int64_t(b) * n + p] = s;
        }
        for (int b = 0; b < fd; ++b) {
            int2 s = a.fslot[lp][int64_t(b) * n + src];
            s.x = a.inv[s.x];
            s.y = a.inv[s.y];
            a.fslot[nl][int64_t(b) * n + p] = s;
        }
    }
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < a.nfaces; f += gridDim.x * blockDim.x) {
        int4 q = a.faces[f];
        q.x = a.inv[q.x];
        q.y = a.inv[q.y];
        q.z = a.inv[q.z];
        a.faces[f] = q;
    }
}

/* End of a list build: block max of the candidate counts -> global max and
 * overflow flag; the last block to finish makes the new buffers current and
 * clears the rebuild request. */
template<class R> __device__ __forceinline__ void nlist_finalise(const KArgs<R> &a, int maxc, int cur, int lp) {
    __shared__ int smax[8];
    __shared__ bool last;
    int m = maxc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        int bm = 0;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) bm = max(bm, smax[w]);
        atomicMax(&a.S->max_nnb, bm);
        if (bm > a.cap) atomicOr(&a.S->error, ERRB_NBR_OVERFLOW);
        __threadfence();
        const unsigned ticket = atomicAdd(&a.S->blk_counter, 1u);
        last = (ticket == gridDim.x - 1);
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        a.S->cur = cur;
        a.S->lp = lp;
        a.S->rebuild = 0;
        a.S->rebuilds += 1;
        a.S->since_rebuild = 0;
        a.S->blk_counter = 0;
        __threadfence();
    }
}

/* Neighbour list, in two phases per warp.  For each distinct cell of a
 * warp's particles 27 lanes fetch the neighbour cells' ranges and the
 * candidates are staged pre-shifted into that cell's frame, padded (never
 * accepted) to a multiple of 32.  Phase 1: for two particles of the cell at a
 * time the warp tests 32 candidates per ballot pair, branch-free (one staged
 * load serves both particles), and each particle's own lane keeps the accept
 * masks (in range at all / inside the interaction range) in registers; where
 * particles and candidates are of types 0..3, which share one list cutoff, the
 * cutoffs are two registers instead of two table lookups per test.  The
 * candidates' list entries stay staged in shared memory for as many cells as
 * fit, so that phase 2 -- every lane expands its masks in candidate order into
 * its own column, inner rows upwards and shell rows downwards -- runs for most
 * warps once, with all their lanes.
 *
 * SW warps share 32 slots, each taking 32 / SW of their particles: one warp's
 * chain of cells, ballots and expansions is some 80 thousand cycles long, which
 * is the time of the build while the GPU is not full. */
// Bound by instruction issue (69 % of peak) and each warp's chain; FP64: by the FP64 pipe (86 %).  1.0M-particle
// cell 0.357 -> 0.266 ms, 4.03M 1.34 -> 0.98, 1.0M lipids in 23 vesicles 0.359 ->
// 0.279 against table lookups, searched staging and blocks of four warps; a third
// copy of phase 1 for lipids alone made the cell with anchors slower (0.379 ms:
// the instruction cache).
// 28 resident warps per SM: the staging below (about 15 KB per block) and at
// most 72 registers (FP64: 24 and 80, where 72 spill); more warps in flight beat
// fewer passes per warp.  Blocks of two warps: one of four holds its memory until
// its slowest warp is done (4.03M 1.08 ms), single warps fit only 26 (1.10 ms).
constexpr int NLW = 2;  // warps per block of the list build
template<class R> constexpr int nlist_warps = sizeof(R) == 8 ? 24 : 28;  // resident per SM
template<class R, int SW> __global__ void __launch_bounds__(32 * NLW, nlist_warps<R> / NLW) k_nlist(KArgs<R> a, int gated) {
    using T4 = typename Vec<R>::T4;
    if (gated && !__ldcg(&a.S->rebuild)) return;
    constexpr int MB = 8;                                 // accept masks (32 candidates each) per lane
    constexpr int REG = 32 * MB;                          // candidates of one cell (or chunk) per phase 1
    constexpr int SU = 2;                                 // blocks of 32 candidates staged together
    constexpr int SE = 704;                               // list entries staged per warp until phase 2
    __shared__ float4 s_pos[NLW][REG];                    // the current cell's candidates (FP64: rounded)
    __shared__ uint32_t s_ent[NLW][SE];                   // j | shift code of its cell << NB_SHIFT
    __shared__ float4 s_seg[NLW][27];                     // occupied neighbour cells: shift, first slot - first candidate
    __shared__ uint32_t s_code[NLW][27];                  // and their shift code << NB_SHIFT
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // (list cutoff^2, inner cutoff^2) of a type pair
    auto cuts = [&](int k) { return make_float2(__ldg(&a.ff->rlist2[k]), __ldg(&a.ff->rin2[k])); };
    const int cur = 1 - __ldcg(&a.S->cur), lp = 1 - __ldcg(&a.S->lp);
    // the grid covers npad (a multiple of the block size) SW times
    const int wid = blockIdx.x * NLW + warp;
    const int i = wid / SW * 32 + lane;
    const bool mine = SW == 1 || lane / (32 / SW) == wid % SW;
    const T4 p = a.pos[cur][i];
    const int ty = w_type(wbits(p.w));
    const bool real = ty != GHOST && mine;
    const SysDev &sd = a.sys[a.blk_sys[i / SYS_PAD]];  // one system per warp (SYS_PAD-aligned)
    const int c = a.cell[lp][i];
    const int cc[3] = {cx_of(c), cy_of(c), cz_of(c)};
    const R L[3] = {lc_of<R>(sd, 0), lc_of<R>(sd, 1), lc_of<R>(sd, 2)};
    // Candidate j seen from i's cell: o_j + d * Lc (d = cell_j - cell_i);
    // x_i - x_j = o_i - (o_j + d * Lc).
    auto shifted = [&](const T4 &q, int dx, int dy, int dz) {
        T4 r = q;
        r.x = q.x + R(dx) * L[0];
        r.y = q.y + R(dy) * L[1];
        r.z = q.z + R(dz) * L[2];
        return r;
    };
    auto dist2 = [&](const T4 &pi, const T4 &qs) {
        const R ex = pi.x - qs.x, ey = pi.y - qs.y, ez = pi.z - qs.z;
        return ex * ex + ey * ey + ez * ez;
    };
    // FP64: the two comparisons of a test are decided in FP32 (from rounded positions) unless r^2 lies within the
    // rounding of a cutoff for some lane.  Some 124 FP64 tests per particle otherwise bound the build: 250 thousand
    // particle cell 0.84 -> 0.15 ms
    const float slack = sizeof(R) == 8 ? rounding_slack(sd) : 0.f;
    // ballots of r^2 < cut.x, cut.y for candidate q of lane; et: its list entry (FP64)
    auto inside = [&](const T4 &pi, const float4 &pf, const float4 &q, const float2 &cut, const uint32_t *et, bool pad,
                      unsigned &ma, unsigned &mi) {
        const float ex = pf.x - q.x, ey = pf.y - q.y, ez = pf.z - q.z;
        const float r2 = ex * ex + ey * ey + ez * ez;
        ma = __ballot_sync(0xffffffffu, r2 < cut.x);
        mi = __ballot_sync(0xffffffffu, r2 < cut.y);
        if constexpr (sizeof(R) == 8) {
            const bool near = fabsf(r2 - cut.x) < slack * cut.x || fabsf(r2 - cut.y) < slack * cut.y;
            if (__any_sync(0xffffffffu, near)) {
                R d2 = R(1e30);
                if (!pad) {
                    const int l = int(*et >> NB_SHIFT);
                    d2 = dist2(pi, shifted(a.pos[cur][*et & NB_MASK], l % 3 - 1, (l / 3) % 3 - 1, l / 9 - 1));
                }
                ma = __ballot_sync(0xffffffffu, d2 < R(cut.x));
                mi = __ballot_sync(0xffffffffu, d2 < R(cut.y));
            }
        }
    };
    const int kme = cc[0] | (cc[1] << 11) | (cc[2] << 22);
    float4 *seg = s_seg[warp];
    uint32_t *code = s_code[warp];
    float4 *sp = s_pos[warp];
    uint32_t *se = s_ent[warp];
    uint32_t *col = a.nbr + nbr_index(i, 0, a.cap);  // row k of slot i at col[32 k]
    const int cap = a.cap;
    const float2 cut_ll = cuts(0);
    int qin = 0, qout = 0, qtot = 0;
    // neighbour ranges of cell kd: this lane's candidates [first, first + cnt) of the cell's; the occupied
    // cells' table; returns the candidate count.  own_first: where the centre cell's candidates begin
    int first = 0, cnt = 0, own_first = 0, own_slot = 0;
    auto fetch = [&](int kd) {
        const int xd = kd & 2047, yd = (kd >> 11) & 2047, zd = (kd >> 22) & 1023;
        int2 rg = make_int2(0, 0);
        if (lane < 27) {
            int x = xd + lane % 3 - 1, y = yd + (lane / 3) % 3 - 1, z = zd + lane / 9 - 1;
            bool ok = true;
            if (sd.per[0]) x = x < 0 ? x + sd.nc[0] : (x >= sd.nc[0] ? x - sd.nc[0] : x);
            else ok = ok && x >= 0 && x < sd.nc[0];
            if (sd.per[1]) y = y < 0 ? y + sd.nc[1] : (y >= sd.nc[1] ? y - sd.nc[1] : y);
            else ok = ok && y >= 0 && y < sd.nc[1];
            if (sd.per[2]) z = z < 0 ? z + sd.nc[2] : (z >= sd.nc[2] ? z - sd.nc[2] : z);
            else ok = ok && z >= 0 && z < sd.nc[2];
            if (ok) rg = a.ranges[sd.cell_base + cell_code(sd, x, y, z)];
        }
        cnt = rg.y > rg.x ? rg.y - rg.x : 0;
        int inc = cnt;  // inclusive warp scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        first = inc - cnt;
        own_first = __shfl_sync(0xffffffffu, first, 13);
        own_slot = __shfl_sync(0xffffffffu, rg.x, 13);
        const unsigned occ = __ballot_sync(0xffffffffu, cnt > 0);
        __syncwarp();  // the previous cell's staging is done with the table
        if (cnt > 0) {
            const int r = __popc(occ & ((1u << lane) - 1u));
            seg[r] = make_float4(float(lane % 3 - 1) * sd.Lcf[0], float((lane / 3) % 3 - 1) * sd.Lcf[1],
                                 float(lane / 9 - 1) * sd.Lcf[2], __int_as_float(rg.x - first));
            code[r] = uint32_t(lane) << NB_SHIFT;
        }
        __syncwarp();
        return __shfl_sync(0xffffffffu, inc, 31);
    };
    // candidates [c0, c0 + nch) of the fetched cell -> sp[0 ...] and se[ebase ...]; the or of their types
    // (c0 a multiple of 32).  A candidate's cell is the number of occupied cells that begin at or before it: a
    // population count on the mask of beginnings in its block of 32, where a search over the 27 offsets
    // takes five dependent lookups
    auto stage = [&](int c0, int nch, int ebase) {
        unsigned types = 0;
        int before = __popc(__ballot_sync(0xffffffffu, cnt > 0 && first < c0));
        for (int t0 = 0; t0 < nch; t0 += 32 * SU) {
            int r[SU], j[SU];
            float4 g[SU];
            T4 q[SU];
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                const int b = (t0 >> 5) + u;
                const unsigned begins =
                    __reduce_or_sync(0xffffffffu, cnt > 0 && (first - c0) >> 5 == b ? 1u << (first & 31) : 0u);
                r[u] = before + __popc(begins & (0xffffffffu >> (31 - lane))) - 1;
                before += __popc(begins);
            }
#pragma unroll
            for (int u = 0; u < SU; ++u) {  // every load of the batch before its first store
                g[u] = seg[r[u]];
                j[u] = t0 + 32 * u + lane < nch ? c0 + t0 + 32 * u + lane + __float_as_int(g[u].w) : i;
                q[u] = a.pos[cur][j[u]];
            }
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                const int t = t0 + 32 * u + lane;
                if (t < nch) {
                    const int tj = w_type(wbits(q[u].w));
                    types |= tj;
                    sp[t] = make_float4(float(q[u].x) + g[u].x, float(q[u].y) + g[u].y, float(q[u].z) + g[u].z,
                                        __int_as_float(tj));
                    se[ebase + t] = uint32_t(j[u]) | code[r[u]];
                }
            }
        }
        if (nch + lane < ((nch + 31) & ~31)) {  // far away: never accepted
            sp[nch + lane] = make_float4(1e18f, 1e18f, 1e18f, 0.f);
        }
        __syncwarp();
        return __reduce_or_sync(0xffffffffu, types);
    };
    uint32_t macc[MB], minn[MB];
    // phase 1 for the particles grp, two per pass, over the staged candidates [0, nch), nch <= REG.
    // ONE: one list and one inner cutoff; otherwise cutoffs by type pair
    auto phase1 = [&](unsigned grp, int nch, int ebase, auto one_cutoff) {
        constexpr bool ONE = decltype(one_cutoff)::value;
        for (unsigned g = grp; g;) {
            const int il = __ffs(int(g)) - 1;
            g &= g - 1u;
            const int il2 = g ? __ffs(int(g)) - 1 : il;  // the second particle of the pass (il again if none)
            if (g) g &= g - 1u;
            T4 pi = p, pi2 = p;
            pi.x = __shfl_sync(0xffffffffu, p.x, il);
            pi.y = __shfl_sync(0xffffffffu, p.y, il);
            pi.z = __shfl_sync(0xffffffffu, p.z, il);
            pi2.x = __shfl_sync(0xffffffffu, p.x, il2);
            pi2.y = __shfl_sync(0xffffffffu, p.y, il2);
            pi2.z = __shfl_sync(0xffffffffu, p.z, il2);
            const float4 pf = make_float4(float(pi.x), float(pi.y), float(pi.z), 0.f),
                         pf2 = make_float4(float(pi2.x), float(pi2.y), float(pi2.z), 0.f);
            const int ti = ONE ? 0 : __shfl_sync(0xffffffffu, ty, il) * 16;
            const int ti2 = ONE ? 0 : __shfl_sync(0xffffffffu, ty, il2) * 16;
#pragma unroll
            for (int b = 0; b < MB; ++b) {
                if (b * 32 < nch) {
                    const float4 q = sp[b * 32 + lane];
                    const int tj = ONE ? 0 : w_type(wbits(q.w));
                    const uint32_t *et = se + ebase + b * 32 + lane;
                    const bool pad = b * 32 + lane >= nch;
                    const float2 cut = ONE ? cut_ll : cuts(ti + tj);
                    const float2 cut2 = ONE ? cut_ll : cuts(ti2 + tj);
                    // inner cutoff <= list cutoff; a particle's own bit is cleared in phase 2
                    unsigned ma, mi, ma2, mi2;
                    inside(pi, pf, q, cut, et, pad, ma, mi);
                    inside(pi2, pf2, q, cut2, et, pad, ma2, mi2);
                    if (lane == il) {
                        macc[b] = ma;
                        minn[b] = mi;
                    }
                    if (lane == il2) {
                        macc[b] = ma2;
                        minn[b] = mi2;
                    }
                }
            }
        }
    };
    int mybase = 0;   // where this lane's candidates start in se
    int myself = -1;  // this lane's own candidate index, -1 if absent
    // phase 2: this lane's accepted candidates, in order; the masks are cleared
    auto phase2 = [&]() {
        int nall = 0, ninn = 0;
#pragma unroll
        for (int b = 0; b < MB; ++b) {
            const unsigned own = (myself >> 5) == b ? 1u << (myself & 31) : 0u;
            macc[b] &= ~own;
            minn[b] &= ~own;
            nall += __popc(macc[b]);
            ninn += __popc(minn[b]);
        }
        qtot += nall;
        if (!__any_sync(0xffffffffu, qin + qout + nall > cap)) {
            uint32_t *up = col + 32 * qin;
            uint32_t *down = col + 32 * (cap - 1 - qout);
            qin += ninn;
            qout += nall - ninn;
#pragma unroll
            for (int b = 0; b < MB; ++b) {
                for (unsigned m = minn[b]; m; m &= m - 1u) {
                    *up = se[mybase + b * 32 + __ffs(int(m)) - 1];
                    up += 32;
                }
            }
#pragma unroll
            for (int b = 0; b < MB; ++b) {
                for (unsigned m = macc[b] & ~minn[b]; m; m &= m - 1u) {
                    *down = se[mybase + b * 32 + __ffs(int(m)) - 1];
                    down -= 32;
                }
            }
        } else {  // entries past the capacity are counted, not written
#pragma unroll
            for (int b = 0; b < MB; ++b) {
                for (unsigned m = macc[b]; m; m &= m - 1u) {
                    const int bit = __ffs(int(m)) - 1;
                    const bool in = (minn[b] >> bit) & 1u;
                    if (qin + qout < cap) {
                        col[32 * (in ? qin : cap - 1 - qout)] = se[mybase + b * 32 + bit];
                        qin += in;
                        qout += !in;
                    }
                }
            }
        }
#pragma unroll
        for (int b = 0; b < MB; ++b) macc[b] = minn[b] = 0u;
        myself = -1;
        __syncwarp();  // every lane is done with se before it is restaged
    };
    auto test = [&](unsigned grp, int nch, int ebase, unsigned types) {
        types |= __reduce_or_sync(0xffffffffu, (grp >> lane) & 1u ? unsigned(ty) : 0u);
        if (types < 4u && a.uniform_cut) {
            phase1(grp, nch, ebase, std::true_type());
            if (types) {  // the inner partners of types 0..3 are the lipids
#pragma unroll
                for (int b = 0; b < MB; ++b) {
                    if (b * 32 < nch) {
                        const unsigned m = __ballot_sync(0xffffffffu, w_type(wbits(sp[b * 32 + lane].w)) == 0);
                        if ((grp >> lane) & 1u) minn[b] &= m;
                    }
                }
            }
        } else {
            phase1(grp, nch, ebase, std::false_type());
        }
    };
#pragma unroll
    for (int b = 0; b < MB; ++b) macc[b] = minn[b] = 0u;
    unsigned todo = __ballot_sync(0xffffffffu, real);
    unsigned pend = 0u;  // lanes whose masks refer to se
    int eused = 0;       // entries staged in se
    while (todo) {
        const int kd = __shfl_sync(0xffffffffu, kme, __ffs(int(todo)) - 1);
        const unsigned grp = __ballot_sync(0xffffffffu, real && kme == kd) & todo;
        const int total_c = fetch(kd);
        todo &= ~grp;
        const int ts = own_first + (i - own_slot);
        const bool member = (grp >> lane) & 1u;
        if (total_c > REG) {  // in chunks of REG, each placed at once
            if (pend) phase2();
            pend = 0u;
            eused = 0;
            mybase = 0;
            for (int c0 = 0; c0 < total_c; c0 += REG) {
                const int nch = min(REG, total_c - c0);
                test(grp, nch, 0, stage(c0, nch, 0));
                if (member) myself = (ts >= c0 && ts < c0 + nch) ? ts - c0 : -1;
                phase2();
            }
            continue;
        }
        if (eused + total_c > SE) {  // se is full: place what it holds
            phase2();
            pend = 0u;
            eused = 0;
        }
        test(grp, total_c, eused, stage(0, total_c, eused));
        if (member) {
            mybase = eused;
            myself = ts;
        }
        eused += total_c;
        pend |= grp;
    }
    if (pend) phase2();
    if (mine) a.nnb[i] = real ? (qin | (qout << 16)) : 0;
    nlist_finalise(a, real ? qtot : 0, cur, lp);
}

/* As many warps per 32 slots (4, 2 or 1) as are all resident at once: there the
 * chain of one warp sets the time.  Four / two / one warps, FP32 (4,256 resident):
 * 2,048 particles 16 / 17 / 22 us, 34,000 (four fit) 22 / 22 / 25, 40,000 33 / 22 / 25, 67,000
 * (two fit) 42 / 27 / 28, 75,000 47 / 38 / 29, 200,000 115 / 75 / 59; FP64 (3,648): 2,048 21 / 29 /
 * 43 us, 26,000 (four fit) 33 / 33 / 45, 32,768 47 / 36 / 45, 58,000 (two fit) 65 / 52 / 52, 62,000 73 /
 * 69 / 55. */
template<class R> void launch_nlist(const KArgs<R> &a, cudaStream_t st, int gated) {
    const int nw = a.npad / 32, room = NUM_SM * nlist_warps<R>;  // nw is a multiple of 8
    if (nw * 4 <= room)
        k_nlist<R, 4><<<nw * 4 / NLW, 32 * NLW, 0, st>>>(a, gated);
    else if (nw * 2 <= room)
        k_nlist<R, 2><<<nw * 2 / NLW, 32 * NLW, 0, st>>>(a, gated);
    else
        k_nlist<R, 1><<<nw / NLW, 32 * NLW, 0, st>>>(a, gated);
}

static int grid_for(int64_t n, int per_block = 256) {
    int64_t g = (n + per_block - 1) / per_block;
    const int64_t cap = NUM_SM * 8;
    return int(g < 1 ? 1 : (g > cap ? cap : g));
}

template<class R> void launch_rebuild_stage(const KArgs<R> &a, cudaStream_t st, bool gated, int stage) {
    const int g = grid_for(a.npad);
    switch (stage) {
        case 0:
            k_rebin<R><<<a.npad / 256, 256, 0, st>>>(a, gated ? 1 : 0);
            break;
        case 1:
            k_tile_scan<<<std::min(a.nscan, SCAN_GRID), 1024, 0, st>>>(a.tcnt, a.tstart, a.bsum, a.nscan,
                                                                       &a.S->scan_counter,
                                                                       gated ? &a.S->rebuild : nullptr);
            k_tile_cells<R><<<std::min(a.nctile / 256, 16 * SCAN_GRID), 256, 0, st>>>(a, gated ? 1 : 0);
            k_place<R><<<a.npad / 256, 256, 0, st>>>(a, gated ? 1 : 0);
            k_rank<R><<<a.npad / 256, 256, 0, st>>>(a, gated ? 1 : 0);
            break;
        case 2:
            k_gather<R><<<g, 256, 0, st>>>(a, gated ? 1 : 0);
            break;
        default:
            launch_nlist<R>(a, st, gated ? 1 : 0);
            break;
    }
}

template<class R> void launch_rebuild(const KArgs<R> &a, cudaStream_t st, bool gated) {
    for (int k = 0; k < 4; ++k) launch_rebuild_stage<R>(a, st, gated, k);
}

/* ------------------------------------------------------------------------- */
/* State conversion                                                          */
/* ------------------------------------------------------------------------- */
/* Host state -> device slots for upload indices [k0, k1).  The staged host
 * arrays hold the particles from upload index `first` on, `stride` values of
 * type TH per particle (AoS; FP64 vectors of 3, or the reference's own `real`
 * = float vectors of 3, or of 4 under its _VEC4 layout). */
template<class R, class TH>
__device__ __forceinline__ void set_one(const KArgs<R> &a, int cur, int lp, int64_t k, const TH *x, const TH *nv,
                                        const TH *v, const TH *o, int &out, int &moved) {
    using T4 = typename Vec<R>::T4;
    {
        const int p = a.slot_of_home[k];
        const int hk = 0;
        const SysDev &sd = a.sys[a.blk_sys[p / SYS_PAD]];
        T4 q = a.pos[cur][p];
        // A particle still within skin/2 of where the list was built keeps its
        // cell (the list's shift codes stay valid) and no rebuild is needed:
        // the offset is taken from that cell's centre (minimum image on
        // periodic axes).  Otherwise it is binned afresh and the list rebuilt.
        const int c0 = a.cell[lp][p];
        const int cc0[3] = {cx_of(c0), cy_of(c0), cz_of(c0)};
        const T4 xr = a.xref[lp][p];
        const R xrv[3] = {xr.x, xr.y, xr.z};
        R keep[3];
        R md2 = 0;
        for (int d = 0; d < 3; ++d) {
            const double center = __dadd_rn(sd.lo[d], __dmul_rn(double(cc0[d]) + 0.5, sd.Lc[d]));
            double u = __dsub_rn(double(x[hk + d]), center);
            if (sd.per[d]) {
                const double L = double(sd.nc[d]) * sd.Lc[d];
                u -= L * rint(u / L);
            }
            keep[d] = R(u);
            md2 += (keep[d] - xrv[d]) * (keep[d] - xrv[d]);
        }
        if (md2 <= a.skin_half2) {
            q.x = keep[0];
            q.y = keep[1];
            q.z = keep[2];
            a.pos[cur][p] = q;
        } else {
            moved = 1;
            a.ranges[sd.cell_base + cell_code(sd, cc0[0], cc0[1], cc0[2])] = make_int2(0, 0);
            int cc[3];
            R off[3];
            for (int d = 0; d < 3; ++d) {
                const double xd = double(x[hk + d]);
                const int cu = int(floor(__ddiv_rn(__dsub_rn(xd, sd.lo[d]), sd.Lc[d])));
                int c = cu;
                if (sd.per[d]) {
                    c %= sd.nc[d];
                    if (c < 0) c += sd.nc[d];
                } else {
                    c = min(max(cu, 0), sd.nc[d] - 1);
                    if (c != cu) out = 1;
                }
                const int cref = sd.per[d] ? cu : c;
                const double center = __dadd_rn(sd.lo[d], __dmul_rn(double(cref) + 0.5, sd.Lc[d]));
                off[d] = R(__dsub_rn(xd, center));
                cc[d] = c;
            }
            q.x = off[0];
            q.y = off[1];
            q.z = off[2];
            a.pos[cur][p] = q;
            a.xref[lp][p] = q;
            a.cell[lp][p] = cpack(cc[0], cc[1], cc[2]);
        }
        T4 t = a.nrm[cur][p];
        t.x = R(nv[hk]);
        t.y = R(nv[hk + 1]);
        t.z = R(nv[hk + 2]);
        a.nrm[cur][p] = t;
        t = a.vel[lp][p];
        t.x = R(v[hk]);
        t.y = R(v[hk + 1]);
        t.z = R(v[hk + 2]);
        a.vel[lp][p] = t;
        t = a.omg[lp][p];
        t.x = R(o[hk]);
        t.y = R(o[hk + 1]);
        t.z = R(o[hk + 2]);
        a.omg[lp][p] = t;
    }
}

template<class R, class TH>
__global__ void k_set_state(KArgs<R> a, const TH *x, const TH *nv, const TH *v, const TH *o, int64_t k0, int64_t k1,
                            int64_t first, int stride) {
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    int out = 0, moved = 0;
    for (int64_t k = k0 + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < k1; k += int64_t(gridDim.x) * blockDim.x) {
        const int64_t hk = (k - first) * stride;
        set_one<R, TH>(a, cur, lp, k, x + hk, nv + hk, v + hk, o + hk, out, moved);
    }
    if (out) atomicOr(&a.S->error, ERRB_GRID);
    if (__syncthreads_or(moved) && threadIdx.x == 0) a.S->rebuild = 1;
}

/* In-place transfers over the host link (the caller's arrays are reachable
 * from the GPU).  Host memory gives full link bandwidth only to wide, fully
 * coalesced accesses, so each block moves a tile of HOST_TILE particles of
 * each array through shared memory with 16-byte loads or stores (a base that
 * is not 16-byte aligned falls back to contiguous scalar accesses), and the
 * per-particle conversion works on the staged tile. */
constexpr int HOST_TILE = 256;
template<class TH> __device__ __forceinline__ void tile_in(TH *dst, const TH *src, int nvals) {
    const uintptr_t addr = reinterpret_cast<uintptr_t>(src);
    if ((addr & 15u) == 0) {
        const int nv4 = int(nvals * sizeof(TH) / 16);
        const int4 *s4 = reinterpret_cast<const int4 *>(src);
        int4 *d4 = reinterpret_cast<int4 *>(dst);
        for (int t = threadIdx.x; t < nv4; t += blockDim.x) d4[t] = s4[t];
        for (int t = nv4 * int(16 / sizeof(TH)) + threadIdx.x; t < nvals; t += blockDim.x) dst[t] = src[t];
    } else {
        for (int t = threadIdx.x; t < nvals; t += blockDim.x) dst[t] = src[t];
    }
}
template<class TH> __device__ __forceinline__ void tile_out(TH *dst, const TH *src, int nvals) {
    const uintptr_t addr = reinterpret_cast<uintptr_t>(dst);
    if ((addr & 15u) == 0) {
        const int nv4 = int(nvals * sizeof(TH) / 16);
        const int4 *s4 = reinterpret_cast<const int4 *>(src);
        int4 *d4 = reinterpret_cast<int4 *>(dst);
        for (int t = threadIdx.x; t < nv4; t += blockDim.x) d4[t] = s4[t];
        for (int t = nv4 * int(16 / sizeof(TH)) + threadIdx.x; t < nvals; t += blockDim.x) dst[t] = src[t];
    } else {
        for (int t = threadIdx.x; t < nvals; t += blockDim.x) dst[t] = src[t];
    }
}

template<class R, class TH>
__global__ void __launch_bounds__(HOST_TILE) k_set_state_host(KArgs<R> a, const TH *x, const TH *nv, const TH *v,
                                                              const TH *o, int64_t k0, int64_t k1, int64_t first,
                                                              int stride) {
    __shared__ __align__(16) TH buf[4][HOST_TILE * 4];
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    const int64_t kb = k0 + int64_t(blockIdx.x) * HOST_TILE;
    const int m = int(k1 - kb < HOST_TILE ? k1 - kb : HOST_TILE);
    const TH *src[4] = {x, nv, v, o};
    for (int q = 0; q < 4; ++q) tile_in<TH>(buf[q], src[q] + (kb - first) * stride, m * stride);
    __syncthreads();
    int out = 0, moved = 0;
    const int t = threadIdx.x;
    if (t < m) {
        const int hk = t * stride;
        set_one<R, TH>(a, cur, lp, kb + t, buf[0] + hk, buf[1] + hk, buf[2] + hk, buf[3] + hk, out, moved);
    }
    if (out) atomicOr(&a.S->error, ERRB_GRID);
    if (__syncthreads_or(moved) && threadIdx.x == 0) a.S->rebuild = 1;
}

template<class R, class TH>
void launch_set_state(const KArgs<R> &a, const TH *x, const TH *n, const TH *v, const TH *o, int64_t k0, int64_t k1,
                      int64_t first, int stride, cudaStream_t st) {
    k_set_state<R, TH><<<grid_for(k1 - k0), 256, 0, st>>>(a, x, n, v, o, k0, k1, first, stride);
}
template<class R, class TH>
void launch_set_state_host(const KArgs<R> &a, const TH *x, const TH *n, const TH *v, const TH *o, int64_t k0,
                           int64_t k1, int64_t first, int stride, cudaStream_t st) {
    const int64_t nb = (k1 - k0 + HOST_TILE - 1) / HOST_TILE;
    if (nb > 0) k_set_state_host<R, TH><<<int(nb), HOST_TILE, 0, st>>>(a, x, n, v, o, k0, k1, first, stride);
}

/* Device state -> caller-order AoS vectors of TH for upload indices [h0, h1),
 * written from upload index `first` on with `stride` values per particle (a
 * fourth value, when stride is 4, is written as 0).  One thread per upload
 * index (the slot comes from slot_of_home), so the writes -- the side that
 * streams to the host -- are coalesced; the slot-side reads are gathers. */
template<class R, class TH>
__device__ __forceinline__ void get_one(const KArgs<R> &a, int cur, int lp, int64_t h, int64_t hk, int stride, TH *x,
                                        TH *nv, TH *v, TH *o, TH *f, TH *t, double *e) {
    using T4 = typename Vec<R>::T4;
    {
        const int p = a.slot_of_home[h];
        const SysDev &sd = a.sys[a.blk_sys[p / SYS_PAD]];
        if (x) {
            const T4 q = a.pos[cur][p];
            const int c = a.cell[lp][p];
            const int cc[3] = {cx_of(c), cy_of(c), cz_of(c)};
            const double off[3] = {double(q.x), double(q.y), double(q.z)};
            for (int d = 0; d < 3; ++d)
                x[hk + d] = TH(__dadd_rn(__dadd_rn(sd.lo[d], __dmul_rn(double(cc[d]) + 0.5, sd.Lc[d])), off[d]));
            if (stride == 4) x[hk + 3] = TH(0);
        }
        auto put = [&](TH *dst, const T4 &q) {
            if (!dst) return;
            dst[hk] = TH(q.x);
            dst[hk + 1] = TH(q.y);
            dst[hk + 2] = TH(q.z);
            if (stride == 4) dst[hk + 3] = TH(0);
        };
        if (nv) put(nv, a.nrm[cur][p]);
        if (v) put(v, a.vel[lp][p]);
        if (o) put(o, a.omg[lp][p]);
        if (f) put(f, a.frc[lp][p]);
        if (t) put(t, a.trq[lp][p]);
        if (e) e[h] = a.epart[p];
    }
}

template<class R, class TH>
__global__ void k_download(KArgs<R> a, int64_t h0, int64_t h1, int64_t first, int stride, TH *x, TH *nv, TH *v,
                           TH *o, TH *f, TH *t, double *e) {
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    for (int64_t h = h0 + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; h < h1; h += int64_t(gridDim.x) * blockDim.x)
        get_one<R, TH>(a, cur, lp, h, (h - first) * stride, stride, x, nv, v, o, f, t, e);
}

/* In-place download: the tile's values are formed in shared memory, then
 * each array's tile is written to the host with 16-byte stores. */
template<class R, class TH>
__global__ void __launch_bounds__(HOST_TILE) k_download_host(KArgs<R> a, int64_t h0, int64_t h1, int64_t first,
                                                             int stride, TH *x, TH *nv, TH *v, TH *o) {
    __shared__ __align__(16) TH buf[4][HOST_TILE * 4];
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    const int64_t hb = h0 + int64_t(blockIdx.x) * HOST_TILE;
    const int m = int(h1 - hb < HOST_TILE ? h1 - hb : HOST_TILE);
    TH *dst[4] = {x, nv, v, o};
    const int t = threadIdx.x;
    if (t < m)
        get_one<R, TH>(a, cur, lp, hb + t, int64_t(t) * stride, stride, x ? buf[0] : nullptr, nv ? buf[1] : nullptr,
                       v ? buf[2] : nullptr, o ? buf[3] : nullptr, nullptr, nullptr, nullptr);
    __syncthreads();
    for (int q = 0; q < 4; ++q)
        if (dst[q]) tile_out<TH>(dst[q] + (hb - first) * stride, buf[q], m * stride);
}

template<class R, class TH>
void launch_download(const KArgs<R> &a, int64_t h0, int64_t h1, int64_t first, int stride, TH *x, TH *n, TH *v, TH *o,
                     TH *f, TH *t, double *e, cudaStream_t st) {
    k_download<R, TH><<<grid_for(h1 - h0), 256, 0, st>>>(a, h0, h1, first, stride, x, n, v, o, f, t, e);
}
template<class R, class TH>
void launch_download_host(const KArgs<R> &a, int64_t h0, int64_t h1, int64_t first, int stride, TH *x, TH *n, TH *v,
                          TH *o, cudaStream_t st) {
    const int64_t nb = (h1 - h0 + HOST_TILE - 1) / HOST_TILE;
    if (nb > 0) k_download_host<R, TH><<<int(nb), HOST_TILE, 0, st>>>(a, h0, h1, first, stride, x, n, v, o);
}
template<class R> void launch_download(const KArgs<R> &a, int64_t h0, int64_t h1, double *x, double *n, double *v,
                                       double *o, double *f, double *t, double *e, cudaStream_t st) {
    launch_download<R, double>(a, h0, h1, 0, 3, x, n, v, o, f, t, e, st);
}

__global__ void k_set_cond(cudaGraphConditionalHandle h, const Scalars *S) {
    cudaGraphSetConditional(h, __ldcg(&S->rebuild) ? 1u : 0u);
}
void launch_set_cond(cudaGraphConditionalHandle h, Scalars *S, cudaStream_t st) {
    k_set_cond<<<1, 1, 0, st>>>(h, S);
}

/* ------------------------------------------------------------------------- */
/* Reference Morton key (src/reorder_morton.h:25-42).                        */
/* ------------------------------------------------------------------------- */
__device__ __forceinline__ uint32_t bit_space3(uint32_t x) {
    x = (x | (x << 12)) & 0x00FC003Fu;
    x = (x | (x << 6)) & 0x381C0E07u;
    x = (x | (x << 4)) & 0x190C8643u;
    x = (x | (x << 2)) & 0x49249249u;
    return x;
}
__global__ void k_morton(const double *p3, int64_t n, double b0, double b1, double b2, uint32_t *keys) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const uint32_t cx = __double2uint_rz(__dadd_rn(2.0 * p3[3 * i], b0));
        const uint32_t cy = __double2uint_rz(__dadd_rn(2.0 * p3[3 * i + 1], b1));
        const uint32_t cz = __double2uint_rz(__dadd_rn(2.0 * p3[3 * i + 2], b2));
        keys[i] = bit_space3(cx) | (bit_space3(cy) << 1) | (bit_space3(cz) << 2);
    }
}
void launch_morton(const double *p3, int64_t n, const double *b, uint32_t *keys, cudaStream_t st) {
    k_morton<<<grid_for(n), 256, 0, st>>>(p3, n, b[0], b[1], b[2], keys);
}

template void launch_rebuild<float>(const KArgs<float> &, cudaStream_t, bool);
template void launch_rebuild_stage<float>(const KArgs<float> &, cudaStream_t, bool, int);
template void launch_rebuild_stage<double>(const KArgs<double> &, cudaStream_t, bool, int);
template void launch_rebuild<double>(const KArgs<double> &, cudaStream_t, bool);
#define ORBC_IO_INST(R, TH)                                                                                    \
    template void launch_set_state<R, TH>(const KArgs<R> &, const TH *, const TH *, const TH *, const TH *, int64_t, \
                                          int64_t, int64_t, int, cudaStream_t);                                      \
    template void launch_download<R, TH>(const KArgs<R> &, int64_t, int64_t, int64_t, int, TH *, TH *, TH *, TH *,    \
                                         TH *, TH *, double *, cudaStream_t);                                          \
    template void launch_set_state_host<R, TH>(const KArgs<R> &, const TH *, const TH *, const TH *, const TH *,     \
                                               int64_t, int64_t, int64_t, int, cudaStream_t);                           \
    template void launch_download_host<R, TH>(const KArgs<R> &, int64_t, int64_t, int64_t, int, TH *, TH *, TH *,    \
                                              TH *, cudaStream_t);
ORBC_IO_INST(float, float)
ORBC_IO_INST(float, double)
ORBC_IO_INST(double, float)
ORBC_IO_INST(double, double)
#undef ORBC_IO_INST
template void launch_download<float>(const KArgs<float> &, int64_t, int64_t, double *, double *, double *, double *,
                                     double *, double *, double *, cudaStream_t);
template void launch_download<double>(const KArgs<double> &, int64_t, int64_t, double *, double *, double *,
                                      double *, double *, double *, double *, cudaStream_t);

}  // namespace orbc
