// Pair kernel, histogram form over frame lists sorted by the row DOF's bin.
//
// Same work as the other histogram kernels (the 2D fill + epilogue loops of
// PARENT.cpp :786-1479). Once a row DOF's frames are listed bin by bin, the
// part of a pair's 2D histogram that belongs to row bin a is the plain 1D
// histogram of the column DOF's bins over the frames of that list segment.
// A CTA then needs B counters per column at a time instead of B x B, so
//   - a warp counts 128 columns at once (the tiles of the other kernels hold
//     32 pairs at 50 bins, 4 at 51-100, 1 above),
//   - a counter's address is one multiply-add of the column's bin byte: no
//     row bin, no index arithmetic, and
//   - counters are private to a team of a few warps, so nothing waits on the
//     whole CTA.
//
// Data. The column bins are transposed to frame-major rows of 128 bytes
// (128 columns, one block; row F holds the dummy bin). A list segment holds
// the frame numbers of one row bin, padded with F to a multiple of 4. A warp
// reads 4 rows per load (8 lanes x 16 bytes each): lane (fr, sub) holds
// columns 16 sub .. 16 sub + 15 of frame fr.
//
// Counters. 16-bit halves: columns 2h and 2h + 1 of a 16-column group share a
// word. A team's table has two planes (h >> 2) of one 32-word row per bin, and
// the word of (sub, h) is sub * 4 + (h & 3): at every step the four frames of
// a load take four different h of one plane (their order rotated by fr), so
// the 32 lanes of a reduction lie in 32 banks. A half cannot pass the frames counted since
// the last read-out, so pieces of at most kPiece frames never overflow;
// longer segments move their counts to 32-bit sums between pieces.
//
// Read-out: per row bin, every count's n ln n (fixed point, exact integer
// sums: the result does not depend on the order, and equals the other
// kernels' bit for bit) and the occupied bins, kept in registers over the
// segments of an item and added to the MI matrix's storage, which the
// finishing kernel turns into S2D and MI.
//
// What bounds it: the shared-memory / L1 data pipe, 91 % busy (894 DOFs x 100k
// frames, 50 bins), two thirds of it the reductions: one cycle per 32 updates,
// a quarter of one for the row bytes, a tenth for the frame numbers' shuffles.
// 2,994 DOFs x 100k frames at 50 bins: pair phase 90.5 ms with the streamed
// tiles (83 % busy at one and a half cycles and 6.7 instructions per 32
// updates), 72.8 ms here, 0.6 ms of it the lists, 0.2 the transposition, 0.3
// the finish.
//
// The counters stay below 128 KB: beyond that the lines that the loads bring
// into L1 share the arrays with the counters and every line costs the
// reductions one more cycle (160 KB of counters: 8.3e12 reductions of this
// loop per second against 10.4e12 below 128 KB).
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "pg_internal.h"
#include "pg_sync.cuh"

namespace pg {

namespace {

using namespace dev;

// 16 warps with 8 row loads in flight each (2,994 DOFs x 100k frames at 50
// bins: 76.9 ms; 24 warps with 4 or 8 loads 79.7 and 84.1, 32 with 4 85.4, 16
// with 4 111.5)
constexpr int kWarps = 16, kThreads = kWarps * 32;
constexpr int kLoads = 8, kBatch = 4 * kLoads;  // row loads in flight per warp, and their frames
constexpr int kBlk = 128;                 // columns of a block: bytes of a row
constexpr int kRowBytes = 256;            // a team's counters of one bin
constexpr int kTableMax = 120 * 1024;     // counter bytes of a CTA
constexpr int kPiece = 64512;             // frames between read-outs: a half holds 65,535
constexpr int kMaxTeams = 8;

// ------------------------------------------------------------ preparation

// Frame lists of one row DOF per CTA. The segments' places come from the
// marginal counts of the preprocessing. A chunk of 8,192 frames is sorted in
// shared memory (a returning atomic per frame gives its place among the
// chunk's frames of its bin), then written run by run: consecutive threads
// write consecutive entries. Scattered 4-byte stores straight from the frames,
// one sector each, took 1.66 ms at 2,994 DOFs x 100k frames; this takes
// 0.62 (894 DOFs x 1M frames 5.1 -> 1.8).
constexpr int kSortThreads = 512, kChunk = kSortThreads * 16;

__device__ __forceinline__ const SortedSys &sorted_sys(const SortedArgs &a, int s) { return a.many ? a.many[s] : a.one; }

__global__ void __launch_bounds__(kSortThreads) sort_frames_kernel(const __grid_constant__ SortedArgs a, const int2 *map,
                                                                   int row0) {
    __shared__ uint32_t stage[kChunk];           // frame of the chunk | bin << 16
    __shared__ int s_next[256];                  // next free entry of every segment
    __shared__ int s_cnt[256], s_loc[256];       // the chunk's counts and their starts
    __shared__ int s_warp[8];
    const int2 m = map ? map[blockIdx.x] : make_int2(0, row0 + (int)blockIdx.x);
    const SortedSys &d = sorted_sys(a, m.x);
    const int row = m.y, F = d.geo.F;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int B = d.geo.bins[3 + dof_type(row, d.geo.nb, d.geo.na)];
    const uint8_t *src = d.bins + (int64_t)row * d.geo.ldb;
    uint32_t *list = d.list + (int64_t)(row - d.row_first) * d.list_ld;
    int *seg = d.seg + (int64_t)(row - d.row_first) * kSegLd;
    // exclusive scan of 256 counts by the first 8 warps
    auto scan256 = [&](int n) -> int {
        int x = n;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (warp < 8 && lane == 31) s_warp[warp] = x;
        __syncthreads();
        for (int w = 0; w < min(warp, 8); w++) x += s_warp[w];
        return x - n;
    };
    {  // segments start on multiples of 4, padded with frame F
        const int n = tid < B ? d.dof.h2[(int64_t)row * kSegLd + tid] : 0, np = (n + 3) & ~3;
        const int start = scan256(np);
        if (tid <= B) seg[tid] = start;
        if (tid < 256) {
            s_next[tid] = start;
            s_cnt[tid] = 0;
        }
        for (int k = n; k < np; k++) list[start + k] = (uint32_t)F;
    }
    __syncthreads();
    for (int c0 = 0; c0 < F; c0 += kChunk) {
        const int f0 = tid * 16, n = min(16, F - c0 - f0);  // the row is padded past F
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (n > 0) v = __ldg((const uint4 *)(src + c0 + f0));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        int at[16];
#pragma unroll
        for (int k = 0; k < 16; k++) at[k] = k < n ? atomicAdd(&s_cnt[(w[k >> 2] >> (8 * (k & 3))) & 0xffu], 1) : 0;
        __syncthreads();
        {
            const int x = scan256(tid < 256 ? s_cnt[tid] : 0);
            if (tid < 256) s_loc[tid] = x;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const uint32_t b = (w[k >> 2] >> (8 * (k & 3))) & 0xffu;
            if (k < n) stage[s_loc[b] + at[k]] = (uint32_t)(f0 + k) | b << 16;
        }
        __syncthreads();
        const int total = min(kChunk, F - c0);
        for (int k = tid; k < total; k += kSortThreads) {
            const uint32_t x = stage[k], b = x >> 16;
            list[s_next[b] + k - s_loc[b]] = (uint32_t)c0 + (x & 0xffffu);
        }
        __syncthreads();
        if (tid < 256) {
            s_next[tid] += s_cnt[tid];
            s_cnt[tid] = 0;
        }
        __syncthreads();
    }
}

// DOF-major bins -> blocks of 128 columns, frame-major: 256 frames of one
// block per CTA through shared memory; a thread writes 32 columns (a whole
// sector) of one frame. Columns outside the system and row F get the dummy
// bin a.dummy.
constexpr int kTrFrames = 256, kTrPitch = kTrFrames + 4;

__global__ void __launch_bounds__(256) transpose_bins_kernel(const __grid_constant__ SortedArgs a, const int2 *map) {
    __shared__ uint8_t tile[kBlk * kTrPitch];
    const int2 m = map ? map[blockIdx.y] : make_int2(0, (int)blockIdx.y);
    const SortedSys &d = sorted_sys(a, m.x);
    const int F = d.geo.F, f0 = blockIdx.x * kTrFrames;
    if (f0 > F) return;
    const int c0 = m.y * kBlk - d.pad;
    const uint32_t dummy4 = 0x01010101u * (uint32_t)a.dummy;
    for (int k = threadIdx.x; k < kBlk * (kTrFrames / 16); k += 256) {
        const int r = k / (kTrFrames / 16), q = (k % (kTrFrames / 16)) * 16, c = c0 + r;
        uint4 v = make_uint4(dummy4, dummy4, dummy4, dummy4);
        if (c >= 0 && f0 + q < F) v = __ldg((const uint4 *)(d.bins + (int64_t)c * d.geo.ldb + f0 + q));
        uint32_t *t = (uint32_t *)(tile + r * kTrPitch + q);
        t[0] = v.x;
        t[1] = v.y;
        t[2] = v.z;
        t[3] = v.w;
    }
    __syncthreads();
    uint8_t *out = d.mat + ((int64_t)m.y * (F + 1) + f0) * kBlk;
    for (int k = threadIdx.x; k < kTrFrames * 4; k += 256) {
        const int f = k % kTrFrames, q = (k / kTrFrames) * 32;
        if (f0 + f > F) continue;
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (f0 + f == F) {
                w[j] = dummy4;
            } else {
                const uint8_t *t = tile + (q + 4 * j) * kTrPitch + f;
                w[j] = t[0] | (uint32_t)t[kTrPitch] << 8 | (uint32_t)t[2 * kTrPitch] << 16 | (uint32_t)t[3 * kTrPitch] << 24;
            }
        }
        uint4 *o = (uint4 *)(out + (int64_t)f * kBlk + q);
        o[0] = make_uint4(w[0], w[1], w[2], w[3]);
        o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// ------------------------------------------------------------ pair kernel

// 16 bytes of a row, not kept in L1 (a CTA reads a row once) but kept in L2
// like any other line: a load that only says no_allocate is the first to be
// evicted there, and the other rows' CTAs then re-read the block from DRAM
// (2.1 TB/s of it; 894 DOFs x 1M frames 77.9 -> 73.4 ms with the policy).
__device__ __forceinline__ uint4 ldg_row(const void *p, uint64_t policy) {
    uint4 r;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(p), "l"(policy));
    return r;
}
__device__ __forceinline__ uint64_t row_policy() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void team_barrier(int team, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(threads) : "memory");
}

// Counts the 16 columns that a lane holds of its frame.
__device__ __forceinline__ void count_rows(const uint4 &x, bool swap, const uint32_t (&wgt)[2][2],
                                           const uint32_t (&base)[4][2]) {
    const uint32_t c[4] = {swap ? x.y : x.x, swap ? x.x : x.y, swap ? x.w : x.z, swap ? x.z : x.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            red_add_nc(__dp4a(c[k], wgt[e][0], base[k][e]), 1u);
            red_add_nc(__dp4a(c[k], wgt[e][1], base[k][e]), 65536u);
        }
    }
}

// One warp's place in the lists: 32 entries from `base` of segment a (n of
// them valid, a multiple of 4; n == 0: past the item's end).
struct Place {
    int a, base, n;
};

template <bool BIG>
__global__ void __launch_bounds__(kThreads, 1) pairs_sorted_kernel(const __grid_constant__ SortedArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_item[kMaxTeams];
    __shared__ int s_seg[kMaxTeams][kSegLd];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wpt = kWarps / a.teams, team = warp / wpt, tw = warp % wpt, tthreads = wpt * 32;
    const int ttid = tw * 32 + lane;
    uint32_t *table = (uint32_t *)(smem + (size_t)team * a.rows * kRowBytes);
    for (int k = ttid * 4; k < a.rows * 64; k += tthreads * 4) *(uint4 *)(table + k) = make_uint4(0u, 0u, 0u, 0u);
    team_barrier(team, tthreads);

    const int fr = lane >> 3, sub = lane & 7;
    const bool swap = (fr & 2) != 0, odd = (fr & 1) != 0;
    // half-word pair e of register k after the swap: its word in bin 0, and the
    // byte weights that add 128 (a row) times its low / high bin byte
    uint32_t base[4][2], wgt[2][2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int h = e ^ (int)odd;
#pragma unroll
        for (int k = 0; k < 4; k++)
            base[k][e] = smem_u32(table) + (uint32_t)(((k >> 1) * a.rows) * 32 + sub * 4 + ((k & 1) ^ (int)swap) * 2 + h) * 4;
        wgt[e][0] = 128u << (16 * h);
        wgt[e][1] = wgt[e][0] << 8;
    }
    const uint64_t pol = row_policy();
    uint32_t *ovf = BIG ? a.ovf + ((size_t)blockIdx.x * a.teams + team) * (size_t)a.rows * 128 : nullptr;

    for (;;) {
        if (ttid == 0) s_item[team] = atomicAdd(a.counter, 1);
        team_barrier(team, tthreads);
        const int it = s_item[team];
        if (it >= a.n_items) break;
        const SortedItem item = a.items[it];
        const SortedSys &d = sorted_sys(a, item.sys);
        const int F = d.geo.F, D = d.geo.D, row = item.row;
        const int B = d.geo.bins[3 + dof_type(row, d.geo.nb, d.geo.na)];
        const int c0 = item.blk * kBlk - d.pad;
        const uint32_t *list = d.list + (int64_t)(row - d.row_first) * d.list_ld;
        {
            const int *seg = d.seg + (int64_t)(row - d.row_first) * kSegLd;
            for (int k = ttid; k <= B; k += tthreads) s_seg[team][k] = __ldg(seg + k);
        }
        // largest bin count of the block's columns
        const int clast = min(D, c0 + kBlk) - 1;
        int bblk = 1;
        if (c0 < d.geo.nb) bblk = max(bblk, d.geo.bins[3]);
        if (c0 < d.geo.nb + d.geo.na && clast >= d.geo.nb) bblk = max(bblk, d.geo.bins[4]);
        if (clast >= d.geo.nb + d.geo.na) bblk = max(bblk, d.geo.bins[5]);
        team_barrier(team, tthreads);
        const int *seg = s_seg[team];
        // the item's segments [a0, a1): those that start in its share of the list
        int a0 = 0, a1 = B;
        if (d.parts > 1) {
            const int64_t total = seg[B];
            const int lo = (int)(total * item.part / d.parts), hi = (int)(total * (item.part + 1) / d.parts);
            while (a0 < B && seg[a0] < lo) a0++;
            a1 = a0;
            while (a1 < B && (seg[a1] < hi || item.part == d.parts - 1)) a1++;
        }
        const unsigned char *mat = d.mat + (int64_t)item.blk * (F + 1) * kBlk + sub * 16;

        auto settle = [&](Place p) -> Place {  // moves p to the first segment that has entries for this warp
            while (p.a < a1 && p.base >= seg[p.a + 1]) {
                p.a++;
                if (p.a < a1) p.base = seg[p.a] + kBatch * tw;
            }
            p.n = p.a < a1 ? min(kBatch, seg[p.a + 1] - p.base) : 0;
            return p;
        };
        auto entries = [&](const Place &p) -> uint32_t {
            return lane < p.n ? __ldg(list + p.base + lane) : (uint32_t)F;
        };
        Place p0{a0, a0 < a1 ? seg[a0] + kBatch * tw : 0, 0};
        p0 = settle(p0);
        Place p1 = settle(Place{p0.a, p0.base + kBatch * wpt, 0});
        uint4 v[kLoads];
        {
            const uint32_t f = entries(p0);
#pragma unroll
            for (int g = 0; g < kLoads; g++)
                if (4 * g < p0.n) v[g] = ldg_row(mat + (int64_t)__shfl_sync(0xffffffffu, f, 4 * g + fr) * kBlk, pol);
        }
        uint32_t f1 = entries(p1);

        unsigned long long snl[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
        uint32_t occ[2] = {0u, 0u};
        for (int s = a0; s < a1; s++) {
            const int s_end = seg[s + 1];
            int p_end = BIG ? min(s_end, seg[s] + kPiece) : s_end;
            bool spilled = false;
            for (;;) {
                while (p0.a == s && (!BIG || p0.base < p_end) && p0.n > 0) {
                    const Place p2 = settle(Place{p1.a, p1.base + kBatch * wpt, 0});
                    const uint32_t f2 = entries(p2);
                    if (p0.n == kBatch && p1.n == kBatch) {  // whole batches, without a test per load
#pragma unroll
                        for (int g = 0; g < kLoads; g++) {
                            count_rows(v[g], swap, wgt, base);
                            v[g] = ldg_row(mat + (int64_t)__shfl_sync(0xffffffffu, f1, 4 * g + fr) * kBlk, pol);
                        }
                    } else {
#pragma unroll
                        for (int g = 0; g < kLoads; g++) {
                            if (4 * g < p0.n) count_rows(v[g], swap, wgt, base);
                            if (4 * g < p1.n) v[g] = ldg_row(mat + (int64_t)__shfl_sync(0xffffffffu, f1, 4 * g + fr) * kBlk, pol);
                        }
                    }
                    p0 = p1;
                    p1 = p2;
                    f1 = f2;
                }
                team_barrier(team, tthreads);
                if (!BIG || p_end >= s_end) break;
                // the piece's counts to the team's 32-bit sums
                for (int b = tw; b < bblk; b += wpt) {
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const int w = (q * a.rows + b) * 32 + lane;
                        const uint32_t x = table[w];
                        if (x) {
                            table[w] = 0u;
                            ovf[2 * w] += x & 0xffffu;
                            ovf[2 * w + 1] += x >> 16;
                        }
                    }
                }
                spilled = true;
                p_end = min(s_end, p_end + kPiece);
                team_barrier(team, tthreads);
            }
            // read-out of row bin s, zeroing the counters: a word that no column
            // of the warp counted in costs one load and a vote
            for (int b = tw; b < bblk; b += 2 * wpt) {
                uint32_t x[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int r = b + (j >> 1) * wpt;
                    x[j] = r < bblk ? table[((j & 1) * a.rows + r) * 32 + lane] : 0u;
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int q = j & 1, w = (q * a.rows + b + (j >> 1) * wpt) * 32 + lane;
                    uint32_t n0 = x[j] & 0xffffu, n1 = x[j] >> 16;
                    if (BIG && spilled && b + (j >> 1) * wpt < bblk) {
                        n0 += ovf[2 * w];
                        n1 += ovf[2 * w + 1];
                        ovf[2 * w] = 0u;
                        ovf[2 * w + 1] = 0u;
                    }
                    if (__any_sync(0xffffffffu, n0 | n1)) {
                        table[w] = 0u;
                        if (n0 > 1u) snl[q][0] += __ldg(a.nfix + n0);  // n ln n is 0 below 2
                        if (n1 > 1u) snl[q][1] += __ldg(a.nfix + n1);
                        occ[q] += (n0 != 0u) + ((n1 != 0u) << 16);  // at most 218 x 218 a half
                    }
                }
            }
            team_barrier(team, tthreads);
        }
        unsigned long long *acc = (unsigned long long *)d.out.mi;
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int c = c0 + (lane >> 2) * 16 + (q * 4 + (lane & 3)) * 2 + h;
                const uint32_t o = h ? occ[q] >> 16 : occ[q] & 0xffffu;
                if (c > row && c < D && o) {
                    atomicAdd(acc + (int64_t)row * D + c, snl[q][h]);
                    atomicAdd(acc + (int64_t)c * D + row, (unsigned long long)o);
                }
            }
        team_barrier(team, tthreads);  // before the next item number replaces this one
    }
}

// The 1D entropies into the body, and the sums -> S2D and MI, in place: the sum of n ln n of pair r < c lies at (r, c)
// of the MI matrix and its occupied bins at (c, r). 32 x 32 tiles, one per
// CTA; a tile reads both of its corners before it writes them.
__global__ void __launch_bounds__(256) sorted_finish_kernel(const __grid_constant__ SortedArgs a) {
    const SortedSys &d = sorted_sys(a, blockIdx.z);
    const int D = d.geo.D, r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    if (c0 < r0 || r0 >= D || c0 >= D) return;
    __shared__ double t[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (r0 == c0 && ty == 0 && r0 + tx < D) d.out.par[d.out.L.s1b + r0 + tx] = d.dof.s1[r0 + tx];  // s1_b | s1_a | s1_d
    double *mi = d.out.mi;
    const unsigned long long *acc = (const unsigned long long *)mi;
    for (int k = ty; k < 32; k += 8) {  // occupied bins: row c0 + k, column r0 + tx
        const int r = r0 + tx, c = c0 + k;
        t[k][tx] = (r < c && c < D) ? (double)acc[(int64_t)c * D + r] : 0.0;
    }
    unsigned long long s[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int r = r0 + ty + 8 * u, c = c0 + tx;
        s[u] = (r < c && c < D) ? acc[(int64_t)r * D + c] : 0ull;
    }
    __syncthreads();
    const double N = (double)d.geo.F;
    double out[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int k = ty + 8 * u, r = r0 + k, c = c0 + tx;
        out[u] = 0.0;
        if (r < c && c < D) {
            const double sn = (double)s[u] / a.fix;
            const double o = t[tx][k];
            const double S2 = d.lnN + d.dof.acon[r] + d.dof.acon[c] - sn / N + (o - 1.0) / (2.0 * N);
            d.out.par[par_pair_index(d.out.L, d.geo.nb, d.geo.na, d.geo.nd, r, c)] = S2;
            out[u] = d.dof.s1[r] + d.dof.s1[c] - S2;
            mi[(int64_t)r * D + c] = out[u];
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; u++) t[tx][ty + 8 * u] = out[u];
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int r = r0 + tx, c = c0 + k;
        if (r < c && c < D) mi[(int64_t)c * D + r] = t[k][tx];
    }
}

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
    }
    return n;
}

int table_rows(int bmax) { return bmax + 1; }
// teams of a CTA: as many tables as fit, a power of two
int team_count(int bmax) {
    int t = kMaxTeams;
    while (t > 1 && t * table_rows(bmax) * kRowBytes > kTableMax) t >>= 1;
    return t;
}

}  // namespace

int64_t sorted_list_ld(const SysGeom &g) { return ((int64_t)g.F + 3 * bmax2d(g) + 31) / 32 * 32; }
int sorted_blocks(int D) { return (D + kBlk - 1) / kBlk; }
size_t sorted_mat_bytes(const SysGeom &g) { return (size_t)sorted_blocks(g.D) * ((size_t)g.F + 1) * kBlk; }
// columns lie at the end of their blocks, so that the one block that is not
// full is the first, which the fewest rows visit
int sorted_pad(int D) { return sorted_blocks(D) * kBlk - D; }
size_t sorted_ovf_bytes(const SysGeom &g) {
    return g.F > kPiece ? (size_t)sm_count() * team_count(bmax2d(g)) * table_rows(bmax2d(g)) * 128 * sizeof(uint32_t) : 0;
}

// Items per (row, block) unit: enough to give every team work, and about 24
// rounds of items where that leaves an item 4,096 frames.
int sorted_parts(const SysGeom &g, int64_t units) {
    const int64_t slots = (int64_t)sm_count() * team_count(bmax2d(g));
    units = std::max<int64_t>(units, 1);
    const int64_t fill = std::min<int64_t>((slots + units - 1) / units, bmax2d(g));
    const int64_t even = std::min<int64_t>((24 * slots + units - 1) / units, g.F / 4096);
    return (int)std::max<int64_t>(1, std::min<int64_t>(std::max(fill, even), bmax2d(g)));
}

int64_t sorted_units(int D) {
    const int pad = sorted_pad(D);
    int64_t n = 0;
    for (int b = 0; b < sorted_blocks(D); b++) n += std::min(D, (b + 1) * kBlk - pad) - 1;
    return n;
}

// Items of rows [row0, row1) of system s: block after block from the last
// (the rows that run together read the same block), all rows with a column to
// their right.
void sorted_items(int s, int D, int row0, int row1, int parts, std::vector<SortedItem> &out) {
    const int pad = sorted_pad(D);
    for (int b = sorted_blocks(D) - 1; b >= 0; b--) {
        const int last = std::min(D, (b + 1) * kBlk - pad) - 1;  // last column of the block
        for (int r = row0; r < std::min(row1, last); r++)
            for (int p = 0; p < parts; p++) out.push_back(SortedItem{s, r, b, p});
    }
}

static SortedArgs complete(const SortedArgs &in, int bmax) {
    SortedArgs a = in;
    a.rows = table_rows(bmax);
    a.teams = team_count(bmax);
    a.dummy = bmax;
    return a;
}

cudaError_t launch_sorted_transpose(const SortedArgs &in, int bmax, int max_F, const int2 *map, int n_blocks,
                                    cudaStream_t st) {
    const SortedArgs a = complete(in, bmax);
    for (int b = 0; b < n_blocks; b += 32768) {  // the grid's y extent is limited to 65,535
        dim3 grid((unsigned)(max_F / kTrFrames + 1), (unsigned)std::min(32768, n_blocks - b));
        transpose_bins_kernel<<<grid, 256, 0, st>>>(a, map ? map + b : nullptr);
    }
    return cudaGetLastError();
}

cudaError_t launch_sorted_lists(const SortedArgs &in, int bmax, const int2 *map, int row0, int n_rows, cudaStream_t st) {
    const SortedArgs a = complete(in, bmax);
    sort_frames_kernel<<<n_rows, kSortThreads, 0, st>>>(a, map, row0);
    return cudaGetLastError();
}

cudaError_t launch_pairs_sorted(const SortedArgs &in, int bmax, bool big, cudaStream_t st) {
    const SortedArgs a = complete(in, bmax);
    if (a.n_items <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.counter, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    const size_t smem = (size_t)a.teams * a.rows * kRowBytes;
    auto kern = big ? pairs_sorted_kernel<true> : pairs_sorted_kernel<false>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = std::min(sm_count(), (a.n_items + a.teams - 1) / a.teams);
    kern<<<grid, kThreads, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sorted_finish(const SortedArgs &in, int n_sys, int max_D, cudaStream_t st) {
    const unsigned n = (unsigned)((max_D + 31) / 32);
    sorted_finish_kernel<<<dim3(n, n, (unsigned)n_sys), 256, 0, st>>>(in);
    return cudaGetLastError();
}

}  // namespace pg
