// Inverse BWT on the GPU (sm_103a): psi table by a stable counting sort, then a parallel walk of many short chains.
//
// Conventions are the reference's (src/algo/sais/sais.c:12055-12082, the LF walk of tests/bwt_reference.py:270-290
// in adnaneben/kolmo): the L column is U with the sentinel re-inserted at row p0 = I[0]; row 0 of the sorted matrix
// is the sentinel rotation. Instead of LF (backwards) this decodes forwards with psi = LF^-1:
//   F row x holds the first byte of the suffix at row x, psi[x] is the row of the next suffix,
//   T[0] = F(p0), T[j + 1] = F(psi^(j+1)(p0)), and the walk ends at row 0 (the suffix of length 0).
// psi is built by a stable counting sort of the L column by byte (psi[C[c] + k] = row of the k-th c in L).
//
// Parallel decode (the chain idea of libsais's split decoder, sais.c:11573-11703, re-designed for a GPU):
//   * row p0 and about one row in MARK are marks; bit 31 of psi[x] flags "psi[x] is a mark" so a walk learns it
//     reached the next mark from the load it needs anyway. The regular marks are the rows (m * hmul) mod 2^k for
//     m = 1..n/MARK (2^k >= n, hmul odd near 2^k / golden ratio): a Weyl sequence, so the marks spread evenly over
//     every arithmetic progression of rows. Rows every MARK apart would leave whole stretches of a periodic text
//     unmarked (its rows interleave the periods), and one thread would walk each such stretch alone;
//   * one chain per mark walks psi until the next mark (or row 0), writing its bytes into its own CAPC-byte
//     buffer; a walk that reaches CAPC bytes closes its chain and continues as a new chain, so buffers never overflow
//     and no row is walked twice;
//   * chains are ranked by pointer jumping over (successor, length), in place; a chain's text position is n minus its
//     distance to the end of the text;
//   * chains are copied to their positions.
// A string that is not a valid BWT has more than one psi cycle: the walk from p0 then reaches row 0 before n bytes.
// That block is reported (-1) instead of decoded. Every loop is bounded by the number of rows.
#include "inv.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "kgbwt.h"

namespace cg = cooperative_groups;

namespace kgb {

constexpr int ITPB = 256;
constexpr u32 ITILE = 4096;
constexpr u32 MARK = 64;
// Small batches (the drop-in call on a block of a few MiB) mark more rows: they have too few chains to fill the GPU
// otherwise, and their walk is as long as the longest chain, about MARK ln(chains) rows. Whole inverse of one block, one
// row in 4 / 8 / 16 / 32 / 64, us (the mean of log lines and Markov bytes):
//    20 KB    61 / 67 / 79 / 94 / 172       768 KiB  98 / 92 / 111 / 136 / 197     3 MiB  213 / 162 / 162 / 188 / 271
//   128 KiB   62 / 67 / 80 / 103 / 155      1 MiB   111 / 98 / 97 / 123 / 172      4 MiB  294 / 198 / 168 / 181 / 220
//   192 KiB   68 / 76 / 94 / 120 / 180    1.5 MiB   137 / 117 / 128 / 148 / 225    5 MiB    - / - / 207 / 223 / 303
//   256 KiB   66 / 70 / 85 / 111 / 171      2 MiB   178 / 130 / 128 / 144 / 196    8 MiB    - / - / 260 / 239 / 281
//   512 KiB   82 / 76 / 86 / 119 / 168                                            16 MiB    - / - / 475 / 419 / 444
// Both sides of each line: one in 4 stays ahead to about 300 KiB (6-12% between 128 KiB, where the line lies, and there),
// 8 and 16 meet between 1 and 3 MiB, and past 4 MiB one in 16 or 32 would be ahead of 64 (46% at 5 MiB, 18% at 8, 6% at 16)
// at two to four times the chain records. At 30 MB one in 32 takes 0.10 ms off the walk and adds as much to the ranking and
// the copies.
static u32 mark_of(u64 total) { return total <= 128u << 10 ? 4 : total <= 1536u << 10 ? 8 : total <= 4u << 20 ? 16 : MARK; }
constexpr u32 CAPC = 256;
constexpr u32 ENDC = 0xFFFFFFFFu;
// The byte of a row (its place in C) by a table over the rows' leading bits: entry i holds the byte values of the first
// and last row of its range, and a search between the two (mostly none) ends the look-up.
constexpr u32 FT_LOG = 10, FT = 1u << FT_LOG;
// Tiles per chunk of the psi build: 16 on large batches, halved while the batch has at most CHUNKS_MIN chunks, so that
// small ones fill the GPU (a 1 MiB block: 256 chunks of one tile instead of 16 of 16).
constexpr u32 CHUNKT = 16, CHUNKS_MIN = 1024;
constexpr int STPB = 1024;   // threads of the chunk scan
// Its CTAs per block where blocks average more than so many chunks and the clusters fit the GPU at once. One block of 5,
// 32, 256 or 1024 chunks: 7, 8, 14 or 38 us with one CTA and 8, 9, 9.5 or 12.5 with eight; 64 blocks of 16 or 32 chunks: 8
// and 24, 400 blocks: 12.5 and 108.
constexpr u32 SCL = 8, SCL_CHUNKS = 64;

struct InvArgs {
    const u8 *U;
    u8 *out;
    u32 *psi;
    u32 *csum;
    u32 *C;
    u16 *ft;  // per block: FT entries, lowest byte value | highest << 8
    const InvBlock *blk;
    u32 B;
    u64 nchunk_all;
    u32 chunkt;  // tiles per chunk
    u64 nchains;
    u32 *len, *dyn, *status;
    // per chain record: successor (high word, ENDC: none) and length (low word); after the ranking the end of its list
    // and the length from its start to there. Read and written whole: both words always belong together.
    u64 *pair;
    u8 *buf;
    u32 nwalk;  // chains in the walk's sequence over all blocks (sum of nreg + 1)
    u64 cap_n;  // bytes of the text buffers (checked build)
    u32 nmax;   // length of the longest block
};

// Chain id of a regular mark at row q (in 1..nreg when q is one).
__device__ __forceinline__ u32 mark_id(u32 q, const InvBlock &B) { return (q * B.hinv) & B.hmask; }
__device__ __forceinline__ u32 is_mark(u32 q, const InvBlock &B) {
    if (q == 0) return 0;
    const u32 m = mark_id(q, B);
    return q == B.p0 || (m >= 1 && m <= B.nreg);
}
// Start row of chain id (0: p0; m >= 1: the m-th regular mark, or none (0) when that row is past n or is p0).
__device__ __forceinline__ u32 chain_start(u32 id, const InvBlock &B) {
    if (id == 0) return B.p0;
    const u32 q = (id * B.hmul) & B.hmask;
    return q > B.n || q == B.p0 ? 0u : q;
}

// Rows of a block are 0..n; an entry of its byte table spans 2^ft_shift of them.
__device__ __forceinline__ u32 ft_shift(u32 n) {
    const u32 bits = 32 - __clz(n);
    return bits > FT_LOG ? bits - FT_LOG : 0u;
}
// The largest c in [lo, hi] with C[c] <= row (C[lo] <= row).
__device__ __forceinline__ u32 f_search(const u32 *Cs, u32 row, u32 lo, u32 hi) {
    while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (Cs[mid] <= row) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The block of psi-build chunk q: the last one whose first chunk is <= q.
__device__ __forceinline__ u32 chunk_block(const InvArgs &a, u64 q) {
    u32 lo = 0, hi = a.B - 1;
    while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (__ldg(&a.blk[mid].chunk_base) <= q) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Per-chunk byte histograms (a chunk is chunkt consecutive tiles of one block), one per warp while counting. Bound by
// the latency of its loads, so a thread has two 16-byte words in flight (byte loads, one in flight: 0.136 ms for 64 MiB
// of prose and 0.39 for 216 MB of mixed blocks; now 0.042 and 0.155). BWT strings are full of short runs: a thread
// counts each run inside its word with one atomic, which also keeps lanes off each other's counters.
__global__ void __launch_bounds__(ITPB) k_inv_chunkhist(InvArgs a) {
    constexpr int NW = ITPB / 32, HU = 2;  // 16-byte words a thread has in flight
    __shared__ u32 h[NW][256];
    const u32 t = threadIdx.x;
    u32 *hw = h[warp_id()];
    for (u64 q = blockIdx.x; q < a.nchunk_all; q += gridDim.x) {
        const InvBlock B = a.blk[chunk_block(a, q)];
        const u32 start = (u32)(q - B.chunk_base) * (ITILE * a.chunkt);
        const u32 cnt = min(ITILE * a.chunkt, B.n - start);
        const u8 *src = a.U + (u64)B.off + start;
        // bytes before the first and after the last aligned word go one by one
        const u32 head = min(cnt, (u32)(0 - (uintptr_t)src) & 15u), nv = (cnt - head) / 16, tail = (cnt - head) & 15u;
        const uint4 *words = reinterpret_cast<const uint4 *>(src + head);
#pragma unroll
        for (int w = 0; w < NW; w++) h[w][t] = 0;
        __syncthreads();
        if (t < head) atomicAdd(&hw[src[t]], 1u);
        if (t < tail) atomicAdd(&hw[src[head + nv * 16 + t]], 1u);
        for (u32 i0 = t; i0 < nv; i0 += HU * ITPB) {
            uint4 v[HU];
#pragma unroll
            for (int k = 0; k < HU; k++)
                if (i0 + k * ITPB < nv) v[k] = __ldg(words + i0 + k * ITPB);
#pragma unroll
            for (int k = 0; k < HU; k++) {
                if (i0 + k * ITPB >= nv) break;
                const u32 w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                u32 cur = w[0] & 255u, len = 1;  // the run in progress
#pragma unroll
                for (int p = 1; p < 16; p++) {
                    const u32 c = __byte_perm(w[p / 4], 0, 0x4440 + p % 4);
                    if (c != cur) {
                        atomicAdd(&hw[cur], len);
                        cur = c;
                        len = 0;
                    }
                    len++;
                }
                atomicAdd(&hw[cur], len);
            }
        }
        __syncthreads();
        u32 sum = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) sum += h[w][t];
        a.csum[q * 256 + t] = sum;
        __syncthreads();
    }
}

// Per block: C array (C[c] = 1 + number of bytes below c: F row 0 is the sentinel), the table from a row's leading bits
// to its byte values, and the exclusive scan of the chunk histograms, so csum[q][c] becomes the first psi slot of chunk
// q's c bytes. CL CTAs share a block, each a slice of the byte values, whose totals they read from each other's shared
// memory; the threads of a CTA that share a byte value take consecutive chunks. One CTA is bound by what one SM reads
// and writes (1 MB of counts three times for a 64 MiB block).
template <int CL>
__device__ __forceinline__ void chunk_scan(const InvArgs &a) {
    constexpr u32 CW = 256 / CL, G = STPB / CW;
    __shared__ u32 ws[STPB / 32 + 1];
    __shared__ u32 part[G][CW];
    __shared__ u32 tots[CW];
    __shared__ u32 first[257];
    const u32 t = threadIdx.x, k = t % CW, g = t / CW, rank = CL > 1 ? blockIdx.x % CL : 0;
    const u32 c = rank * CW + k;
    for (u32 b = blockIdx.x / CL; b < a.B; b += gridDim.x / CL) {  // (the same blocks for every CTA of a cluster)
        const InvBlock B = a.blk[b];
        u32 *col = a.csum + (u64)B.chunk_base * 256 + c;
        const u32 per = (B.nchunk + G - 1) / G, q0 = min(B.nchunk, g * per), q1 = min(B.nchunk, q0 + per);
        u32 tot = 0;
        u32 q = q0;
        for (; q + 8 <= q1; q += 8) {
            u32 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = col[(u64)(q + i) * 256];
#pragma unroll
            for (int i = 0; i < 8; i++) tot += v[i];
        }
        for (; q < q1; q++) tot += col[(u64)q * 256];
        part[g][k] = tot;
        __syncthreads();
        if (g == 0) {
            u32 sum = 0;
            for (u32 w = 0; w < G; w++) sum += part[w][k];
            tots[k] = sum;
        }
        u32 sum = 0;
        if constexpr (CL > 1) {
            cg::cluster_group cl = cg::this_cluster();
            cl.sync();
            if (t < 256) sum = *cl.map_shared_rank(&tots[t % CW], t / CW);
        } else {
            __syncthreads();
            if (t < 256) sum = tots[t];
        }
        u32 all;
        const u32 cc = 1 + block_excl_sum<STPB>(sum, ws, &all);  // (threads 0..255 carry the sums)
        if (t < 256) {
            first[t] = cc;
            if (t / CW == rank) a.C[(u64)b * 257 + t] = cc;
            if (t == 255) {
                first[256] = 1 + all;
                if (rank == CL - 1) a.C[(u64)b * 257 + 256] = 1 + all;
            }
        }
        __syncthreads();
        static_assert(FT == STPB, "one entry per thread");
        if (t < FT / CL) {
            const u32 e = rank * (FT / CL) + t;
            const u32 sh = ft_shift(B.n);
            const u64 r0 = (u64)e << sh, r1 = ((u64)(e + 1) << sh) - 1;
            const u32 lo = f_search(first, (u32)max(r0, (u64)1), 0, 255);
            const u32 hi = f_search(first, (u32)min(r1, (u64)B.n), 0, 255);
            a.ft[(u64)b * FT + e] = (u16)(lo | max(lo, hi) << 8);
        }
        u32 run = first[c];
        for (u32 w = 0; w < g; w++) run += part[w][k];
        q = q0;
        for (; q + 8 <= q1; q += 8) {
            u32 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = col[(u64)(q + i) * 256];
#pragma unroll
            for (int i = 0; i < 8; i++) { col[(u64)(q + i) * 256] = run; run += v[i]; }
        }
        for (; q < q1; q++) {
            const u32 v = col[(u64)q * 256];
            col[(u64)q * 256] = run;
            run += v;
        }
        if (t == 0 && rank == 0) a.psi[B.psi_base] = B.p0 | 0x80000000u;  // psi[0]: the sentinel row leads to row p0
        if constexpr (CL > 1) cg::this_cluster().sync();  // the others have read tots: free for the next block, or to exit
        else __syncthreads();
    }
}
__global__ void __launch_bounds__(STPB) k_inv_chunkscan(InvArgs a) { chunk_scan<1>(a); }
__global__ void __cluster_dims__(SCL, 1, 1) __launch_bounds__(STPB) k_inv_chunkscan_cl(InvArgs a) { chunk_scan<SCL>(a); }

// Stable scatter, one CTA per chunk walking its tiles in order: psi[C[c] + occurrences of c before row q] = q,
// with the mark flag of q.
__global__ void __launch_bounds__(ITPB, 3) k_inv_scatter(InvArgs a) {
    constexpr int NW = ITPB / 32, IPT = ITILE / ITPB, WS = 32 * IPT;
    constexpr int RQ = 4;  // elements a lane ranks at once
    __shared__ u32 wc[NW][256];
    __shared__ u32 mask[NW][256 * RQ];  // (zero between uses)
    __shared__ u32 woff[NW][256];
    __shared__ u32 run_s[256];
    const u32 lane = lane_id(), warp = warp_id();
    for (int i = threadIdx.x; i < NW * 256 * RQ; i += ITPB) (&mask[0][0])[i] = 0;
    for (u64 q = blockIdx.x; q < a.nchunk_all; q += gridDim.x) {
        const u32 b = chunk_block(a, q);
        const InvBlock B = a.blk[b];
        const u32 cstart = (u32)(q - B.chunk_base) * (ITILE * a.chunkt);
        const u32 ccnt = min(ITILE * a.chunkt, B.n - cstart);
        run_s[threadIdx.x] = a.csum[q * 256 + threadIdx.x];
        u32 *psi = a.psi + B.psi_base;
        for (u32 t0 = 0; t0 < ccnt; t0 += ITILE) {
            const u32 start = cstart + t0;
            const u32 cnt = min(ITILE, ccnt - t0);
            for (int i = threadIdx.x; i < NW * 256; i += ITPB) (&wc[0][0])[i] = 0;
            __syncthreads();
            u32 cs[IPT], rk[IPT];
#pragma unroll
            for (int j = 0; j < IPT; j++) {
                const u32 x = warp * WS + j * 32 + lane;
                cs[j] = x < cnt ? (u32)a.U[(u64)B.off + start + x] : 0x100u;
            }
#pragma unroll
            for (int j = 0; j < IPT; j += RQ) {
                u32 c[RQ], r[RQ];
#pragma unroll
                for (int q = 0; q < RQ; q++) c[q] = cs[j + q];
                warp_rank<RQ, true>(mask[warp], wc[warp], c, r);
#pragma unroll
                for (int q = 0; q < RQ; q++) rk[j + q] = r[q];
            }
            __syncthreads();
            {
                u32 run = run_s[threadIdx.x];
#pragma unroll
                for (int w = 0; w < NW; w++) { woff[w][threadIdx.x] = run; run += wc[w][threadIdx.x]; }
                run_s[threadIdx.x] = run;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < IPT; j++) {
                const u32 x = warp * WS + j * 32 + lane;
                if (x < cnt) {
                    const u32 u = start + x;
                    const u32 qr = u + (u >= B.p0);
                    const u32 dst = woff[warp][cs[j]] + rk[j];
                    KGB_GUARD(dst >= 1 && dst <= B.n, &a.status[b], 0x100) psi[dst] = qr | (is_mark(qr, B) << 31);
                }
            }
            __syncthreads();
        }
    }
}

// CTAs per SM of the walk. More chains in flight spread over more blocks of a batch, whose psi tables then push each
// other out of L2 (mixed batch: 2.75 ms with 3, 4.16 with 6, 4.18 with 1; a 64 MiB block 1.36, 1.41 and 1.86).
constexpr int WALK_CTAS = 3;
constexpr int WSTEP = 8;  // rows between two looks at finished chains (one 8-byte word of text)
static_assert(CAPC % (2 * WSTEP) == 0, "records fill with whole 16-byte words");

// A finished chain record: its bytes and its successor.
__device__ __forceinline__ void close_chain(const InvArgs &a, u64 g, u32 len, u32 succ) {
    a.len[g] = len;
    a.pair[g] = (u64)succ << 32 | len;
}

// The block whose walk range holds chain q of the sequence over all blocks (blocks in order of qbase).
__device__ __forceinline__ u32 walk_block(const InvArgs &a, u32 q) {
    u32 lo = 0, hi = a.B - 1;
    while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (__ldg(&a.blk[mid].qbase) <= q) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Walk every chain: chain 0 of a block starts at p0, chain m >= 1 at its mark (none when that row is past n or is p0).
// Chains that reach CAPC bytes continue under a new id taken from the block's counter. ONE: the batch is one block,
// whose byte tables fit shared memory (a batch of several reads them through L1).
//
// Bound by dependent random psi loads: 77 G rows/s over the small blocks of a batch, 50-55 G on a 64 MiB block, whose
// 256 MiB table is twice L2 (independent 4-byte loads reach 79 G/s there, 280 where the table fits). One chain per
// thread; CTA c takes runs c, c + G, c + 2G, ... of ITPB chains of the sequence, its threads the next of them as they
// finish, so that the GPU works on one stretch of the sequence at a time. Chains are closed, stored and replaced only
// every WSTEP rows (an ended chain waits 4 rows of about 64), so that a warp runs that code once for all its lanes; the
// load of the next row is issued before the current row's byte is looked up; bytes leave in 16-byte words (4-byte words
// cost a quarter of the walk in partial sectors). The psi loads keep the default cache policy: L1::no_allocate marks
// their lines for early eviction from L2 too and took 4.13 ms where this takes 2.75 (mixed batch).
template <bool ONE>
__global__ void __launch_bounds__(ITPB, 6) k_inv_walk(InvArgs a) {
    __shared__ u32 Cs0[ONE ? 257 : 1];
    __shared__ u16 ft0[ONE ? FT : 1];
    __shared__ u32 qnext;
    if (threadIdx.x == 0) qnext = 0;
    if (ONE) {
        for (u32 i = threadIdx.x; i < 257; i += ITPB) Cs0[i] = a.C[i];
        for (u32 i = threadIdx.x; i < FT; i += ITPB) ft0[i] = a.ft[i];
    }
    __syncthreads();
    u32 b = 0, sh = 0, bn = 0, row = 0, v = 0, steps = 0, rec = 0;
    const u32 *psi = nullptr;
    // the thread's next chain; false: none is left
    auto take = [&]() -> bool {
        for (;;) {
            const u32 i = atomicAdd(&qnext, 1u);
            const u64 q64 = ((u64)(i / ITPB) * gridDim.x + blockIdx.x) * ITPB + i % ITPB;
            if (q64 >= a.nwalk) return false;
            const u32 q = (u32)q64;
            if (!ONE) b = walk_block(a, q);
            const InvBlock B = a.blk[b];
            const u32 id = q - B.qbase, start = chain_start(id, B);
            if (start == 0) continue;  // no such row, or chain 0 covers the mark at p0
            psi = a.psi + B.psi_base;
            bn = B.n;
            sh = ft_shift(B.n);
            row = start; steps = 0; rec = B.chain_base + id;
            v = __ldg(psi + row);
            return true;
        }
    };
    bool act = take();
    u64 prev = 0, cur = 0;  // the chain's last two 8-byte words
    // (the vote brings the warp's lanes together again: left to themselves they drift apart, nine to an instruction)
    while (__any_sync(0xffffffffu, act)) {
        // WSTEP rows; a lane whose chain ends waits for the others
        bool live = act;
        cur = 0;
#pragma unroll
        for (int j = 0; j < WSTEP; j++) {
            const bool go = live;
            const u32 r = row;
            if (go) {
                u32 nxt = v & 0x7FFFFFFFu;
                if (nxt > bn) {  // psi entries are rows 0..n: anything else is an internal error
                    a.status[b] = 3;
                    nxt = 0;
                }
                live = !(v >> 31) && nxt != 0;
                row = nxt;
                if (live) v = __ldg(psi + nxt);
                steps++;
            }
            u32 c = 0;
            if (go) {
                const u16 *ft = ONE ? ft0 : a.ft + (u64)b * FT;
                const u32 t = ft[r >> sh];
                c = f_search(ONE ? Cs0 : a.C + (u64)b * 257, r, t & 255u, t >> 8);
            }
            cur = cur >> 8 | (u64)c << 56;
            __syncwarp();
        }
        if (act) {
            const u32 w = (steps - 1) / WSTEP;
            if (w & 1 || !live)
                reinterpret_cast<ulonglong2 *>(a.buf + (u64)rec * CAPC)[w >> 1] =
                    w & 1 ? make_ulonglong2(prev, cur) : make_ulonglong2(cur, 0);
            prev = cur;
            if (!live) {
                const InvBlock B = a.blk[b];
                close_chain(a, rec, steps, row == 0 ? ENDC : B.chain_base + (row == B.p0 ? 0u : mark_id(row, B)));
                act = take();
            } else if (steps == CAPC) {
                const InvBlock B = a.blk[b];
                const u32 nid = B.nreg + 1 + atomicAdd(&a.dyn[b], 1u);
                if (nid >= B.chain_cap) {  // cannot happen for any input: each record covers CAPC rows
                    a.status[b] = 2;
                    close_chain(a, rec, steps, ENDC);
                    act = take();
                } else {
                    close_chain(a, rec, steps, B.chain_base + nid);
                    rec = B.chain_base + nid;
                    steps = 0;
                }
            }
        }
    }
}

// Chain ranking by pointer jumping in place, in one launch: every record's pair (where its list of chains has been
// followed to, the bytes on the way) is a true statement whenever it is read, so a thread may jump over a record that
// its own thread has not finished, is changing or has finished: it reads the pair whole (64-bit loads and stores) and
// moves on by what it says. No step waits for another. A record's loop ends at the end of its list, or, on a cycle off
// the main path (an invalid string), when the bytes pass the largest block or after as many jumps as there are records.
// (Against a launch per doubling step, two arrays a side: 0.30 ms for the 1.3 M chains of a 64 MiB block, 18 launches
// and 0.11 ms for a 1 MiB block.)
__global__ void __launch_bounds__(ITPB) k_inv_rank(InvArgs a) {
    volatile u64 *pair = a.pair;
    for (u64 g = (u64)blockIdx.x * ITPB + threadIdx.x; g < a.nchains; g += (u64)gridDim.x * ITPB) {
        u64 p = pair[g];
        u32 nx = (u32)(p >> 32), d = (u32)p;
        for (u64 jumps = 0; nx != ENDC && d <= a.nmax && jumps < a.nchains; jumps++) {
            p = pair[nx];
            const u64 s = (u64)d + (u32)p;
            nx = (u32)(p >> 32);
            d = s > 0xFFFFFFFFull ? 0xFFFFFFFFu : (u32)s;
            pair[g] = (u64)nx << 32 | d;
        }
    }
}

// Copy every chain on the main path to its text position (eight lanes per chain, aligned 4-byte words of the text) and
// set the block status.
__global__ void __launch_bounds__(ITPB) k_inv_emit(InvArgs a) {
    constexpr u32 EL = 8;  // lanes per chain
    const u32 sl = threadIdx.x & (EL - 1);
    const u64 gid = ((u64)blockIdx.x * ITPB + threadIdx.x) / EL, ng = (u64)gridDim.x * ITPB / EL;
    for (u64 g = gid; g < a.nchains; g += ng) {
        u32 lo = 0, hi = a.B - 1;  // block of chain g: last block with chain_base <= g
        while (lo < hi) {
            u32 mid = (lo + hi + 1) >> 1;
            if (a.blk[mid].chain_base <= g) lo = mid; else hi = mid - 1;
        }
        const InvBlock B = a.blk[lo];
        if (g >= (u64)B.chain_base + B.chain_cap) continue;
        const u64 p = a.pair[g];
        const u32 x = (u32)(p >> 32), d = (u32)p, L = a.len[g];
        if (g == B.chain_base && sl == 0 && a.status[lo] != 2) a.status[lo] = (x == ENDC && d == B.n) ? 0 : 1;
        if (x != ENDC || L == 0 || d > B.n || L > d) continue;
        const u64 dst = (u64)B.off + (B.n - d);
        if (!KGB_OK(L <= CAPC && dst + L <= a.cap_n, &a.status[lo], 0x100)) continue;
        const u32 *src = reinterpret_cast<const u32 *>(a.buf + g * CAPC);
        u8 *out = a.out + dst;
        const u32 sh = (u32)(reinterpret_cast<uintptr_t>(out) & 3u);  // the chain starts at byte sh of its first word
        const u32 nw = (sh + L + 3) / 4;
        for (u32 i = sl; i < nw; i += EL) {
            const int k = (int)(4 * i) - (int)sh, w = k >> 2;  // the word's first byte in the chain (negative: before it)
            const u32 lo4 = w >= 0 ? src[w] : 0u, hi4 = w + 1 < (int)(CAPC / 4) ? src[w + 1] : 0u;
            const u32 v = __funnelshift_r(lo4, hi4, 8 * (k & 3));
            if (k >= 0 && k + 4 <= (int)L) {
                *reinterpret_cast<u32 *>(out + k) = v;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (k + j >= 0 && k + j < (int)L) out[k + j] = (u8)(v >> (8 * j));
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ host engine
static size_t ialign(size_t x, size_t al) { return (x + al - 1) / al * al; }

InvEngine::InvEngine() {}
InvEngine::~InvEngine() { free_all(); }

void InvEngine::free_all() {
    if (up_pending) cudaEventSynchronize(up_done);
    if (up_done) cudaEventDestroy(up_done);
    up_done = nullptr;
    up_pending = false;
    if (cap_stream) cudaStreamDestroy(cap_stream);
    cap_stream = nullptr;
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
    gexec = nullptr; graph = nullptr;
    if (pool) cudaFree(pool);
    pool = nullptr;
    if (h_status) cudaFreeHost(h_status);
    h_status = nullptr;
    Ncap = Tcap = Ccap = Pcap = 0; Bcap = 0;
}

// The workspace for ncap text bytes, bcap blocks, tcap psi-build chunks, ccap chain records and pcap psi rows, in pool
// order.
template <typename Add>
void InvEngine::layout(u64 ncap, u32 bcap, u64 tcap, u64 ccap, u64 pcap, Add add) {
    add((void **)&own_U, ncap + 64);
    add((void **)&own_out, ncap + 64);
    add((void **)&d_psi, (pcap + 16) * 4);
    add((void **)&d_csum, tcap * 256 * 4);
    add((void **)&d_C, (size_t)bcap * 257 * 4);
    add((void **)&d_ft, (size_t)bcap * FT * 2);
    add((void **)&d_blk, (size_t)bcap * sizeof(InvBlock));
    add((void **)&d_len, ccap * 4);
    add((void **)&d_pair, ccap * 8);
    add((void **)&d_buf, ccap * CAPC);
    add((void **)&d_dyn, (size_t)bcap * 4);
    add((void **)&d_status, (size_t)bcap * 4);
}

int InvEngine::grow(u64 ncap, u32 bcap, u64 tcap, u64 ccap, u64 pcap) {
    if (ncap <= Ncap && bcap <= Bcap && tcap <= Tcap && ccap <= Ccap && pcap <= Pcap) return 0;
    ncap = std::max(ncap, Ncap); bcap = std::max(bcap, Bcap); tcap = std::max(tcap, Tcap); ccap = std::max(ccap, Ccap);
    pcap = std::max(pcap, Pcap);
    if (gexec) { cudaGraphExecDestroy(gexec); gexec = nullptr; }
    if (graph) { cudaGraphDestroy(graph); graph = nullptr; }
    if (pool) { cudaFree(pool); pool = nullptr; }
    struct Item { void **p; size_t bytes; };
    std::vector<Item> items;
    layout(ncap, bcap, tcap, ccap, pcap,
           [&](void **p, size_t bytes) { items.push_back({p, ialign(std::max<size_t>(bytes, 16), 256)}); });
    size_t total = 0;
    for (auto &it : items) total += it.bytes;
    cudaError_t e = cudaMalloc(&pool, total);
    if (e != cudaSuccess) {
        cudaGetLastError();
        pool = nullptr;
        Ncap = 0;
        return record_cuda_error(e, "cudaMalloc(inverse workspace)", __FILE__, __LINE__);
    }
    pool_bytes = total;
    size_t off = 0;
    for (auto &it : items) { *it.p = (char *)pool + off; off += it.bytes; }
    if (h_status) cudaFreeHost(h_status);
    KGB_CHECK(cudaMallocHost(&h_status, (size_t)bcap * sizeof(int)));
    Ncap = ncap; Bcap = bcap; Tcap = tcap; Ccap = ccap; Pcap = pcap;
    return 0;
}

// Mark parameters of a block of B.n bytes: the smallest 2^k >= n, the Weyl multiplier and its inverse. Rows run
// 0..n; when n = 2^k, row n maps to id 0 and is never a regular mark.
static void mark_params(InvBlock &B) {
    int k = 1;
    while (k < 32 && (1ull << k) < B.n) k++;
    B.hmask = (u32)((1ull << k) - 1);
    B.hmul = (u32)(0x9E3779B97F4A7C15ull >> (64 - k)) | 1u;
    u32 inv = B.hmul;  // Newton iteration for the inverse mod 2^32 (each step doubles the correct low bits)
    for (int it = 0; it < 5; it++) inv *= 2u - B.hmul * inv;
    B.hinv = inv;
}

static u32 mark_of(const u32 *n, int count) {
    u64 t = 0;
    for (int b = 0; b < count; b++) t += n[b];
    return mark_of(t);
}

static int plan_layout(const u32 *off, const u32 *n, const u32 *p0, int count, std::vector<InvBlock> &blk,
                       u64 &nchunk_all, u64 &nchains, u32 &chunkt,
                       u32 &nwalk, u64 &nrows) {
    blk.resize(count);
    nwalk = 0;
    nrows = 0;
    const u32 mark = mark_of(n, count);
    nchunk_all = 0; nchains = 0;
    auto chunks_of = [&](u32 t) {
        u64 c = 0;
        for (int b = 0; b < count; b++) c += ((u64)n[b] + ITILE * t - 1) / (ITILE * t);
        return c;
    };
    for (chunkt = CHUNKT; chunkt > 1 && chunks_of(chunkt / 2) <= CHUNKS_MIN; chunkt /= 2) {}
    for (int b = 0; b < count; b++) {
        if (n[b] < 2 || p0[b] < 1 || p0[b] > n[b]) return -1;
        InvBlock B;
        B.off = off[b]; B.n = n[b]; B.p0 = p0[b];
        B.chunk_base = (u32)nchunk_all;
        B.nchunk = (u32)(((u64)n[b] + ITILE * chunkt - 1) / (ITILE * chunkt));
        B.nreg = n[b] / mark;
        mark_params(B);
        B.chain_base = (u32)nchains;
        B.chain_cap = B.nreg + 1 + n[b] / CAPC + 4;
        B.qbase = nwalk;
        B.psi_base = nrows;
        nrows += (u64)n[b] + 1;
        nwalk += B.nreg + 1;
        nchunk_all += B.nchunk;
        nchains += B.chain_cap;
        blk[b] = B;
        if (nchunk_all > 0xFFFF0000ull || nchains > 0xFFFF0000ull || nwalk > 0xFFFF0000u) return -1;
    }
    return 0;
}

u64 InvEngine::estimate_bytes(const u32 *n, int count) {
    std::vector<u32> off(count), p0(count, 1);
    u64 o = 0;
    for (int b = 0; b < count; b++) { off[b] = (u32)o; o += ((u64)n[b] + 15) / 16 * 16; }
    std::vector<InvBlock> blk;
    u64 nch = 0, nchains_ = 0, nr = 0;
    u32 ct = 0, nw = 0;
    if (plan_layout(off.data(), n, p0.data(), count, blk, nch, nchains_, ct, nw, nr)) return ~0ull;
    u64 total = 0;
    layout(std::max<u64>(o, Ncap), std::max<u32>((u32)count, Bcap), std::max<u64>(nch, Tcap),
           std::max<u64>(nchains_, Ccap), std::max<u64>(nr, Pcap),
           [&](void **, size_t bytes) { total += ialign(std::max<size_t>(bytes, 16), 256); });
    return total;
}

// The block table's upload of the call before: its source is changed only once it is done.
int InvEngine::uploads_done() {
    if (!up_pending) return 0;
    up_pending = false;
    KGB_CHECK(cudaEventSynchronize(up_done));
    return 0;
}

int InvEngine::plan(const u32 *n, const u32 *p0, int count) {
    if (count <= 0) return -1;
    if (int rc = uploads_done()) return rc;
    h_off.resize(count);
    u64 off = 0;
    for (int b = 0; b < count; b++) {
        h_off[b] = (u32)off;
        off += ((u64)n[b] + 15) / 16 * 16;
        if (off > 0xFFFF0000ull) return -1;
    }
    if (plan_layout(h_off.data(), n, p0, count, h_blk, nchunk_all, nchains, chunkt, nwalk, nrows)) return -1;
    N = off; B = (u32)count;
    int rc = grow(N, B, nchunk_all, nchains, nrows);
    if (rc) return rc;
    ext = false;
    d_U = own_U; d_out = own_out;
    return 0;
}

int InvEngine::plan_external(const u32 *off, const u32 *n, const u32 *p0, int count, u8 *dU, u8 *dOut) {
    if (count <= 0) return -1;
    if (int rc = uploads_done()) return rc;
    h_off.assign(off, off + count);
    if (plan_layout(off, n, p0, count, h_blk, nchunk_all, nchains, chunkt, nwalk, nrows)) return -1;
    u64 end = 0;
    for (int b = 0; b < count; b++) end = std::max<u64>(end, (u64)off[b] + n[b]);
    N = end; B = (u32)count;
    int rc = grow(N, B, nchunk_all, nchains, nrows);
    if (rc) return rc;
    ext = true;
    d_U = dU; d_out = dOut;
    return 0;
}

u32 InvEngine::nmax() const {
    u32 m = 0;
    for (const InvBlock &b : h_blk) m = std::max(m, b.n);
    return m;
}

int InvEngine::enqueue(cudaStream_t s, long long *launches) {
    InvArgs a;
    memset(&a, 0, sizeof(a));
    a.U = d_U; a.out = d_out; a.psi = d_psi; a.csum = d_csum; a.C = d_C; a.ft = d_ft; a.blk = d_blk; a.B = B;
    a.nchunk_all = nchunk_all; a.chunkt = chunkt; a.nchains = nchains; a.len = d_len; a.pair = d_pair; a.dyn = d_dyn;
    a.status = d_status; a.buf = d_buf; a.nwalk = nwalk; a.cap_n = Ncap;
    a.nmax = nmax();
    const int g8 = (int)std::min<u64>((u64)sm_count * 8, (nchains + ITPB - 1) / ITPB);
    KGB_CHECK(cudaMemsetAsync(d_len, 0, nchains * 4, s));
    KGB_CHECK(cudaMemsetAsync(d_pair, 0xFF, nchains * 8, s));
    KGB_CHECK(cudaMemsetAsync(d_dyn, 0, (size_t)B * 4, s));
    KGB_CHECK(cudaMemsetAsync(d_status, 0, (size_t)B * 4, s));
    Profiler *P = prof_run ? &prof : nullptr;
    auto go = [&](int kid, u32 elems, auto fn) -> cudaError_t {
        (*launches)++;
        if (!P) { fn(); return cudaGetLastError(); }
        P->tag(kid, elems);
        return P->launch(s, [&]() -> cudaError_t { fn(); return cudaGetLastError(); });
    };
    const u32 nbytes = (u32)std::min<u64>(N, 0xFFFFFFFFull);
    const int gch = (int)std::min<u64>(nchunk_all, (u64)sm_count * 8);
    KGB_CHECK(go(K_INV_TILEHIST, nbytes, [&] { k_inv_chunkhist<<<gch, ITPB, 0, s>>>(a); }));
    KGB_CHECK(go(K_INV_COLSCAN, (u32)nchunk_all, [&] {
        const u32 nb = std::min<u32>(B, 4096u);
        if (nchunk_all > (u64)B * SCL_CHUNKS && B * SCL <= (u32)sm_count) k_inv_chunkscan_cl<<<nb * SCL, STPB, 0, s>>>(a);
        else k_inv_chunkscan<<<nb, STPB, 0, s>>>(a);
    }));
    KGB_CHECK(go(K_INV_SCATTER, nbytes, [&] { k_inv_scatter<<<gch, ITPB, 0, s>>>(a); }));
    // the CTAs the GPU holds at once, or fewer when there are fewer chains than threads
    const int gw = (int)std::max<u64>(1, std::min<u64>((u64)walk_grid, ((u64)nwalk + ITPB - 1) / ITPB));
    KGB_CHECK(go(K_INV_WALK, nbytes, [&] {
        if (B == 1) k_inv_walk<true><<<gw, ITPB, 0, s>>>(a);
        else k_inv_walk<false><<<gw, ITPB, 0, s>>>(a);
    }));
    KGB_CHECK(go(K_INV_JUMP, (u32)nchains, [&] { k_inv_rank<<<g8, ITPB, 0, s>>>(a); }));
    KGB_CHECK(go(K_INV_EMIT, nbytes, [&] { k_inv_emit<<<sm_count * 8, ITPB, 0, s>>>(a); }));
    return 0;
}

int InvEngine::run(cudaStream_t s, bool use_graph) {
    stats = InvStats{};
    if (!up_done) KGB_CHECK(cudaEventCreateWithFlags(&up_done, cudaEventDisableTiming));
    if (!sm_count) {
        int dev;
        KGB_CHECK(cudaGetDevice(&dev));
        KGB_CHECK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
        walk_grid = WALK_CTAS * sm_count;
    }
    KGB_CHECK(cudaMemcpyAsync(d_blk, h_blk.data(), h_blk.size() * sizeof(InvBlock), cudaMemcpyHostToDevice, s));
    KGB_CHECK(cudaEventRecord(up_done, s));
    up_pending = true;
    prof.reset();
    prof_run = !use_graph && prof.on;
    if (!use_graph) return enqueue(s, &stats.launches);
    prof_run = false;
    const GraphKey key{N, Ncap, (u64)nchunk_all, (u64)nchains, (u32)B, chunkt, nwalk, nmax(), d_U, d_out};
    if (!gexec || !(key == graph_key)) {
        if (!(seen_valid && key == seen_key)) {  // first sight of this shape: plain launches, no capture
            seen_key = key;
            seen_valid = true;
            return enqueue(s, &stats.launches);
        }
        if (gexec) { cudaGraphExecDestroy(gexec); gexec = nullptr; }
        if (graph) { cudaGraphDestroy(graph); graph = nullptr; }
        if (!cap_stream) KGB_CHECK(cudaStreamCreateWithFlags(&cap_stream, cudaStreamNonBlocking));
        KGB_CHECK(cudaStreamBeginCapture(cap_stream, cudaStreamCaptureModeThreadLocal));
        long long dummy = 0;
        int rc = enqueue(cap_stream, &dummy);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(cap_stream, &g);
        if (rc) { if (g) cudaGraphDestroy(g); return rc; }
        KGB_CHECK(e);
        graph = g;
        KGB_CHECK(cudaGraphInstantiate(&gexec, graph, 0));
        graph_key = key;
    }
    KGB_CHECK(cudaGraphLaunch(gexec, s));
    stats.launches = -1;
    return 0;
}

int InvEngine::fetch_status(cudaStream_t s, std::vector<int> &status) {
    KGB_CHECK(cudaMemcpyAsync(h_status, d_status, (size_t)B * sizeof(int), cudaMemcpyDeviceToHost, s));
    KGB_CHECK(cudaStreamSynchronize(s));
    status.assign(h_status, h_status + B);
    return 0;
}

}  // namespace kgb

// ------------------------------------------------------------------------------------------------ allocation-free
// Inverse BWT for callers that cannot allocate device memory: code that runs where cudaMalloc is not allowed or not
// wanted (a host that owns every device allocation through its own pool, a plugin loaded into such a host, a
// process that must not grow its device footprint after start-up). Its scratch is one file-scope device array
// sized for one block of at most NOALLOC_MAX_N bytes; every GPU that loads this library holds that array
// (about 2.5 MB) until the process exits. The caller passes device input and output buffers.
namespace kgb {

constexpr u32 NOALLOC_MAX_N = 1u << 18;  // 256 KiB
constexpr u32 NA_CHUNKS = NOALLOC_MAX_N / ITILE;  // chunks of one tile
constexpr u32 NA_NREG = NOALLOC_MAX_N / MARK;
constexpr u32 NA_CHAINS = NA_NREG + 1 + NOALLOC_MAX_N / CAPC + 4;

struct NoAllocScratch {
    u32 psi[NOALLOC_MAX_N + 16];
    u32 csum[NA_CHUNKS * 256];
    u32 C[264];
    u16 ft[FT];
    InvBlock blk[1];
    u64 pair[NA_CHAINS];
    u32 len[NA_CHAINS];
    u32 dyn[4], status[4];
    __align__(16) u8 buf[(size_t)NA_CHAINS * CAPC];
};

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

// Device address of the scratch array, looked up once per device (with that device current).
static NoAllocScratch *noalloc_scratch(int *rc) {
    static std::mutex mu;
    static NoAllocScratch *addr[128] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { *rc = record_cuda_error(e, "cudaGetDevice", __FILE__, __LINE__); return nullptr; }
    if (dev < 0 || dev >= 128) { record_error("device index out of range"); *rc = -2; return nullptr; }
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) { *rc = record_cuda_error(e, "cudaGetSymbolAddress", __FILE__, __LINE__); return nullptr; }
        addr[dev] = reinterpret_cast<NoAllocScratch *>(p);
    }
    *rc = 0;
    return addr[dev];
}

static int unbwt_noalloc(const u8 *dU, u8 *dT, u32 n, u32 p0, cudaStream_t s) {
    int rc = 0;
    NoAllocScratch *S = noalloc_scratch(&rc);
    if (!S) return rc;
    // the block's table entry, on the stack
    InvBlock B;
    B.off = 0; B.n = n; B.p0 = p0;
    B.chunk_base = 0; B.nchunk = (n + ITILE - 1) / ITILE;
    B.nreg = n / MARK; B.chain_base = 0; B.chain_cap = B.nreg + 1 + n / CAPC + 4; B.qbase = 0; B.psi_base = 0;
    mark_params(B);
    KGB_CHECK(cudaMemcpyAsync(S->blk, &B, sizeof(B), cudaMemcpyHostToDevice, s));
    // the array keeps the previous call's contents: reset what must start at zero (or at "no successor")
    KGB_CHECK(cudaMemsetAsync(S->len, 0, sizeof(u32) * B.chain_cap, s));
    KGB_CHECK(cudaMemsetAsync(S->pair, 0xFF, sizeof(u64) * B.chain_cap, s));
    KGB_CHECK(cudaMemsetAsync(S->dyn, 0, sizeof(S->dyn), s));
    KGB_CHECK(cudaMemsetAsync(S->status, 0, sizeof(S->status), s));
    InvArgs a;
    memset(&a, 0, sizeof(a));
    a.U = dU; a.out = dT; a.psi = S->psi; a.csum = S->csum; a.C = S->C; a.ft = S->ft; a.blk = S->blk; a.B = 1;
    a.nchunk_all = B.nchunk; a.chunkt = 1; a.nchains = B.chain_cap; a.len = S->len; a.pair = S->pair; a.dyn = S->dyn;
    a.status = S->status; a.buf = S->buf; a.nwalk = B.nreg + 1; a.cap_n = n; a.nmax = n;
    k_inv_chunkhist<<<B.nchunk, ITPB, 0, s>>>(a);
    k_inv_chunkscan<<<1, STPB, 0, s>>>(a);
    k_inv_scatter<<<B.nchunk, ITPB, 0, s>>>(a);
    k_inv_walk<true><<<(B.nreg + ITPB) / ITPB, ITPB, 0, s>>>(a);
    const int g = (int)((B.chain_cap + ITPB - 1) / ITPB);
    k_inv_rank<<<g, ITPB, 0, s>>>(a);
    k_inv_emit<<<8 * g, ITPB, 0, s>>>(a);
    KGB_CHECK(cudaGetLastError());
    u32 status = 0;
    KGB_CHECK(cudaMemcpyAsync(&status, S->status, sizeof(u32), cudaMemcpyDeviceToHost, s));
    KGB_CHECK(cudaStreamSynchronize(s));
    if (status) { record_error("inverse BWT: not a valid BWT string for its primary index"); return -1; }
    return 0;
}

}  // namespace kgb

extern "C" int32_t kgbwt_unbwt_noalloc(const uint8_t *dU, uint8_t *dT, int32_t n, int32_t p0, void *stream) {
    if (!dU || !dT || n < 2 || p0 < 1 || p0 > n) {
        kgb::record_error("kgbwt_unbwt_noalloc: bad arguments (device buffers, n >= 2, 1 <= p0 <= n)");
        return -1;
    }
    if ((uint32_t)n > kgb::NOALLOC_MAX_N) {
        kgb::record_error("kgbwt_unbwt_noalloc: n exceeds the maximum of 262144 bytes of the static scratch");
        return -1;
    }
    // both buffers must be memory the device can address (device or managed allocations): a host pointer would
    // send the kernels to an address they cannot use
    for (const void *p : {(const void *)dU, (const void *)dT}) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess ||
            (at.type != cudaMemoryTypeDevice && at.type != cudaMemoryTypeManaged)) {
            cudaGetLastError();
            kgb::record_error("kgbwt_unbwt_noalloc: dU and dT must be device (or managed) memory");
            return -1;
        }
    }
    // every call reads its status back and waits for the stream, which a stream under capture does not allow
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing((cudaStream_t)stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        kgb::record_error("kgbwt_unbwt_noalloc: the stream is being captured; this call synchronises with it");
        return -1;
    }
    return kgb::unbwt_noalloc(dU, dT, (kgb::u32)n, (kgb::u32)p0, (cudaStream_t)stream);
}
