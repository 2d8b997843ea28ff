// Round 0 of the forward sort as one LSD radix sort: the suffixes of each block of the batch are sorted by a W-byte
// key, with one pass per varying key byte (single-pass scatter with decoupled look-back), then a segmentation turns the
// sorted order into ranks, finished suffixes and the rank rounds' groups (tiny, medium, small and large lists). The
// sort tiles never straddle two blocks: every block's suffixes keep their own range of the dense order (the block's
// soff onward), a pass takes each tile's digit bases from its own block's counts and looks back only over the block's
// earlier tiles, so the block index is neither carried nor sorted. The passes move 8-byte (id, key) items whose key is
// the 4-byte group of key bytes the passes of that group sort; the last pass of a group writes the next group's key
// instead of its own, so each pass reads and writes 16 B per suffix. Included by fwd.cu inside namespace kgb, after the
// kernels it shares (FwdArgs, resolve, tile-map writers).
//
// Raw keys (W = 16 or 12): the first W bytes of the suffix, zero-padded. The first pass builds its items from the text
// (ids still in text order, so the loads coalesce), a group's last pass gathers the next group's bytes from the text.
//
// Coded keys (W = 8): the first 64 bits of the suffix written in an order-preserving prefix code of its block's bytes.
// A block's bytes take codewords of 1..CODE_MAX bits from a weight-balanced binary tree over its byte histogram
// (alphabetic, so comparing encoded suffixes as bit strings compares the suffixes; the smallest byte's codeword is all
// zeros and zeros follow the block's end, so a suffix that ends sorts with the ones that go on in smallest bytes, in
// one group). Suffixes with equal keys share as many bytes as their key holds whole codewords; the smallest such count
// over the groups of two or more is what round 0 has sorted (Ctl::h0), and each group carries its own. Raw bytes take
// 8 bits each whatever they hold, coded ones about their order-0 entropy (prose 4.7 bits, log lines 5.1, ACGT 2.0,
// 64-symbol Markov 6.0), so eight passes reach 10-32 characters where sixteen reach 16.
#pragma once
// (included inside namespace kgb)

constexpr int LSD_IPT = 16, LSD_TILE = TPB * LSD_IPT;  // elements per sort tile
// digit slots: slot s sorts key byte 15 - s, carried in key group (15 - s) / 4 (bytes 4g..4g+3, big-endian)
constexpr int NSLOT = 16;
static_assert(NSLOT <= 32, "the look-back epoch holds the slot in 5 bits");
constexpr int SEG_IPT = 16, SEG_TILE = TPB * SEG_IPT;  // positions per segmentation tile (SEG_IPT <= 32)
// look-back words: epoch (32 bits: call sequence << 5 | digit slot) | flag (2 bits) | value (30 bits); a word of another
// epoch (an earlier slot or call) counts as not yet published
constexpr u64 ST_AGG = 1ull << 30, ST_PRE = 2ull << 30, ST_VAL = (1ull << 30) - 1;
constexpr u64 ST_EPOCH = 0xFFFFFFFF00000000ull;
constexpr int LB_WIN = 4;  // look-back window (predecessor words read per step; 8: 0.5% slower on 64 MiB of prose)

// Which keys: the tuning table's choice per batch size, by measurement; it takes coded keys throughout. They halve the
// passes, compare more in the segmentation and leave slightly larger groups. Forward call in ms at 1, 4, 16 and 64 MiB,
// coded against raw 16 bytes (medians of 7 rounds in turn, which agree within 1%): log lines 0.39 0.87 2.98 12.63 against
// 0.45 1.00 3.27 12.98, Markov bytes 0.22 0.51 1.65 7.50 against 0.36 0.92 2.76 10.72, prose 0.48 0.98 3.48 14.81 against
// 0.47 1.17 3.80 14.74, prose copied over and over 1.40 3.45 6.19 (to 16 MiB) against 1.37 3.50 6.24; 96 mixed blocks 36.5
// against 41.0. So prose gains in the middle sizes only and is 2% slower at 1 MiB (0.5% at 64), which a rule by size
// cannot tell from the texts that gain 3-38% there.
// Raw keys stay for engines that ask for 12 or 16 bytes and where no table is loaded.
__host__ __device__ __forceinline__ bool lsd_coded(const FwdArgs &a) { return a.lsd_bytes == 8; }
__device__ __forceinline__ u32 active_slots(const Ctl *c) { return c->lsd_act; }  // bit s: slot s varies

// A block's code table: entry c holds byte c's codeword left-aligned in bits 31..20 and its length in bits 4..0, entry
// CODE_PAD the symbol past the block's end (zeros of the smallest byte's length), entry CODE_MIN the smallest byte.
constexpr u32 CODE_MAX = 12, CODE_BITS = 0xFFF00000u, CODE_PAD = 256, CODE_MIN = 257, CODE_ROW = 260;  // words

// The 16 text bytes from position q < end on, and the byte before them. Random text reads are bound by the lines a
// warp's loads touch (one a cycle and SM), not by their bytes, so they take two aligned 16-byte granules instead of
// three 8-byte words. Every granule read holds a byte of the block: it ends at most 15 bytes past the block and begins
// in the granule of its first byte.
struct Text16 {
    u64 w, w2;        // bytes q..q+7 and q+8..q+15
    u8 before;        // byte q - 1 when it lies in the first granule
    bool has_before;  // (q not at a granule's start)
};
__device__ __forceinline__ Text16 text16(const u8 *__restrict__ T, u64 q, u64 end) {
    const u8 *p = T + q;
    const u32 s = (u32)(reinterpret_cast<uintptr_t>(p) & 15u);
    const ulonglong2 *g = reinterpret_cast<const ulonglong2 *>(p - s);
    Text16 r;
    const ulonglong2 x = __ldg(g);
    ulonglong2 y = make_ulonglong2(0, 0);
    if (q + (16 - s) < end) y = __ldg(g + 1);
    const u32 h = (s & 7) * 8;
    const u64 a = s & 8 ? x.y : x.x, b = s & 8 ? y.x : x.y, c = s & 8 ? y.y : y.x;
    r.w = h ? (a >> h) | (b << (64 - h)) : a;
    r.w2 = h ? (b >> h) | (c << (64 - h)) : b;
    r.has_before = s != 0;
    r.before = (u8)((((s - 1) & 8) ? x.y : x.x) >> (8 * ((s - 1) & 7)));
    return r;
}
// As text16, with every byte past the block's end replaced by the block's smallest byte (what zeros past the end of a
// coded suffix read as).
__device__ __forceinline__ Text16 text16_padded(const u8 *__restrict__ T, u64 q, u64 end, u32 smallest) {
    const u64 fill = 0x0101010101010101ull * smallest;
    Text16 r;
    r.w = r.w2 = fill;
    r.before = 0;
    r.has_before = false;
    if (q >= end) return r;
    r = text16(T, q, end);
    const u64 rem = end - q;
    if (rem < 8) r.w = (r.w & ~(~0ull << (8 * rem))) | fill << (8 * rem);
    if (rem <= 8) r.w2 = fill;
    else if (rem < 16) r.w2 = (r.w2 & ~(~0ull << (8 * (rem - 8)))) | fill << (8 * (rem - 8));
    return r;
}

// The first 32 NG key bits of the suffix at q into k[], and into m[] the bits where a codeword ends. Eight symbols a
// step: their look-ups are independent, and codewords are joined in pairs before they enter the bit windows. The loop
// ends: every table entry is at least one bit long.
template <int NG>
__device__ __forceinline__ void lsd_encode(const u8 *__restrict__ T, const u32 *tab, u64 q, u64 end, u32 *k, u32 *m) {
    u32 hi = 0, lo = 0, mhi = 0, mlo = 0, fill = 0;
    for (int g = 0; g < NG; q += 8) {
        u64 w = 0;
        if (q < end) w = text16(T, q, end).w;
        u32 e[8];
#pragma unroll
        for (int j = 0; j < 8; j++) e[j] = tab[q + j < end ? (u32)(w >> (8 * j)) & 0xFFu : CODE_PAD];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            // (the funnel shift takes its count modulo 32: a length in the low five bits; two lengths sum below 32)
            const u32 pair = (e[j] & CODE_BITS) | __funnelshift_r(e[j + 1] & CODE_BITS, 0u, e[j]);
            const u32 l = (e[j] + e[j + 1]) & 31u, ends = 1u << (32 - (e[j] & 31u)) | 1u << (32 - l);
            hi |= pair >> fill;
            lo |= __funnelshift_r(0u, pair, fill);
            mhi |= ends >> fill;
            mlo |= __funnelshift_r(0u, ends, fill);
            fill += l;
            if (fill >= 32) {
#pragma unroll
                for (int x = 0; x < NG; x++) if (x == g) { k[x] = hi; m[x] = mhi; }
                g++;
                hi = lo; mhi = mlo;
                lo = mlo = 0;
                fill -= 32;
            }
        }
    }
}
// The zero-padded 8-byte text word at position q of a block ending at end, as a big-endian word (0 past the end).
__device__ __forceinline__ u64 lsd_word(const u8 *__restrict__ T, u64 q, u64 end) {
    if (q >= end) return 0;
    u64 k = load_be64(T, q);
    const u64 rem = end - q;
    if (rem < 8) k &= ~0ull << (8 * (8 - rem));
    return k;
}
// Raw keys: key group g (prefix bytes 4g..4g+3) of the suffix at id, big-endian, zero past the block end.
__device__ __forceinline__ u32 lsd_raw_group(const u8 *__restrict__ T, u32 id, u32 g, u64 end) {
    return (u32)(lsd_word(T, (u64)id + 4 * g, end) >> 32);
}
// Coded keys: key group g (0 or 1) of every suffix, and the whole codewords of its key, in text order (dense order of
// the batch). They live in lists that are empty in round 0, the last group's in the buffer the first pass reads from.
__device__ __forceinline__ u32 *lsd_keys_of(const FwdArgs &a, u32 g) { return g ? a.lval[0] : a.lists[L_KS].eid; }
__device__ __forceinline__ u8 *lsd_whole_of(const FwdArgs &a) { return reinterpret_cast<u8 *>(a.lists[L_M0].eid); }
// Key group of slot s.
__device__ __forceinline__ u32 lsd_slot_group(int slot) { return (15u - (u32)slot) >> 2; }

// The block of sort tile t: the last block whose first tile (lt0) is <= t (blocks in batch order, lt0 ascending).
__device__ __forceinline__ u32 blk_of_tile(const FwdArgs &a, u32 t) {
    u32 lo = 0, hi = a.B - 1;
    while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (__ldg(&a.blk[mid].lt0) <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}
// The block holding dense position p, searched within blocks [lo, hi]: the last block whose soff is <= p.
__device__ __forceinline__ u32 blk_of_pos(const FwdArgs &a, u32 p, u32 lo, u32 hi) {
    while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (__ldg(&a.blk[mid].soff) <= p) lo = mid; else hi = mid - 1;
    }
    return lo;
}
// A sort tile: its block, first dense position and element count.
struct LsdTile {
    u32 b, base, cnt;
};
__device__ __forceinline__ LsdTile lsd_tile(const FwdArgs &a, u32 t) {
    LsdTile r;
    r.b = blk_of_tile(a, t);
    const BlockInfo bi = a.blk[r.b];
    const u32 k = (t - bi.lt0) * (u32)LSD_TILE;
    r.base = bi.soff + k;
    r.cnt = min((u32)LSD_TILE, bi.n - k);
    return r;
}

// Start: clear the blocks' byte and digit histograms, the tile counters, the active mask and the resolved count.
__global__ void k_lsd_begin(FwdArgs a) {
    Ctl *c = a.ctl;
    const u64 nh = (u64)a.B * 256;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += (u64)gridDim.x * blockDim.x) a.lhist[i] = 0;
    const u64 nb = lsd_coded(a) ? (u64)a.B * (NSLOT * 256 / 4) : 0;  // (raw keys: the digit bases are written whole)
    uint4 *base4 = reinterpret_cast<uint4 *>(a.lbase);
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += (u64)gridDim.x * blockDim.x)
        base4[i] = make_uint4(0, 0, 0, 0);
    if (blockIdx.x == 0) {
        if (threadIdx.x < NSLOT) a.ltile[threadIdx.x] = 0;
        if (threadIdx.x == 0) {
            // round 0 lists no finished suffixes: with every id counted as finished, round 1's fixup copies the
            // whole rank buffer
            c->cnt[L_R0 + c->rpar] = a.idn;
            c->lsd_act = 0;
            // coded keys: the segmentation takes the minimum over the groups that survive
            c->h0 = lsd_coded(a) ? 0xFFFFFFFFu : a.lsd_bytes;
            c->m = a.blk[a.B - 1].soff + a.blk[a.B - 1].n;
        }
    }
}

// Each block's byte histogram, from which its code follows, and row 0 of its L column. CTA c takes a
// contiguous run of sort tiles and adds its shared histogram into a block's row when the run leaves it.
__global__ void __launch_bounds__(TPB) k_lsd_key0(FwdArgs a) {
    __shared__ u32 hs[256];
    const u32 nt = a.ctl->lsd_tiles;
    const u32 per = (nt + gridDim.x - 1) / gridDim.x;
    const u32 t0 = blockIdx.x * per, t1 = min(nt, t0 + per);
    hs[threadIdx.x] = 0;
    __syncthreads();
    u32 cur = ~0u;  // block whose counts hs holds
    for (u32 t = t0; t < t1; t++) {
        const LsdTile tl = lsd_tile(a, t);
        if (tl.b != cur) {
            if (cur != ~0u) {
                __syncthreads();
                const u32 v = hs[threadIdx.x];
                if (v) atomicAdd(&a.lhist[(u64)cur * 256 + threadIdx.x], v);
                hs[threadIdx.x] = 0;
                __syncthreads();
            }
            cur = tl.b;
        }
        const BlockInfo bi = a.blk[tl.b];
        const u64 end = (u64)bi.off + bi.n;
        // row 0 of the L column (the sentinel rotation) holds the block's last byte
        if (t == bi.lt0 && threadIdx.x == 0) a.L[(u64)bi.off + tl.b] = a.T[end - 1];
        const u32 id0 = bi.off + (tl.base - bi.soff);
        for (u32 j = threadIdx.x; j < tl.cnt; j += TPB) atomicAdd(&hs[__ldg(a.T + id0 + j)], 1u);
    }
    __syncthreads();
    if (cur != ~0u && hs[threadIdx.x]) atomicAdd(&a.lhist[(u64)cur * 256 + threadIdx.x], hs[threadIdx.x]);
}

// The code of every block (CTAs over blocks, 256 threads, thread = byte value). The bytes that occur, in order, are
// split again and again at the weight midpoint (the cut nearest to half of the interval's count, kept within what the
// remaining levels can hold); a byte's codeword is its path. Every thread walks its own path over the cumulative
// counts in shared memory: at most CODE_MAX levels of a binary search.
__global__ void __launch_bounds__(TPB) k_lsd_code(FwdArgs a) {
    __shared__ u32 C[257];
    __shared__ u32 ws[TPB / 32 + 1];
    __shared__ u32 len0;
    const u32 x = threadIdx.x;
    for (u32 b = blockIdx.x; b < a.B; b += gridDim.x) {
        const u32 h = a.lhist[(u64)b * 256 + x];
        u32 ns, n;
        const u32 idx = block_excl_sum<TPB>(h != 0, ws, &ns);  // the byte's index among those that occur
        const u32 before = block_excl_sum<TPB>(h, ws, &n);
        if (h) C[idx] = before;
        if (x == 0) C[ns] = n;
        __syncthreads();
        u32 code = 0, len = 0;
        if (h) {
            u32 lo = 0, hi = ns;
            while (hi - lo > 1) {
                const u32 half = 1u << (CODE_MAX - len - 1);
                const u32 c0 = C[lo], c1 = C[hi], mid = c0 + (c1 - c0) / 2;
                u32 l = lo + 1, r = hi - 1;  // the first cut in (lo, hi) at or past the midpoint (hi - 1 if none)
                while (l < r) {
                    const u32 m = (l + r) >> 1;
                    if (C[m] >= mid) r = m; else l = m + 1;
                }
                if (l > lo + 1 && C[l] > mid && mid - C[l - 1] < C[l] - mid) l--;
                if (l - lo > half) l = lo + half;
                if (hi - l > half) l = hi - half;
                code <<= 1;
                if (idx < l) hi = l; else { lo = l; code |= 1; }
                len++;
            }
            if (len == 0) len = 1;  // a block of one byte value
            if (idx == 0) { len0 = len; a.ctab[(u64)b * CODE_ROW + CODE_MIN] = x; }
        } else {
            len = 1;  // not in the block; any length keeps the readers' loops finite
        }
        a.ctab[(u64)b * CODE_ROW + x] = code << (32 - len) | len;
        __syncthreads();
        if (x == 0) a.ctab[(u64)b * CODE_ROW + CODE_PAD] = len0;
        __syncthreads();
    }
}

// The keys of all suffixes in text order: each thread encodes 16 consecutive positions from right to left (the key at
// a position is its codeword followed by the key of the next position, so after the first, encoded from the text
// behind the run, each costs a table look-up and G funnel shifts; the codeword ends are carried the same way and
// counted). Counts every key byte of its block (the digit histograms of all passes). CTA c takes a contiguous run of
// sort tiles and adds its shared histograms into the block's rows when the run leaves it.
struct KeySmem {
    static constexpr int G = 2;  // key groups
    u32 hist[4 * G][256];
    u32 key[G][LSD_TILE + LSD_TILE / 16];  // padded: a thread's 16 keys are consecutive
    u32 whole[LSD_TILE / 4];
    u32 tab[CODE_ROW];
};
__global__ void __launch_bounds__(TPB) k_lsd_keys(FwdArgs a) {
    __shared__ KeySmem S;
    constexpr int G = KeySmem::G;
    static_assert(LSD_IPT == 16, "a thread encodes 16 consecutive positions");
    const u32 nt = a.ctl->lsd_tiles;
    const u32 per = (nt + gridDim.x - 1) / gridDim.x;
    const u32 t0 = blockIdx.x * per, t1 = min(nt, t0 + per);
    if (t0 >= t1) return;
    const u32 tid = threadIdx.x, lane = lane_id();
    for (u32 i = tid; i < 4 * G * 256; i += TPB) (&S.hist[0][0])[i] = 0;
    u32 cur = ~0u;  // block whose counts hist holds
    auto flush = [&]() {
        for (u32 i = tid; i < 4 * G * 256; i += TPB) {
            const u32 v = (&S.hist[0][0])[i];
            if (v) {
                atomicAdd(&a.lbase[((u64)cur * NSLOT + (15 - (i >> 8))) * 256 + (i & 255)], v);
                (&S.hist[0][0])[i] = 0;
            }
        }
    };
    for (u32 t = t0; t < t1; t++) {
        const LsdTile tl = lsd_tile(a, t);
        __syncthreads();
        if (tl.b != cur) {
            if (cur != ~0u) flush();
            cur = tl.b;
            for (u32 i = tid; i < CODE_ROW; i += TPB) S.tab[i] = a.ctab[(u64)tl.b * CODE_ROW + i];
            __syncthreads();
        }
        const BlockInfo bi = a.blk[tl.b];
        const u64 end = (u64)bi.off + bi.n;
        const u32 x0 = tid * 16;
        const u64 q0 = (u64)bi.off + (tl.base - bi.soff) + x0;
        u32 k[G], m[G], wh[4] = {0, 0, 0, 0};
#pragma unroll
        for (int g = 0; g < G; g++) k[g] = m[g] = 0;
        Text16 w = {};
        if (x0 < tl.cnt) {  // (the run's first position lies in the block)
            w = text16(a.T, q0, end);
            lsd_encode<G>(a.T, S.tab, q0 + 16, end, k, m);
        }
#pragma unroll
        for (int j = 15; j >= 0; j--) {
            const u32 x = x0 + j;
            const bool ok = x < tl.cnt;
            // (symbols past the end of the block: the run's keys start from the end's zeros and its pad codewords)
            if (ok) {
                const u32 e = S.tab[(u32)((j < 8 ? w.w : w.w2) >> (8 * (j & 7))) & 0xFFu];
                u32 d = 0;
#pragma unroll
                for (int g = G - 1; g > 0; g--) {
                    k[g] = __funnelshift_r(k[g], k[g - 1], e);  // (count modulo 32)
                    m[g] = __funnelshift_r(m[g], m[g - 1], e);
                }
                k[0] = __funnelshift_r(k[0], 0u, e) | (e & CODE_BITS);
                m[0] = __funnelshift_r(m[0], 0u, e) | 1u << (32 - (e & 31u));
#pragma unroll
                for (int g = 0; g < G; g++) {
                    S.key[g][x + (x >> 4)] = k[g];
                    d += __popc(m[g]);
                }
                wh[j >> 2] |= d << (8 * (j & 3));  // at most 32 G <= 128
            }
#pragma unroll
            for (int g = 0; g < G; g++) {
                // runs of one key (padding, repeated records) would serialise 32 atomics on one counter
                const u32 lead = __shfl_sync(0xffffffffu, k[g], 0);
                const bool same = __all_sync(0xffffffffu, ok && k[g] == lead);
                if (same ? lane == 0 : ok) {
                    const u32 add = same ? 32u : 1u;
#pragma unroll
                    for (int b = 0; b < 4; b++) atomicAdd(&S.hist[4 * g + b][(k[g] >> (24 - 8 * b)) & 0xFFu], add);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) S.whole[tid * 4 + i] = wh[i];
        __syncthreads();
#pragma unroll
        for (int g = 0; g < G; g++) {
            u32 *out = lsd_keys_of(a, g) + tl.base;
            for (u32 x = tid; x < tl.cnt; x += TPB) out[x] = S.key[g][x + (x >> 4)];
        }
        u8 *out = lsd_whole_of(a) + tl.base;
        for (u32 x = tid; x < tl.cnt; x += TPB) out[x] = reinterpret_cast<const u8 *>(S.whole)[x];
    }
    __syncthreads();
    flush();
}

// Coded keys: digit bases of every pass and the active slots (CTAs over blocks, one warp per slot, eight digits per lane): the
// exclusive scan of a block's digit counts plus the block's soff is the pass's first position of every digit (lbase
// row (block, slot), in place of the counts). A slot runs when its key byte takes two or more values within some
// block (slots 16 - W..15 only).
__global__ void __launch_bounds__(TPB) k_lsd_base(FwdArgs a) {
    const int first = 16 - (int)a.lsd_bytes;
    for (u32 b = blockIdx.x; b < a.B; b += gridDim.x) {
        const u32 n = a.blk[b].n, soff = a.blk[b].soff;
        for (int slot = first + (int)warp_id(); slot < NSLOT; slot += TPB / 32) {
            uint4 *row = reinterpret_cast<uint4 *>(a.lbase + ((u64)b * NSLOT + slot) * 256) + 2 * lane_id();
            const uint4 u = row[0], v = row[1];
            const u32 d[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
            u32 sum = 0;
            bool vary = false;
#pragma unroll
            for (int i = 0; i < 8; i++) { sum += d[i]; vary = vary || (d[i] != 0 && d[i] != n); }
            u32 run = soff + warp_incl_sum(sum) - sum;
            u32 o[8];
#pragma unroll
            for (int i = 0; i < 8; i++) { o[i] = run; run += d[i]; }
            row[0] = make_uint4(o[0], o[1], o[2], o[3]);
            row[1] = make_uint4(o[4], o[5], o[6], o[7]);
            if (__any_sync(0xffffffffu, vary) && lane_id() == 0 && !((a.ctl->lsd_act >> slot) & 1))
                atomicOr(&a.ctl->lsd_act, 1u << slot);
        }
    }
}

// Raw keys: digit bases of every pass and the active slots (256 threads per CTA, thread = digit value, CTAs over blocks).
// Suffix i of a block of n bytes has key byte d = T[i + d] when i + d < n, else 0, so the counts of key byte d are
// the block's byte counts minus those of its first min(d, n) bytes, plus min(d, n) zeros; their exclusive scan plus
// the block's soff gives the pass's first position of every digit (lbase row (block, slot), slot = 15 - d). A slot
// runs when its key byte takes two or more values within some block (slots 16 - W..15 only).
__global__ void __launch_bounds__(TPB) k_lsd_hist0(FwdArgs a) {
    __shared__ u32 wm[8];
    __shared__ u32 ws[TPB / 32 + 1];
    const u32 x = threadIdx.x;
    const int first = 16 - (int)a.lsd_bytes;
    for (u32 b = blockIdx.x; b < a.B; b += gridDim.x) {
        const BlockInfo bi = a.blk[b];
        const u32 h = a.lhist[(u64)b * 256 + x];
        u32 pre = 0, mask = 0;  // pre: bytes x among the block's first d bytes
        for (int slot = 15; slot >= first; slot--) {
            const u32 d = 15 - slot;
            if (d >= 1 && d <= bi.n) pre += __ldg(a.T + (u64)bi.off + d - 1) == x;
            const u32 v = h - pre + (x == 0 ? min(d, bi.n) : 0u);
            if (v != 0 && v != bi.n) mask |= 1u << slot;
            a.lbase[((u64)b * NSLOT + slot) * 256 + x] = bi.soff + block_excl_sum<TPB>(v, ws, nullptr);
        }
        for (int o = 16; o; o >>= 1) mask |= __shfl_xor_sync(0xffffffffu, mask, o);
        if ((x & 31) == 0) wm[x >> 5] = mask;
        __syncthreads();
        if (x == 0) {
            u32 m = 0;
            for (int w = 0; w < 8; w++) m |= wm[w];
            if (m & ~a.ctl->lsd_act) atomicOr(&a.ctl->lsd_act, m);
        }
        __syncthreads();
    }
}

constexpr int RANK_Q = 4;  // elements a lane ranks at once
struct LsdSmem {
    unsigned long long item[LSD_TILE];
    __align__(16) u32 wcnt[TPB / 32][256];
    u32 gbase[256];
    u32 ws[TPB / 32 + 1];
    u32 tile;
};

// One sort tile of an LSD pass over digit `slot`: rank the tile's suffixes by digit, publish the tile's digit counts,
// look back over the block's earlier tiles for the offsets (bounded spin), stage the tile in shared memory in digit
// order and write it out in runs. FULL: the tile holds LSD_TILE suffixes (every tile but a block's last), so no
// element needs a bounds check.
template <bool CODED, bool FULL>
__device__ __forceinline__ void lsd_pass_tile(const FwdArgs &a, LsdSmem &S, int slot, u32 act, u64 epoch, u32 tile,
                                              const LsdTile &tl) {
    const u32 lower = act & ((1u << slot) - 1), higher = act & ~((2u << slot) - 1);
    const u32 par = __popc(lower) & 1;
    const u32 tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const u32 base = tl.base, cnt = FULL ? (u32)LSD_TILE : tl.cnt;
    const bool head = tile == __ldg(&a.blk[tl.b].lt0);  // the block's first tile: its counts are the inclusive prefix
    // this pass's first position of digit tid in the block
    const u32 dbase = __ldg(a.lbase + ((u64)tl.b * NSLOT + slot) * 256 + tid);
    const unsigned long long *iin = a.lit[par];
    // rr: each item's rank in its warp's digit bucket (< 512), two 16-bit ranks per register; the digit itself is
    // recomputed from the key where it is needed
    u32 v[LSD_IPT], rr[LSD_IPT / 2], k[LSD_IPT];
    const u32 dsh = 8 * (slot & 3);  // byte 15 - slot of the prefix within the key group
    u32 *mask = reinterpret_cast<u32 *>(S.item) + warp * 256 * RANK_Q;  // (zeroed; the staging follows the ranking)
    if (!lower) {
        // the first pass: the suffixes are still in text order, as k_lsd_keys wrote their keys
        const BlockInfo bi = a.blk[tl.b];
        const u32 id0 = bi.off + (base - bi.soff), g = lsd_slot_group(slot);
        const u64 end = (u64)bi.off + bi.n;
        const u32 *keys = CODED ? lsd_keys_of(a, g) : nullptr;
#pragma unroll
        for (int j = 0; j < LSD_IPT; j++) {
            const u32 x = warp * (32 * LSD_IPT) + j * 32 + lane;
            v[j] = id0 + x;
            k[j] = !(FULL || x < cnt) ? 0u : CODED ? __ldcs(keys + base + x) : lsd_raw_group(a.T, id0 + x, g, end);
        }
    } else {
#pragma unroll
        for (int j = 0; j < LSD_IPT; j++) {
            const u32 x = warp * (32 * LSD_IPT) + j * 32 + lane;
            const bool ok = FULL || x < cnt;
            const unsigned long long it = ok ? __ldcs(iin + base + x) : 0ull;
            v[j] = (u32)it;
            k[j] = (u32)(it >> 32);
        }
    }
    // Coded keys spread over the digit values; raw text, sorted by what follows, has few distinct bytes in a warp, and
    // __match_any_sync takes two cycles a distinct value (64 MiB of prose, 16 passes: 7.24 ms with it, 7.34 with
    // warp_rank; 216 MB of mixed blocks, 8 passes over coded keys: 14.4 and 11.7).
    if (CODED) {
#pragma unroll
        for (int j0 = 0; j0 < LSD_IPT; j0 += RANK_Q) {
            u32 d[RANK_Q], r[RANK_Q];
#pragma unroll
            for (int q = 0; q < RANK_Q; q++) {
                const u32 x = warp * (32 * LSD_IPT) + (j0 + q) * 32 + lane;
                d[q] = (FULL || x < cnt) ? (k[j0 + q] >> dsh) & 0xFFu : 0x100u;  // 0x100: past the tile's end
            }
            warp_rank<RANK_Q, !FULL>(mask, S.wcnt[warp], d, r);
#pragma unroll
            for (int q = 0; q < RANK_Q; q += 2) rr[(j0 + q) >> 1] = r[q] | r[q + 1] << 16;
        }
    } else {
#pragma unroll
        for (int j = 0; j < LSD_IPT; j++) {
            const u32 x = warp * (32 * LSD_IPT) + j * 32 + lane;
            const u32 d = (FULL || x < cnt) ? (k[j] >> dsh) & 0xFFu : 0x100u;  // 0x100: past the tile's end
            const u32 peers = __match_any_sync(0xffffffffu, d);
            const u32 before = (FULL || d < 256) ? S.wcnt[warp][d] : 0u;
            const u32 r = before + __popc(peers & lanemask_lt());
            if (j & 1) rr[j >> 1] |= r << 16; else rr[j >> 1] = r;
            __syncwarp();
            if ((FULL || d < 256) && (__ffs(peers) - 1) == (int)lane) S.wcnt[warp][d] = before + __popc(peers);
            __syncwarp();
        }
    }
    __syncthreads();
    // thread tid owns digit tid: tile count, publish, local start, look back
    u32 tot = 0;
#pragma unroll
    for (int w = 0; w < TPB / 32; w++) tot += S.wcnt[w][tid];
    u64 *st = a.lstat + (u64)tile * 256 + tid;
    if (head) atomicExch((unsigned long long *)st, epoch | ST_PRE | tot);
    else atomicExch((unsigned long long *)st, epoch | ST_AGG | tot);
    const u32 dstart = block_excl_sum<TPB>(tot, S.ws, nullptr);
    {
        u32 run = dstart;
#pragma unroll
        for (int w = 0; w < TPB / 32; w++) { const u32 cc = S.wcnt[w][tid]; S.wcnt[w][tid] = run; run += cc; }
    }
    __syncthreads();
    // stage in digit order (tile-local offsets only: the items leave registers before the look-back)
#pragma unroll
    for (int j = 0; j < LSD_IPT; j++) {
        const u32 x = warp * (32 * LSD_IPT) + j * 32 + lane;
        if (FULL || x < cnt) {
            const u32 d = (k[j] >> dsh) & 0xFFu;
            const u32 p = S.wcnt[warp][d] + ((rr[j >> 1] >> (16 * (j & 1))) & 0xFFFFu);
            S.item[p] = (unsigned long long)k[j] << 32 | v[j];
        }
    }
    u32 excl = 0;
    if (!head) {
        // windowed look-back: read LB_WIN predecessors' words at once, add aggregates in order up to the first
        // inclusive prefix (at the latest the block's first tile); a word not yet published ends the window and the
        // walk resumes there
        long j = (long)tile - 1;
        u32 spins = 0;
        while (true) {
            u64 w[LB_WIN];
#pragma unroll
            for (int q = 0; q < LB_WIN; q++)
                w[q] = j - q >= 0 ? *(volatile u64 *)(a.lstat + (u64)(j - q) * 256 + tid) : 0ull;
            int used = 0;
            bool done = false;
#pragma unroll
            for (int q = 0; q < LB_WIN; q++) {
                if (done || used < q) continue;  // stopped earlier in the window
                const u64 x = w[q];
                if ((x & ST_EPOCH) != epoch || !(x & (ST_AGG | ST_PRE))) continue;
                excl += (u32)(x & ST_VAL);
                used = q + 1;
                if (x & ST_PRE) done = true;
            }
            if (done) break;
            j -= used;
            if (used == 0) {
                if (++spins > a.spin_limit) {  // a predecessor never published: report and stop waiting
                    atomicOr(&a.ctl->err, 256u);
                    break;
                }
                __nanosleep(32);
            }
        }
        atomicExch((unsigned long long *)st, epoch | ST_PRE | (u64)(excl + tot));
    }
    S.gbase[tid] = dbase + excl - dstart;
    const u32 g = lsd_slot_group(slot);
    // the key the next pass reads: this group's (carried), the next group's (gathered) or none
    const int gn = higher ? (int)lsd_slot_group(__ffs(higher) - 1) : -1;
    __syncthreads();
    unsigned long long *iout = a.lit[par ^ 1];
    const BlockInfo bi = a.blk[tl.b];
    const u32 bend = bi.soff + bi.n;  // bound of the checked build's write checks
    (void)bend;
    if (gn == (int)g) {
        for (u32 i = tid; i < cnt; i += TPB) {
            const unsigned long long it = S.item[i];
            const u32 dst = S.gbase[((u32)(it >> 32) >> dsh) & 0xFFu] + i;
            if (KGB_OK(dst < bend, &a.ctl->err, E_LIST)) __stcs(iout + dst, it);
        }
    } else if (gn >= 0) {
        const u64 end = (u64)bi.off + bi.n;
        const u32 *keys = CODED ? lsd_keys_of(a, (u32)gn) : nullptr;
        const u32 dense = bi.soff - bi.off;  // (modulo 2^32: a batch with gaps has off > soff)
        constexpr int WB = CODED ? 8 : 4;  // gathers in flight per thread
        for (u32 i0 = tid; i0 < cnt; i0 += WB * TPB) {
            u32 id[WB], dst[WB], kk[WB];
#pragma unroll
            for (int q = 0; q < WB; q++) {
                const u32 i = i0 + q * TPB;
                const bool ok = FULL || i < cnt;
                const unsigned long long it = ok ? S.item[i] : 0ull;
                id[q] = (u32)it;
                dst[q] = ok ? S.gbase[((u32)(it >> 32) >> dsh) & 0xFFu] + i : 0u;
                kk[q] = !ok ? 0u : CODED ? __ldg(keys + (u32)(dense + id[q])) : lsd_raw_group(a.T, id[q], (u32)gn, end);
            }
#pragma unroll
            for (int q = 0; q < WB; q++) {
                if ((FULL || i0 + q * TPB < cnt) && KGB_OK(dst[q] < bend, &a.ctl->err, E_LIST)) {
                    __stcs(iout + dst[q], (unsigned long long)kk[q] << 32 | id[q]);
                }
            }
        }
    } else {  // the last pass: the segmentation reads ids only
        u32 *vout = a.lval[par ^ 1];
        for (u32 i = tid; i < cnt; i += TPB) {
            const unsigned long long it = S.item[i];
            const u32 dst = S.gbase[((u32)(it >> 32) >> dsh) & 0xFFu] + i;
            if (KGB_OK(dst < bend, &a.ctl->err, E_LIST)) __stcs(vout + dst, (u32)it);
        }
    }
}

// One LSD pass over digit `slot` (skipped when that key byte is constant within every block): each CTA takes the
// next sort tile in order.
template <bool CODED>
__global__ void __launch_bounds__(TPB, 3) k_lsd_pass(FwdArgs a, int slot) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LsdSmem &S = *reinterpret_cast<LsdSmem *>(smem_raw);
    const Ctl *c = a.ctl;
    const u32 act = active_slots(c);
    const u32 ntiles = c->lsd_tiles;
    if (!((act >> slot) & 1)) {
        // no key byte varies within any block: the sorted order is the text order, written by the first slot's launch
        if (act == 0 && slot == 16 - (int)a.lsd_bytes && blockIdx.x < ntiles) {
            const LsdTile tl = lsd_tile(a, blockIdx.x);
            const u32 id0 = a.blk[tl.b].off + (tl.base - a.blk[tl.b].soff);
            for (u32 j = threadIdx.x; j < tl.cnt; j += TPB) __stcs(a.lval[0] + tl.base + j, id0 + j);
        }
        return;
    }
    const u64 epoch = (u64)((c->seq << 5) | (u32)slot) << 32;
    const u32 tid = threadIdx.x;
    if (tid == 0) S.tile = atomicAdd(&a.ltile[slot], 1u);
    {  // the ranking's counters and digit masks (the masks borrow the staging area)
        static_assert(sizeof(S.item) == (TPB / 32) * 256 * RANK_Q * 4 && sizeof(S.wcnt) % (16 * TPB) == 0, "");
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (u32 i = tid; i < sizeof(S.wcnt) / 16; i += TPB) reinterpret_cast<uint4 *>(&S.wcnt[0][0])[i] = z;
        for (u32 i = tid; CODED && i < sizeof(S.item) / 16; i += TPB) reinterpret_cast<uint4 *>(S.item)[i] = z;
    }
    __syncthreads();
    const u32 tile = S.tile;
    if (tile >= ntiles) return;
    const LsdTile tl = lsd_tile(a, tile);
    if (tl.cnt == (u32)LSD_TILE) lsd_pass_tile<CODED, true>(a, S, slot, act, epoch, tile, tl);
    else lsd_pass_tile<CODED, false>(a, S, slot, act, epoch, tile, tl);
}

// ---- segmentation of the sorted keys
// Positions are handled in tiles of SEG_TILE; warp w of a tile owns the SEG_IPT * 32 consecutive positions starting at
// tile base + w * 32 * SEG_IPT and visits them lane-striped (position = chunk base + j * 32 + lane), so every load is
// coalesced. Group starts are kept as a bitmask (bit p of the mask: a group starts at position p), written by the
// count kernel (which compares neighbouring sorted keys); the emit kernels read only the bits.
__device__ __forceinline__ u32 lsd_final_par(const Ctl *c) { return __popc(active_slots(c)) & 1; }

struct SegBufs {
    const u32 *val;
    u32 *bits;          // start bitmask
    u8 *dep;            // per position: the bytes its key holds whole (in a list that is empty in round 0)
    u32 *gbase, *gidx;  // per group start: list slot base, list index | GRP_LARGE (free value buffers)
    u32 *rk;            // per position: the round-0 rank, for the rank passes (the free half of the ids' item buffer)
    u32 m;
};
__device__ __forceinline__ SegBufs seg_bufs(const FwdArgs &a) {
    const Ctl *c = a.ctl;
    const u32 par = lsd_final_par(c);
    SegBufs v;
    v.val = a.lval[par];
    v.bits = a.segbits;
    v.dep = reinterpret_cast<u8 *>(a.lists[L_S0].eid);
    v.gbase = a.lval[par ^ 1];
    v.gidx = a.lhi[par ^ 1];  // lval[q] and lhi[q] are the two halves of item buffer q
    v.rk = a.lhi[par];
    v.m = c->m;
    return v;
}
constexpr u32 GRP_LARGE = 0x80000000u, GRP_TINY = 0x40000000u, GRP_MED = 0x20000000u;
constexpr u32 SEG_WORDS = SEG_IPT;  // mask words per warp chunk

// The blocks a warp's chunk of SEG_IPT * 32 positions from cb spans: [lo, hi] (the same for every lane).
__device__ __forceinline__ uint2 seg_chunk_blocks(const FwdArgs &a, u32 cb, u32 m) {
    const u32 lo = blk_of_pos(a, cb, 0, a.B - 1);
    const u32 hi = blk_of_pos(a, min(cb + SEG_IPT * 32, m) - 1, lo, a.B - 1);
    return make_uint2(lo, hi);
}

// Per tile: start bits and the tile's last group start. A position starts a group when it is its block's first or when
// its suffix and the one before it differ in the bytes their keys hold whole (in their number, or in one of them): the
// bits of a last codeword that the key cuts off do not count, so that a group has those bytes in common, and comparing
// the text (which the L column's bytes are taken from here as well, coalesced) costs less than encoding it again.
// Also per position the number of those bytes (at most DEPTH_MAX), and their minimum over the suffixes that start no
// group (every group of two or more has one).
template <bool CODED>
__global__ void __launch_bounds__(TPB, 3) k_seg_count(FwdArgs a) {
    __shared__ u32 ws[TPB / 32];
    const SegBufs v = seg_bufs(a);
    const u8 *whole = lsd_whole_of(a);
    const u32 ntiles = (v.m + SEG_TILE - 1) / SEG_TILE;
    const u32 lane = lane_id(), warp = warp_id();
    u32 depth = 0xFFFFFFFFu;
    for (u32 t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const u32 cb = t * SEG_TILE + warp * 32 * SEG_IPT;
        const uint2 br = cb < v.m ? seg_chunk_blocks(a, cb, v.m) : make_uint2(0u, 0u);
        const BlockInfo bi0 = a.blk[br.x];
        const u32 min0 = CODED ? a.ctab[(u64)br.x * CODE_ROW + CODE_MIN] : 0u;
        // the suffix at the position before the step's first one (its block's: used where that position has the same)
        u32 pid = cb > bi0.soff && cb < v.m ? v.val[cb - 1] : bi0.off, pd;
        u64 pw, pw2;
        {
            const Text16 x = text16_padded(a.T, pid, (u64)bi0.off + bi0.n, min0);
            pd = CODED ? whole[bi0.soff + (pid - bi0.off)] : a.lsd_bytes;
            pw = x.w;
            pw2 = x.w2;
        }
        u32 last = 0;
        constexpr int QB = 4;  // positions whose ids, text and counts are loaded at once
#pragma unroll 1
        for (int j0 = 0; j0 < SEG_IPT; j0 += QB) {
            u32 id[QB], d[QB], b[QB];
            Text16 tx[QB];
#pragma unroll
            for (int q = 0; q < QB; q++) {
                const u32 p = cb + (j0 + q) * 32 + lane;
                b[q] = p < v.m && br.x != br.y ? blk_of_pos(a, p, br.x, br.y) : br.x;
                id[q] = p < v.m ? __ldcs(v.val + p) : bi0.off;
            }
#pragma unroll
            for (int q = 0; q < QB; q++) {
                BlockInfo bi = bi0;
                u32 mn = min0;
                if (br.x != br.y) { bi = a.blk[b[q]]; mn = CODED ? a.ctab[(u64)b[q] * CODE_ROW + CODE_MIN] : 0u; }
                tx[q] = text16_padded(a.T, id[q], (u64)bi.off + bi.n, mn);
                d[q] = CODED ? whole[bi.soff + (id[q] - bi.off)] : a.lsd_bytes;
            }
#pragma unroll
            for (int q = 0; q < QB; q++) {
                const u32 p = cb + (j0 + q) * 32 + lane;
                const bool ok = p < v.m;
                BlockInfo bi = bi0;
                if (br.x != br.y) bi = a.blk[b[q]];
                const u64 end = (u64)bi.off + bi.n;
                // the neighbour's text, count and id: the lane below's, for lane 0 the last lane's of the step before
                const u32 below = (lane + 31) & 31;
                u64 nw = __shfl_sync(0xffffffffu, tx[q].w, below), nw2 = __shfl_sync(0xffffffffu, tx[q].w2, below);
                u32 nd = d[q], nid = __shfl_sync(0xffffffffu, id[q], below);
                if (CODED) nd = __shfl_sync(0xffffffffu, d[q], below);
                if (lane == 0) {
                    const u64 cw = nw, cw2 = nw2;
                    const u32 cd = nd, cid = nid;
                    nw = pw; nw2 = pw2; nd = pd; nid = pid;
                    pw = cw; pw2 = cw2; pd = cd; pid = cid;
                }
                const u32 D = d[q];  // at least 5: CODE_MAX-bit codewords in 64 bits
                bool eq = ok && p != bi.soff && nd == D;
                const u64 x = tx[q].w ^ nw, x2 = tx[q].w2 ^ nw2;
                eq = eq && (D >= 8 ? x == 0 : x << (8 * (8 - D)) == 0);
                eq = eq && (D <= 8 || (D >= 16 ? x2 == 0 : x2 << (8 * (16 - D)) == 0));
                // short codewords: the bytes past the first 16
                for (u32 o = 16; CODED && __any_sync(0xffffffffu, eq && D > o); o += 16) {
                    if (eq && D > o) {
                        const u32 mn = a.ctab[(u64)b[q] * CODE_ROW + CODE_MIN];
                        const Text16 y = text16_padded(a.T, (u64)id[q] + o, end, mn);
                        const Text16 z = text16_padded(a.T, (u64)nid + o, end, mn);
                        const u64 u = y.w ^ z.w, u2 = y.w2 ^ z.w2;
                        const u32 r = D - o;
                        eq = r >= 8 ? u == 0 : u << (8 * (8 - r)) == 0;
                        eq = eq && (r <= 8 || (r >= 16 ? u2 == 0 : u2 << (8 * (16 - r)) == 0));
                    }
                }
                const bool st = ok && !eq;
                const u32 sb = __ballot_sync(0xffffffffu, st);
                if (lane == 0 && ok) v.bits[(cb >> 5) + j0 + q] = sb;
                if (ok) {
                    if (CODED) v.dep[p] = (u8)min(D, DEPTH_MAX);
                    // the L column of the sorted order so far: final for groups of one, overwritten for the others
                    const u8 c = id[q] == bi.off ? (u8)0 : tx[q].has_before ? tx[q].before : __ldg(a.T + id[q] - 1);
                    KGB_GUARD(p >= bi.soff && p - bi.soff < bi.n, &a.ctl->err, E_RANK)
                    __stcs(a.L + (u64)bi.off + b[q] + (p - bi.soff) + 1, c);
                }
                if (st) last = p;
                if (CODED && eq) depth = min(depth, D);
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
        if (lane == 0) ws[warp] = last;
        __syncthreads();
        if (threadIdx.x == 0) {
            u32 tl = 0;
            for (int w = 0; w < TPB / 32; w++) tl = max(tl, ws[w]);
            a.segagg[(u64)t * 2] = tl;
        }
        __syncthreads();
    }
    if (!CODED) return;
    depth = __reduce_min_sync(0xffffffffu, depth);
    if (lane == 0 && depth != 0xFFFFFFFFu && depth < *(volatile u32 *)&a.ctl->h0) atomicMin(&a.ctl->h0, depth);
}

// Exclusive max-scan of the tiles' last starts (one CTA): the start of the group open at each tile's first position.
__global__ void __launch_bounds__(1024) k_seg_scan(FwdArgs a) {
    __shared__ u32 ws[33];
    __shared__ u32 prev[1024];
    const u32 m = a.ctl->m;
    const u32 ntiles = (m + SEG_TILE - 1) / SEG_TILE;
    u32 carry = 0;
    for (u32 t0 = 0; t0 < ntiles; t0 += 1024) {
        const u32 t = t0 + threadIdx.x;
        const u32 l = t < ntiles ? a.segagg[(u64)t * 2] : 0u;
        const u32 il = block_incl_max<1024>(l, ws);
        prev[threadIdx.x] = il;
        __syncthreads();
        if (t < ntiles) a.segagg[(u64)t * 2 + 1] = max(carry, threadIdx.x ? prev[threadIdx.x - 1] : 0u);
        carry = max(carry, prev[1023]);
        __syncthreads();
    }
}

// The warp's view of its chunk: the mask words (lane j holds word j), and the start of the group open at the chunk's
// first position.
struct SegChunk {
    u32 cb, word, nextw, carry0;
    u32 blo, bhi;  // the blocks the chunk spans
};
__device__ __forceinline__ SegChunk seg_chunk(const FwdArgs &a, const SegBufs &v, u32 t, u32 *wl) {
    const u32 lane = lane_id(), warp = warp_id();
    SegChunk c;
    c.cb = t * SEG_TILE + warp * 32 * SEG_IPT;
    const u32 w0 = c.cb >> 5;
    const u32 nw = (v.m + 31) >> 5;
    c.word = lane < SEG_WORDS && w0 + lane < nw ? v.bits[w0 + lane] : 0u;
    // bit 0 of the word after the chunk: the start flag of the first position past it
    c.nextw = w0 + SEG_WORDS < nw ? v.bits[w0 + SEG_WORDS] : 1u;
    u32 last = 0;
    if (lane < SEG_WORDS && c.word) last = c.cb + lane * 32 + 31 - __clz(c.word);
#pragma unroll
    for (int o = 16; o; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    if (lane == 0) wl[warp] = last;
    __syncthreads();
    u32 cr = a.segagg[(u64)t * 2 + 1];
    for (u32 w = 0; w < warp; w++) cr = max(cr, wl[w]);
    c.carry0 = cr;
    const uint2 br = c.cb < v.m ? seg_chunk_blocks(a, c.cb, v.m) : make_uint2(0u, 0u);
    c.blo = br.x; c.bhi = br.y;
    return c;
}
// Position j * 32 + lane of the chunk: start / end flags and the group's first position (carry: running start).
__device__ __forceinline__ void seg_step(const SegBufs &v, const SegChunk &c, int j, u32 &carry, u32 &p, bool &valid,
                                         bool &st, bool &en, u32 &gfirst) {
    const u32 lane = lane_id();
    const u32 w = __shfl_sync(0xffffffffu, c.word, j);
    const u32 wn = j + 1 < SEG_IPT ? __shfl_sync(0xffffffffu, c.word, (j + 1) & 31) : c.nextw;
    p = c.cb + j * 32 + lane;
    valid = p < v.m;
    st = (w >> lane) & 1;
    en = p + 1 >= v.m || (lane < 31 ? (w >> (lane + 1)) & 1 : wn & 1);
    const u32 x = warp_incl_max(valid && st ? p : 0u);
    gfirst = max(carry, x);
    carry = __shfl_sync(0xffffffffu, gfirst, 31);
}

// Block-wide exclusive sum of a 64-bit value (TPB threads); contains __syncthreads().
__device__ __forceinline__ u64 block_excl_sum64(u64 v, u64 *ws, u64 *total) {
    u64 inc = v;
    const u32 lane = lane_id(), warp = warp_id();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (u32)o) inc += t;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    u64 before = 0, tot = 0;
    for (u32 w = 0; w < TPB / 32; w++) {
        const u64 x = ws[w];
        if (w < warp) before += x;
        tot += x;
    }
    __syncthreads();
    *total = tot;
    return before + inc - v;
}

// Emit, part 1 (group ends): groups of one resolve (rank unless k_seg_rank writes the ranks); every other group takes
// its slots in the next tiny-group list (<= GTINY), medium-group list (<= GMED), small-group list (<= SMAX) or
// large-group list, writes its descriptor (and tile-map entries), and records its slot base and index at its first
// position for part 2. Slots are allocated once per tile (a count pass, a block scan, one atomic per list).
__global__ void __launch_bounds__(TPB) k_seg_emit1(FwdArgs a) {
    __shared__ u32 wl[TPB / 32];
    __shared__ u64 ws[4][TPB / 32];
    __shared__ u64 base[5];
    Ctl *c = a.ctl;
    const SegBufs v = seg_bufs(a);
    const u32 rpar = c->rpar, round = c->round;
    const ListView sl = a.lists[L_S0 + (rpar ^ 1)], ll = a.lists[L_L0 + (rpar ^ 1)], tl_ = a.lists[L_P0 + (rpar ^ 1)];
    const ListView ml_ = a.lists[L_M0 + (rpar ^ 1)];
    const u32 ntiles = (v.m + SEG_TILE - 1) / SEG_TILE;
    const u32 TS = a.smax;
    for (u32 t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const SegChunk ch = seg_chunk(a, v, t, wl);
        // count: singles | small groups << 16 | small elements << 32 ; large groups | large elements << 32 ;
        // tiny groups | tiny elements << 32 ; medium groups | medium elements << 32
        u64 cs = 0, cl = 0, ct = 0, cm = 0;
        {
            u32 carry = ch.carry0;
            for (int j = 0; j < SEG_IPT; j++) {
                u32 p, gf; bool ok, st, en;
                seg_step(v, ch, j, carry, p, ok, st, en, gf);
                if (!ok || !en) continue;
                const u32 len = p - gf + 1;
                if (len == 1) cs += 1;
                else if (len <= GTINY) ct += 1ull | ((u64)len << 32);
                else if (len <= GMED) cm += 1ull | ((u64)len << 32);
                else if (len <= TS) cs += (1ull << 16) | ((u64)len << 32);
                else cl += 1ull | ((u64)len << 32);
            }
        }
        u64 ts, tl, tt;
        u64 xs = block_excl_sum64(cs, ws[0], &ts);
        u64 xl = block_excl_sum64(cl, ws[1], &tl);
        u64 xt = block_excl_sum64(ct, ws[2], &tt);
        u64 tm;
        u64 xm = block_excl_sum64(cm, ws[3], &tm);
        if (threadIdx.x == 0) {
            base[4] = (u32)tm ? atomicAdd(&c->cnt[L_M0 + (rpar ^ 1)], (tm << 32) | (tm >> 32)) : 0ull;
            if ((u32)tt) {
                const uint2 o = alloc_tiny(c, rpar, (u32)tt, (u32)(tt >> 32));
                base[3] = ((u64)o.y << 32) | o.x;
            } else {
                base[3] = 0;
            }
            base[1] = (ts >> 16) & 0xFFFF ? atomicAdd(&c->cnt[L_S0 + (rpar ^ 1)], (((ts >> 16) & 0xFFFF) << 32) | (ts >> 32)) : 0ull;
            base[2] = (u32)tl ? atomicAdd(&c->cnt[L_L0 + (rpar ^ 1)], (tl << 32) | (tl >> 32)) : 0ull;
        }
        __syncthreads();
        u32 sidx = (u32)(base[1] >> 32) + (u32)((xs >> 16) & 0xFFFF), se = (u32)base[1] + (u32)(xs >> 32);
        u32 lidx = (u32)(base[2] >> 32) + (u32)xl, le = (u32)base[2] + (u32)(xl >> 32);
        u32 tidx = (u32)(base[3] >> 32) + (u32)xt, te = (u32)base[3] + (u32)(xt >> 32);
        u32 midx = (u32)(base[4] >> 32) + (u32)xm, me = (u32)base[4] + (u32)(xm >> 32);
        u32 carry = ch.carry0;
        constexpr int QB = 8;  // positions per phase: group ends first, then their loads, then the writes
        for (int j0 = 0; j0 < SEG_IPT; j0 += QB) {
            u32 pv[QB], gfv[QB], live = 0;
#pragma unroll
            for (int q = 0; q < QB; q++) {
                u32 p, gf; bool ok, st, en;
                seg_step(v, ch, j0 + q, carry, p, ok, st, en, gf);
                pv[q] = p; gfv[q] = gf;
                if (ok && en) live |= 1u << q;
            }
            u32 bv[QB], idv[QB];  // idv: the id of a finished suffix (a group of one), else the group's shared characters
            const bool ids = !a.rank_passes || a.SA;
#pragma unroll
            for (int q = 0; q < QB; q++) {
                if (!((live >> q) & 1)) continue;
                bv[q] = ch.blo == ch.bhi ? ch.blo : blk_of_pos(a, pv[q], ch.blo, ch.bhi);
                idv[q] = pv[q] != gfv[q] ? (lsd_coded(a) ? (u32)__ldg(v.dep + pv[q]) : 0u) : ids ? __ldcs(v.val + pv[q]) : 0u;
            }
#pragma unroll
            for (int q = 0; q < QB; q++) {
                if (!((live >> q) & 1)) continue;
                const u32 p = pv[q], gf = gfv[q];
                const u32 len = p - gf + 1;
                const u32 b = bv[q];
                const u32 head = gf - a.blk[b].soff;
                if (len == 1) {
                    if (ids) resolve_round0(a, a.rank_passes ? nullptr : a.isa[rpar ^ 1], idv[q], head, b);
                    continue;
                }
                Seg g;
                g.len = len; g.head = head; g.bd = b | idv[q] << DEPTH_SHIFT;
                if (len <= GTINY) {
                    g.start = te;
                    KGB_GUARD(tidx < a.cap_segt && (u64)te + len <= a.cap_n, &c->err, E_SEG) {
                        tl_.seg[tidx] = g;
                        v.gbase[gf] = te;
                        v.gidx[gf] = tidx | GRP_TINY;
                    }
                    tidx++; te += len;
                } else if (len <= GMED) {
                    g.start = me;
                    KGB_GUARD(midx < a.cap_segm && (u64)me + len <= a.cap_n, &c->err, E_SEG) {
                        ml_.seg[midx] = g;
                        v.gbase[gf] = me;
                        v.gidx[gf] = midx | GRP_MED;
                    }
                    midx++; me += len;
                } else if (len <= TS) {
                    g.start = se;
                    KGB_GUARD(sidx < a.cap_segs && (u64)se + len <= a.cap_n, &c->err, E_SEG) {
                        sl.seg[sidx] = g;
                        write_tmap_small(a, sl.tmap, TS, se, len, sidx);
                        if (len > WARP_GROUP) sl.tbig[se / TS] = round + 1;
                        v.gbase[gf] = se;
                        v.gidx[gf] = sidx;
                    }
                    sidx++; se += len;
                } else {
                    g.start = le;
                    KGB_GUARD(lidx < a.cap_segl && (u64)le + len <= a.cap_n, &c->err, E_SEG) {
                        ll.seg[lidx] = g;
                        ll.lab[lidx] = head | LAB_BOTH;  // (round 1's fixup copies every rank to the other buffer)
                        v.gbase[gf] = le;
                        v.gidx[gf] = lidx | GRP_LARGE;
                    }
                    lidx++; le += len;
                }
            }
        }
        __syncthreads();
    }
}

// Emit, part 2 (every suffix of a group of two or more): its rank (the group's first position) unless k_seg_rank
// writes the ranks, its slot in its group's list, and for large groups the bucket-pass tile map (the suffix at a
// multiple of TSM names its group).
__global__ void __launch_bounds__(TPB) k_seg_emit2(FwdArgs a) {
    __shared__ u32 wl[TPB / 32];
    Ctl *c = a.ctl;
    const SegBufs v = seg_bufs(a);
    const u32 rpar = c->rpar;
    const ListView sl = a.lists[L_S0 + (rpar ^ 1)], ll = a.lists[L_L0 + (rpar ^ 1)], tl_ = a.lists[L_P0 + (rpar ^ 1)];
    const ListView ml_ = a.lists[L_M0 + (rpar ^ 1)];
    const u32 ntiles = (v.m + SEG_TILE - 1) / SEG_TILE;
    constexpr int QB = 8;  // positions per phase: group starts first, then every load, then every store
    for (u32 t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const SegChunk ch = seg_chunk(a, v, t, wl);
        u32 carry = ch.carry0;
        for (int j0 = 0; j0 < SEG_IPT; j0 += QB) {
            u32 pv[QB], gfv[QB], live = 0;
#pragma unroll
            for (int q = 0; q < QB; q++) {
                u32 p, gf; bool ok, st, en;
                seg_step(v, ch, j0 + q, carry, p, ok, st, en, gf);
                pv[q] = p; gfv[q] = gf;
                if (ok && !(st && en)) live |= 1u << q;  // groups of one were resolved by part 1
                if (ok && a.rank_passes) {  // every position's rank, streamed by the rank passes
                    const u32 b = ch.blo == ch.bhi ? ch.blo : blk_of_pos(a, p, ch.blo, ch.bhi);
                    __stcg(v.rk + p, gf - a.blk[b].soff);
                }
            }
            u32 idv[QB], giv[QB], gbv[QB];
#pragma unroll
            for (int q = 0; q < QB; q++) {
                if (!((live >> q) & 1)) continue;
                idv[q] = __ldcs(v.val + pv[q]);
                giv[q] = __ldg(v.gidx + gfv[q]);
                gbv[q] = __ldg(v.gbase + gfv[q]);
            }
#pragma unroll
            for (int q = 0; q < QB; q++) {
                if (!((live >> q) & 1)) continue;
                const u32 id = idv[q], gi = giv[q], p = pv[q], gf = gfv[q];
                const u32 slot = gbv[q] + (p - gf);
                KGB_GUARD(id < a.cap_n && slot < a.cap_n, &c->err, E_LIST) {
                    if (!a.rank_passes) {
                        const u32 b = ch.blo == ch.bhi ? ch.blo : blk_of_pos(a, p, ch.blo, ch.bhi);
                        a.isa[rpar ^ 1][id] = gf - a.blk[b].soff;
                    }
                    if (gi & GRP_LARGE) {
                        ll.eid[slot] = id;
                        if (slot % TSM == 0) {
                            KGB_GUARD(slot / TSM < a.cap_tml, &c->err, E_TMAP) ll.tmap[slot / TSM] = gi & ~GRP_LARGE;
                        }
                    } else if (gi & GRP_TINY) {
                        tl_.eid[slot] = id;
                    } else if (gi & GRP_MED) {
                        ml_.eid[slot] = id;
                    } else {
                        sl.eid[slot] = id;
                    }
                }
            }
        }
        __syncthreads();
    }
}

// Ranks after round 0 (every suffix: its group's first position in its block), for the suffixes whose id lies in
// [lo, hi). The host runs one pass per id range of RANK_SPAN ids, so that the rank writes of a pass (a scatter over
// 4 * RANK_SPAN bytes) stay in L2 and reach DRAM as whole sectors, instead of one read-modify-write per suffix;
// every pass streams the sorted ids again and reads the ranks that the second emit kernel wrote per position.
constexpr u32 RANK_SPAN = 16u << 20;
// More passes than this cost more streaming than the random writes they replace (about 4 ps per suffix and pass
// against about 29 ps per random rank write, measured on a 64 MiB block): the emit kernels write the ranks instead,
// as they do when no block exceeds RANK_SPAN suffixes (their writes then stay within one block's ids at a time).
constexpr u32 RANK_PASSES_MAX = 4;
__global__ void __launch_bounds__(TPB) k_seg_rank(FwdArgs a, u32 lo, u32 hi) {
    Ctl *c = a.ctl;
    const SegBufs v = seg_bufs(a);
    u32 *isa_nxt = a.isa[c->rpar ^ 1];
    const u32 span = hi - lo;
    // four positions per thread and step: one 16-byte load of their ids, the ranks loaded only where an id is in range
    const u32 m4 = v.m / 4;
    const uint4 *ids4 = reinterpret_cast<const uint4 *>(v.val);
    for (u32 i = blockIdx.x * TPB + threadIdx.x; i < m4; i += gridDim.x * TPB) {
        const uint4 q = __ldcs(ids4 + i);
        const u32 id[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (id[k] - lo >= span) continue;
            KGB_GUARD(id[k] < a.cap_n, &c->err, E_RANK) isa_nxt[id[k]] = __ldg(v.rk + 4 * i + k);
        }
    }
    for (u32 p = m4 * 4 + blockIdx.x * TPB + threadIdx.x; p < v.m; p += gridDim.x * TPB) {
        const u32 id = v.val[p];
        if (id - lo >= span) continue;
        KGB_GUARD(id < a.cap_n, &c->err, E_RANK) isa_nxt[id] = v.rk[p];
    }
}
