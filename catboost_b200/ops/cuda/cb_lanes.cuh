// Histogram accumulation with one feature per bank.
//
// What bounds a level at 128 borders is the shared-memory atomic pipe.  When the 32 lanes of a reduction hold one feature of
// 32 documents, they hit 32 random banks and the instruction takes 3.4 passes of that pipe (measured; 1.05 without
// conflicts).  Here cell (bin, statistic, feature) lives in bank `feature` and a lane holds one word of a document -- its
// bins of 4 features: lane l of 32 has features 4 g .. 4 g + 3, g = l % 8, of document d = l / 8.  In step j it adds to
// feature 4 g + (j + d) % 4, so that the 32 lanes are on 32 different features, hence banks, in every step, whatever the
// data look like -- also on sparse columns, where most documents share one bin -- and without replicas.
//   FL = 32: 4 documents x 32 features a reduction, cells [bin][statistic][32]
//   FL = 16: 8 documents x 16 features, cells [bin][statistic * 16 + feature]: documents 0-3 add their first statistic while
//            4-7 add their second, then the other way round
//   FL =  8: 16 documents x 8 features, cells [bin][replica * 16 + statistic * 8 + feature]
//
// The bins come from a second copy of the store, made once per training run (cb_lane_store_kernel): groups 8 s .. 8 s + 7
// form row block s, and the row of a document in it is up to 8 words, so that a document's 32 features are one 32-byte
// sector.  From level 1 on only the documents of the lighter children are accumulated: a warp appends them to a ring in
// shared memory (row number, two quantised statistics, slot) and fetches and adds 32 of them at a time, so documents that
// are not taken cost neither traffic nor reductions.
//
// Cells are int32 fixed point.  The scale follows from the number of documents a cell can receive, which is COUNTED once
// per work list (cb_lane_cap_kernel): the largest number of documents of one chunk in one bin, the most frequent bin of
// every feature left out.  That bin's cell may wrap around; it is replaced by (total - sum of the other bins), taken in
// 64 bits, when the tile is written out.
#pragma once
#include "cb_tree.cuh"

// 26 warps: one block per SM, 72 registers a thread (the words of two batches stay in registers; 34 words of the whole level
// kernel are spilled), and the staging areas leave room for six slots of 32 features x 129 bins -- 16 slots, level 5, are
// three passes then and four with 28 warps.
#define CB_LANE_THREADS 832
#define CB_LANE_RING 64                                // documents a warp's ring holds
#define CB_LANE_STAGE_INTS (CB_LANE_RING * 3 + 64)     // {q0, q1 << 8 | slot} and the row number of each; 32 entries in flight

// Words of a document's row in the row block of group g: 8, 4 or 2.
__host__ __device__ __forceinline__ int cb_lane_row(int G, int g) {
    const int left = G - (g & ~7);
    return left > 4 ? 8 : (left > 2 ? 4 : 2);
}

// Rows of a row block: whole steps of a thread block, so that the rows of a partial step can be read without a test.
__host__ __device__ __forceinline__ long long cb_lane_npad(long long n) {
    return (n + 2 * CB_LANE_THREADS - 1) / (2 * CB_LANE_THREADS) * (2 * CB_LANE_THREADS);
}

// Ints of shared memory behind the tile: per slot 2 x 32 lane totals, and the warps' staging area.
__host__ __device__ __forceinline__ int cb_lane_extra_ints(int slots) {
    return slots * 64 + (CB_LANE_THREADS / 32) * CB_LANE_STAGE_INTS;
}

// Largest fixed-point value.  From level 1 on it stays a few quanta below 2^23: a ring entry holds 24 bits, and the largest
// value times its scale may round up.  (A cell of level 0 can receive 53 documents or more: the limit there never acts.)
__device__ __forceinline__ float cb_lane_qmax(unsigned int cap, int level) {
    return fminf(level == 0 ? 1.0e9f : 8388600.0f, floorf(2147483647.0f / (float)(cap + 1u)) - 1.0f);
}

// One reduction into shared memory.  Unlike cb_red_shared it does not order other memory accesses: the staged entries are
// read ahead of it.
template <int OFF>
__device__ __forceinline__ void cb_lane_red(unsigned int addr, int v) {
    asm volatile("red.shared.add.s32 [%0 + %2], %1;" ::"r"(addr), "r"(v), "n"(OFF));
}

// ROOT: level 0, where every document is taken and rows are read in order.
// A step is 64 documents of a warp, two a lane: their leaf indices, split column and statistics are fetched one step ahead
// (with one document a lane the loop is bound by the latency of these loads: 67 us for 10.5M documents of which none is
// taken), the words of a batch of 32 one batch ahead.  An entry is read back as 8 bytes (16 would cost the shared-memory
// pipe a second pass).
template <int FL, bool ROOT>
static __device__ __forceinline__ void cb_lane_accumulate(const CbHistArgs& a, int* sh, const CbBundle& bd, float qmax, int chunk,
                                                          int slot_begin, int slot_count, bool writes_leaf, int* list_count) {
    constexpr int NS = FL == 32 ? 2 : 1;               // 32-cell rows of a bin
    constexpr int DW = 128 / FL;                       // documents a load covers: FL / 4 lanes each
    constexpr int NL = 32 / DW;                        // loads of a batch of 32 documents
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane % (FL / 4), d = lane / (FL / 4);
    const unsigned int slot_bytes = (unsigned int)bd.B * NS * 128u;
    const unsigned int sbase = (unsigned int)__cvta_generic_to_shared(sh);
    const unsigned int tbase = sbase + (unsigned int)slot_count * slot_bytes + (unsigned int)lane * 4u;   // [slot][statistic][32]
    int2* ring = reinterpret_cast<int2*>(sh + slot_count * (bd.B * NS * 32 + 64) + warp * CB_LANE_STAGE_INTS);
    unsigned int* rrow = reinterpret_cast<unsigned int*>(ring + CB_LANE_RING);
    int2* flight = reinterpret_cast<int2*>(rrow + CB_LANE_RING);       // the batch whose words are on the way
    // Lane constants of the four steps: which byte of the word comes second, and -- first byte -- the place of the
    // feature's cells in a bin (for FL < 32 times two: bins are 128 bytes there).
    unsigned int sel[4], cell[4];
    const bool flip = FL < 32 && ((d >> 2) & 1);       // adds its second statistic first
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const unsigned int k = (unsigned int)(j + d) & 3u;
        sel[j] = 0x5504u | (k << 4);
        cell[j] = (4u * g + k) * 4u + (FL == 8 ? (unsigned int)(d >> 3) * 64u : 0u) + (flip ? FL * 4u : 0u);
        if (FL < 32) cell[j] *= 2u;
    }
    const int other = flip ? -FL * 4 : FL * 4;         // FL < 32: from a lane's first statistic to its second
    const int level = a.level;
    const unsigned int pmask = (unsigned int)(cb_hist_nslots(a) - 1);
    const long long npad = a.d.npad;
    const int n = (int)a.d.n;                          // the host keeps longer shards off this path
    const float sc0 = qmax / fmaxf(a.statmax[0], 1e-30f), sc1 = qmax / fmaxf(a.statmax[1], 1e-30f);
    // word g of the bundle in row 0 (lanes without a group repeat the first one into cells that nobody reads)
    const unsigned int RS = (unsigned int)cb_lane_row(a.d.G, bd.g0);
    const uint32_t* rows = a.lanes + (bd.g0 & ~7) * cb_lane_npad(n) + (bd.g0 & 7) + (g < bd.gcnt ? g : 0);
    // split of the previous level: its column is read next to the leaf index.  A document goes right when
    // bin - ulo <= uspan (one-hot: exactly this bin)
    const uint32_t* colp = nullptr;
    unsigned int ulo = 0u, uspan = 255u;
    int ush = 0;
    if (!ROOT && a.prev_splits) {
        const CbSplit ps = a.prev_splits[(long long)(*a.prev_iter) * a.prev_depth + level - 1];
        if (ps.feature >= 0) {
            colp = a.d.bins + (long long)(ps.feature >> 2) * npad;
            ush = (ps.feature & 3) * 8;
            ulo = (unsigned int)ps.bin + ((ps.flags & 1) ? 0u : 1u);
            uspan = (ps.flags & 1) ? 0u : 255u;
        }
    }
    const unsigned int mask0 = ROOT ? 0u : a.small_mask[0];
    const unsigned int lt = (1u << lane) - 1u;
    // adds the 32 documents whose entries start at e and whose words are in w
    auto add = [&](const int2* e, const unsigned int (&w)[NL]) {
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            const int2 q = e[i * DW + d];
            const unsigned int base = ROOT ? sbase : sbase + ((unsigned int)q.y & 255u) * slot_bytes;
            const int q1 = ROOT ? q.y : q.y >> 8;
            const int va = flip ? q1 : q.x, vb = flip ? q.x : q1;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned int b = __byte_perm(w[i], cell[j], sel[j]);         // bin << 8 | place of the feature
                const unsigned int addr = base + (FL == 32 ? b : b >> 1);
                cb_lane_red<0>(addr, va);
                if (FL == 32) cb_lane_red<128>(addr, vb);
                else cb_lane_red<0>(addr + other, vb);
            }
        }
    };
    unsigned int w[NL];                                // words of the batch in flight
    bool flying = false;
    // fetches the words of the 32 entries from `head` on, adds the batch before them meanwhile
    auto drain = [&](int head) {
        unsigned int nw[NL];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NL; ++i) nw[i] = rows[rrow[head + i * DW + d]];
        if (flying) add(flight, w);
        const int2 mine = ring[head + lane];
        __syncwarp();
        flight[lane] = mine;
#pragma unroll
        for (int i = 0; i < NL; ++i) w[i] = nw[i];
        flying = true;
    };
    const int stride = bd.nK * (2 * CB_LANE_THREADS);
    int doc = chunk * (2 * CB_LANE_THREADS) + (int)threadIdx.x * 2;
    ushort2 nlf = make_ushort2(0, 0);                  // leaf indices, split column words and statistics of the next step
    uint2 ncw = make_uint2(0, 0);
    float2 ns0 = make_float2(0.f, 0.f), ns1 = ns0;
    auto fetch = [&](int i) {                          // (arrays are padded to a multiple of 256 documents)
        if (i < n) {
            if (!ROOT) nlf = *reinterpret_cast<const ushort2*>(a.leaf + i);
            if (!ROOT && colp) ncw = *reinterpret_cast<const uint2*>(colp + i);
            ns0 = *reinterpret_cast<const float2*>(a.stats + i);
            ns1 = *reinterpret_cast<const float2*>(a.stats + npad + i);
        }
    };
    fetch(doc);
    if (ROOT) {
        // documents 0..31 and 32..63 of a step are a batch each
        unsigned int w1[NL];
        const uint32_t* r = rows + (long long)(doc - 2 * lane + d) * RS;
        const long long rstep = (long long)stride * RS;
        if (doc - 2 * lane < n) {
#pragma unroll
            for (int i = 0; i < NL; ++i) w[i] = r[i * DW * RS];
        }
        for (; doc - 2 * lane < n; doc += stride, r += rstep) {
            const bool v0 = doc < n, v1 = doc + 1 < n;
            const int a0 = v0 ? __float2int_rn(ns0.x * sc0) : 0, a1 = v0 ? __float2int_rn(ns1.x * sc1) : 0;
            const int b0 = v1 ? __float2int_rn(ns0.y * sc0) : 0, b1 = v1 ? __float2int_rn(ns1.y * sc1) : 0;
            fetch(doc + stride);
            __syncwarp();
            reinterpret_cast<int4*>(ring)[lane] = make_int4(a0, a1, b0, b1);
            cb_lane_red<0>(tbase, a0 + b0);
            cb_lane_red<128>(tbase, a1 + b1);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < NL; ++i) w1[i] = r[(i * DW + 32) * RS];
            add(ring, w);
            if (doc - 2 * lane + stride < n) {
#pragma unroll
                for (int i = 0; i < NL; ++i) w[i] = r[rstep + i * DW * RS];
            }
            add(ring + 32, w1);
        }
        return;
    }
    int head = 0, tail = 0;
    auto push = [&](bool take, unsigned int m, int q0, int q1, int slot, unsigned int row) {
        if (take) {
            const int at = (tail + __popc(m & lt)) & (CB_LANE_RING - 1);
            ring[at] = make_int2(q0, (int)((unsigned int)q1 << 8) | slot);
            rrow[at] = row;
            const unsigned int t = tbase + (unsigned int)slot * 256u;
            cb_lane_red<0>(t, q0);
            cb_lane_red<128>(t, q1);
        }
        tail += __popc(m);
        if (tail - head >= 32) {
            drain(head & (CB_LANE_RING - 1));
            head += 32;
        }
    };
    // The list of the documents that later passes of this item take: entries as in the ring, with the slot of the level.
    int2* lq = a.list_q + (long long)blockIdx.x * a.list_len;
    unsigned int* lr = a.list_row + (long long)blockIdx.x * a.list_len;
    if (bd.seq && slot_begin > 0) {
        const int cnt = *list_count;
        int i = warp * 32 + lane;
        int2 ne = make_int2(0, 0);
        unsigned int nr = 0u;
        if (i < cnt) { ne = lq[i]; nr = lr[i]; }
        for (; i - lane < cnt; i += CB_LANE_THREADS) {
            const int2 e = ne;
            const unsigned int row = nr;
            if (i + CB_LANE_THREADS < cnt) { ne = lq[i + CB_LANE_THREADS]; nr = lr[i + CB_LANE_THREADS]; }
            const int slot = (e.y & 255) - slot_begin;
            const bool take = i < cnt && (unsigned)slot < (unsigned)slot_count;
            const unsigned int m = __ballot_sync(0xffffffffu, take);
            if (m) push(take, m, e.x, e.y >> 8, slot, row);
        }
    } else {
        const bool keep = bd.seq && bd.npass > 1;
        for (; doc - 2 * lane < n; doc += stride) {    // doc - 2 lane is the same in all lanes
            const float s0[2] = {ns0.x, ns0.y}, s1[2] = {ns1.x, ns1.y};
            unsigned int lf[2] = {nlf.x, nlf.y};
            const uint2 cw = ncw;
            fetch(doc + stride);
            if (colp) {
                lf[0] |= (unsigned int)(((cw.x >> ush) & 255u) - ulo <= uspan) << (level - 1);
                lf[1] |= (unsigned int)(((cw.y >> ush) & 255u) - ulo <= uspan) << (level - 1);
                if (writes_leaf && doc < n)
                    *reinterpret_cast<ushort2*>(a.leaf_rw + doc) = make_ushort2((unsigned short)lf[0], (unsigned short)lf[1]);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const unsigned int p = lf[k] & pmask;
                const unsigned int mw = pmask < 32u ? mask0 : a.small_mask[p >> 5];
                const bool light = doc + k < n && (((lf[k] >> (level - 1)) ^ (mw >> (p & 31))) & 1u) == 0u;
                const int q0 = __float2int_rn(s0[k] * sc0), q1 = __float2int_rn(s1[k] * sc1);
                const unsigned int row = (unsigned int)(doc + k) * RS;
                if (keep) {
                    const bool later = light && p >= (unsigned)slot_count;
                    const unsigned int m = __ballot_sync(0xffffffffu, later);
                    if (m) {
                        int at = 0;
                        if (lane == 0) at = atomicAdd(list_count, __popc(m));
                        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & lt);
                        if (later) { lq[at] = make_int2(q0, (int)((unsigned int)q1 << 8) | (int)p); lr[at] = row; }
                    }
                }
                const int slot = (int)p - slot_begin;
                const bool take = light && (unsigned)slot < (unsigned)slot_count;
                const unsigned int m = __ballot_sync(0xffffffffu, take);
                push(take, m, q0, q1, slot, row);
            }
        }
    }
    if (tail > head) {
        // the rest, filled up with documents that add nothing
        const int at = (head + lane) & (CB_LANE_RING - 1);
        if (head + lane >= tail) { ring[at] = make_int2(0, 0); rrow[at] = 0u; }
        drain(head & (CB_LANE_RING - 1));
    }
    __syncwarp();
    if (flying) add(flight, w);
}

// One work item: zero the tile, accumulate, write it out as floats, priv[chunk][slot][bin][NS][32] of this bundle (the
// tile's own order, coalesced), adding up every lane's column without the feature's most frequent bin meanwhile.
template <int FL>
static __device__ __forceinline__ void cb_lane_item(const CbHistArgs& a, int* sh, const CbBundle& bd, unsigned int cap, int chunk,
                                                 int slot_begin, int slot_count, bool writes_leaf, int* list_count) {
    constexpr int SG = FL == 32 ? 1 : 2;
    constexpr int DP = 32 / (FL * SG);
    constexpr int NS = 2 / SG;
    constexpr int NWARP = CB_LANE_THREADS / 32;
    const int B = bd.B;
    const int slot_ints = B * NS * 32;
    const int tile = slot_count * slot_ints;
    int* tot = sh + tile;                              // [slot][statistic][32]
    for (int i = threadIdx.x; i < (tile + slot_count * 64) >> 2; i += CB_LANE_THREADS)
        reinterpret_cast<int4*>(sh)[i] = make_int4(0, 0, 0, 0);
    if (threadIdx.x == 0 && slot_begin == 0) *list_count = 0;
    __syncthreads();
    const float qmax = cb_lane_qmax(cap, a.level);
    if (a.level == 0) cb_lane_accumulate<FL, true>(a, sh, bd, qmax, chunk, slot_begin, slot_count, writes_leaf, list_count);
    else cb_lane_accumulate<FL, false>(a, sh, bd, qmax, chunk, slot_begin, slot_count, writes_leaf, list_count);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int fl = lane & (FL - 1), sg = (lane / FL) & (SG - 1), dg = lane / (FL * SG);
    float* dst = a.priv + ((size_t)chunk * cb_hist_nslots(a) + slot_begin) * (size_t)slot_ints + bd.priv0;
    // the reciprocals of the very scales that were used: two separately rounded quotients would bias every sum
    const float inv0 = (float)(1.0 / (double)(qmax / fmaxf(a.statmax[0], 1e-30f)));
    const float inv1 = (float)(1.0 / (double)(qmax / fmaxf(a.statmax[1], 1e-30f)));
    const int dom = fl < bd.gcnt * 4 ? (int)a.ldom[bd.g0 * 4 + fl] : -1;
    long long* part = reinterpret_cast<long long*>(tot + slot_count * 64);      // [warp][NS][32], over the staging area
    for (int s0 = 0; s0 < slot_count; s0 += NWARP) {
        // warps per slot: as many as there are, at most 8 (the sums of a slot are added up by one warp)
        const int here = min(NWARP, slot_count - s0);
        int wps = 1;
        while (wps < 8 && wps * 2 * here <= NWARP) wps *= 2;
        const int sl = warp / wps, sub = warp - sl * wps;
        const bool on = sl < here;
        long long acc[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[s] = 0;
        if (on) {
            const int* src = sh + (size_t)(s0 + sl) * slot_ints + lane;
            float* out = dst + (size_t)(s0 + sl) * slot_ints + lane;
#pragma unroll 4
            for (int bin = sub; bin < B; bin += wps) {
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int v = src[(bin * NS + s) * 32];
                    if (bin != dom) {
                        acc[s] += v;
                        out[(bin * NS + s) * 32] = (float)v * ((NS == 2 ? s : sg) ? inv1 : inv0);
                    }
                }
            }
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) part[(warp * NS + s) * 32 + lane] = acc[s];
        __syncthreads();
        if (on && sub == 0) {
            float* out = dst + (size_t)(s0 + sl) * slot_ints + lane;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const int st = NS == 2 ? s : sg;
                long long rest = 0;
                // FL = 8: the documents of both halves count into either total, so the second replica's cell stays empty
                const int* tt = tot + (s0 + sl) * 64 + st * 32;
                for (int l = 0; l < 32; ++l) rest += tt[l];
                for (int u = 0; u < wps; ++u) {
                    const long long* pp = part + ((warp + u) * NS + s) * 32;
                    rest -= pp[lane];
                    if (DP == 2) rest -= pp[lane ^ 16];
                }
                if (dom >= 0) out[(dom * NS + s) * 32] = (DP == 2 && dg) ? 0.0f : (float)rest * (st ? inv1 : inv0);
            }
        }
        __syncthreads();
    }
}

// All work items of a level: (bundle, slot pass, document chunk), handed out by a counter when there are more than blocks.
static __device__ void cb_lane_phase(const CbHistArgs& a, int* sh, int cta, int ncta) {
    const int nslots = cb_hist_nslots(a);
    const bool dyn = a.work && a.nbitems > ncta;
    __shared__ int s_item, s_list;
    for (int item = cta;; item += ncta) {
        if (dyn) {
            __syncthreads();
            if (threadIdx.x == 0) s_item = (int)atomicAdd(a.work + a.d.G, 1u);
            __syncthreads();
            item = s_item;
        }
        if (item >= a.nbitems) break;
        const int2 it = a.bitems[item];
        const int bi = it.x & 0xFFFF;
        const CbBundle bd = a.btab[bi];
        const unsigned int cap = a.bcap[bi];
        const int pass0 = it.x >> 16, pass1 = bd.seq ? bd.npass : pass0 + 1;
        for (int ps = pass0; ps < pass1; ++ps) {
            const int sb = ps * bd.spp, sc = min(bd.spp, nslots - sb);
            const bool wl = bi == 0 && ps == 0;
            if (bd.FL == 32) cb_lane_item<32>(a, sh, bd, cap, it.y, sb, sc, wl, &s_list);
            else if (bd.FL == 16) cb_lane_item<16>(a, sh, bd, cap, it.y, sb, sc, wl, &s_list);
            else cb_lane_item<8>(a, sh, bd, cap, it.y, sb, sc, wl, &s_list);
        }
    }
    if (dyn) __syncthreads();
}

// Largest number of documents of one chunk in one bin of one feature, most frequent bins left out; bcap[bundle] must
// hold at least the documents per lane total on entry.  One block per work item of the first slot pass.
static __global__ void __launch_bounds__(CB_LANE_THREADS, 1)
cb_lane_cap_kernel(CbData d, const uint32_t* lanes, const short* ldom, const CbBundle* btab, const int2* items, int nitems,
                   unsigned int* bcap) {
    extern __shared__ __align__(16) int cb_lane_sh[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int sbase = (unsigned int)__cvta_generic_to_shared(cb_lane_sh);
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int2 it = items[item];
        if (it.x >> 16) continue;                      // later slot passes see the same documents
        const int bi = it.x & 0xFFFF;
        const CbBundle bd = btab[bi];
        for (int i = threadIdx.x; i < bd.B * 32; i += CB_LANE_THREADS) cb_lane_sh[i] = 0;
        __syncthreads();
        const int RS = cb_lane_row(d.G, bd.g0);
        const int g = lane % (bd.FL / 4), dd = lane / (bd.FL / 4), DW = 128 / bd.FL;
        const uint32_t* rows = lanes + (bd.g0 & ~7) * cb_lane_npad(d.n) + (bd.g0 & 7) + g;
        for (long long b = it.y; b * (2 * CB_LANE_THREADS) < d.n; b += bd.nK) {
            const long long doc0 = b * (2 * CB_LANE_THREADS) + warp * 64 + dd;
            if (g >= bd.gcnt) continue;
            for (int i = 0; i < 64; i += DW) {
                if (doc0 + i >= d.n) break;
                const unsigned int w = rows[(doc0 + i) * RS];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned int k = (unsigned int)(j + dd) & 3u;
                    cb_red_shared(sbase + ((w >> (8 * k)) & 255u) * 128u + (4 * g + k) * 4u, 1);
                }
            }
        }
        __syncthreads();
        int best = 0;
        if (lane < bd.gcnt * 4) {
            // (a padding column, dom < 0, holds every document in bin 0; nobody reads its cells, so they may wrap around)
            const int dom = ldom[bd.g0 * 4 + lane];
            for (int bin = warp; bin < bd.B && dom >= 0; bin += CB_LANE_THREADS / 32)
                if (bin != dom) best = max(best, cb_lane_sh[bin * 32 + lane]);
        }
        best = __reduce_max_sync(0xffffffffu, best);
        if (lane == 0 && best > 0) atomicMax(bcap + bi, (unsigned int)best);
        __syncthreads();
    }
}

// The second copy of the store (layout above) from the group-major one: a thread reads 4 documents of one group; eight
// neighbouring threads write whole rows.
static __global__ void cb_lane_store_kernel(CbData d, uint32_t* lanes) {
    const long long npad = cb_lane_npad(d.n), quads = npad >> 2;
    const int blocks = (d.G + 7) >> 3;                 // row blocks
    const long long total = blocks * quads * 8;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const int gl = (int)(t & 7);
        const long long r = t >> 3;
        const long long q = r % quads;
        const int s = (int)(r / quads);
        const int g = s * 8 + gl;
        const int RS = cb_lane_row(d.G, s * 8);
        if (gl >= RS) continue;
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (g < d.G && q * 4 < d.npad) x = *reinterpret_cast<const uint4*>(d.bins + (long long)g * d.npad + q * 4);
        uint32_t* out = lanes + s * 8 * npad + q * 4 * RS + gl;
        out[0] = x.x; out[RS] = x.y; out[2 * RS] = x.z; out[3 * RS] = x.w;
    }
}
