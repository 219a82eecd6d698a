// K6 fused level kernel: ONE cooperative launch per tree level does
//   (0) the leaf-index update for the split chosen at the previous level (inside the histogram pass when the
//       bundled path runs: the pass has the bin words of its documents in registers anyway),
//   (A) streaming histogram accumulation of the local rows (shared-memory integer atomics, one slot per parent
//       leaf: only the lighter child is accumulated, the sibling is parent - child); two-statistic fixed-point levels
//       of three or more feature groups keep every feature in a bank of its own (cb_lanes.cuh),
//   (B) the reduce-scatter: every rank sums its chunk tiles and stores the feature slice that rank r owns straight
//       into rank r's slot buffer over NVLink as tagged 8-byte words (value + level tag),
//   (C) on the owner: the score phase polls the words it needs until they carry this level's tag (bounded), sums the
//       per-source slots in rank order (deterministic), sibling subtraction, bin prefix scan, split scoring, packed
//       64-bit atomicMax argmax -- no fence, flag or grid barrier stands between (B) and (C),
//   (D) an exchange of the per-rank best (key + lighter-child mask) as tagged words through the peer mailboxes and
//       the final argmax, which every rank evaluates identically.
// No NCCL call, no host round trip and no separate scoring kernel per level.  This replaces the reference's
// four-step path: histogram kernel -> GatherHistogramsByLeaves -> host-orchestrated ReduceScatter built from
// cudaMemcpyAsync + add kernel -> FindOptimalSplit -> device-to-host read + host argmin
// (catboost/cuda/methods/histograms_helper.cpp:58-91, cuda_lib/cuda_buffer_helpers/reduce_scatter.h:449-540,
// catboost/cuda/methods/histograms_helper.h:322-331).
//
// Only plain peer stores / loads touch remote memory: no bulk-copy engine, no switch-side reduction.
#include "cb_common.cuh"
#include <cstdlib>
#include "cb_tree.cuh"
#include "cb_lanes.cuh"
#include "cb_comm.cuh"
#include <cooperative_groups.h>
#include <new>
#include <vector>
#include <algorithm>
#include <functional>
#include <queue>
#include <utility>

namespace cg = cooperative_groups;

struct CbFusedArgs {
    CbHistArgs h;            // h.priv = per-block private tiles; h.out is unused by the fused kernel
    CbScoreArgs s;           // s.hsrc[r] = local slot r; s.W = owned width; s.col_base = first owned column
    CbComm c;
    unsigned short* leaf;
    CbSplit* splits; int depth;
    unsigned int* mask_out;          // lighter-child mask for the next level
    unsigned long long* msg_local;   // CB_SELECT_MSG_BYTES scratch in local memory
    unsigned long long* msg_stage;   // [nranks][msg_stage_stride] words: the peers' messages, unpacked from the mailbox
    int msg_stage_stride;
    int fuse_leaf;                   // 1: the histogram pass of this launch also applies the previous level's split
    int own_col[CB_MAX_RANKS + 1];   // rank r owns histogram columns [own_col[r], own_col[r+1]) (multiples of 4)
    int Wmax;                        // row stride (floats) of every slot buffer = max owned width
    int smem_floats;                 // dynamic shared memory of this launch, in floats
    unsigned long long* phase_ts;    // optional globaltimer stamps (phase profiling): [depth][8] by block 0,
                                     // then [4096][2] per-block histogram end + SM id, then [depth][4] inside the score phase
};

// Sum of the per-chunk private tiles of this rank, written to the owner's slot.  A unit of work is one 16-byte column
// group of one (slot, statistic) row.  At the shallow levels there are few units and many chunks (a bundle of all
// groups is cut into as many chunks as there are blocks), so the chunks of a unit are dealt to KS lanes of a warp
// (KS a power of two <= 32, as many as the grid has spare threads for) and combined with shuffles.
static __device__ void cb_reduce_chunks(const CbFusedArgs& a, int cta, int ncta, unsigned int ll_tag) {
    const CbHistArgs& h = a.h;
    const int G = h.d.G, S = h.S, B = h.B, TB = h.d.TB;
    const int nK = cb_hist_chunks(G, ncta, h.d.n, h.nK);
    const int nslots = cb_hist_nslots(h);
    const size_t slot_stride = (size_t)S * 4 * B;
    const size_t item_stride = (size_t)nslots * slot_stride;
    const int rows = nslots * S;
    const int C4 = TB >> 2;
    const int R = a.c.nranks, me = a.c.rank;
    const long long total = (long long)rows * C4;
    const long long gthreads = (long long)ncta * blockDim.x;
    int KS = 1;
    while (KS < 32 && total * (KS * 2) <= gthreads && KS * 2 <= nK) KS <<= 1;
    const int CW = 32 / KS;                      // units per warp
    const int lane = threadIdx.x & 31;
    const int cl = lane & (CW - 1), ks = lane / CW;
    const long long gwarp = ((long long)cta * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = gthreads >> 5;
    for (long long base = gwarp * CW; base < total; base += nwarps * CW) {
        const long long u = base + cl;
        const bool valid = u < total;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        int row = 0, col = 0;
        if (valid) {
            row = (int)(u / C4);
            col = (int)(u % C4) << 2;
            const int f = cb_find_feature(h.d.feat_off, h.d.F, col);
            const int bin = col - h.d.feat_off[f];
            const int slot = row / S, st = row - slot * S;
            const float* src = h.priv + ((size_t)slot * S + st) * 4 * B + (size_t)(f & 3) * B + bin
                               + (size_t)(f >> 2) * item_stride;
            const size_t kstride = (size_t)G * item_stride;
            const int nKg = h.gchunks ? h.gchunks[f >> 2] : nK;       // chunks of this group's bundle
#pragma unroll 4
            for (int k = ks; k < nKg; k += KS) {
                const float4 v = __ldcg(reinterpret_cast<const float4*>(src + (size_t)k * kstride));
                acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
            }
        }
        for (int off = CW; off < 32; off <<= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
            acc.z += __shfl_xor_sync(0xffffffffu, acc.z, off);
            acc.w += __shfl_xor_sync(0xffffffffu, acc.w, off);
        }
        if (valid && ks == 0) {
            if (R > 1) {
                // tagged words: {value, level tag} pairs, two per 16-byte store (each 8-byte half is atomic on its own)
                int r = 0;
                while (r + 1 < R && col >= a.own_col[r + 1]) ++r;
                unsigned long long* dst = reinterpret_cast<unsigned long long*>(a.c.peer_slot[r] + (size_t)me * a.c.slot_floats)
                                          + (size_t)row * a.Wmax + (col - a.own_col[r]);
                const unsigned long long t = (unsigned long long)ll_tag << 32;
                const unsigned long long w0 = t | __float_as_uint(acc.x), w1 = t | __float_as_uint(acc.y);
                const unsigned long long w2 = t | __float_as_uint(acc.z), w3 = t | __float_as_uint(acc.w);
                asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(dst), "l"(w0), "l"(w1) : "memory");
                asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(dst + 2), "l"(w2), "l"(w3) : "memory");
            } else {
                float* dst = const_cast<float*>(a.s.hsrc[0]) + (size_t)row * a.Wmax + col;
                *reinterpret_cast<float4*>(dst) = acc;
            }
        }
    }
}

// The same for the feature-per-lane path, whose tiles are [slot][bin][NS][32 lanes].  A unit is four bins of one (slot,
// statistic of the lane) row: a warp adds four 128-byte rows per chunk and every lane stores the 16 bytes of its feature.
// With few units the chunks of a unit are dealt to KS warps of a block, which meet in shared memory.  Sums in 64 bits: with
// up to 148 chunks an fp32 sum would be the largest error of a dense column's histogram.
static __device__ void cb_reduce_lanes(const CbFusedArgs& a, float* sh, int cta, int ncta, unsigned int ll_tag) {
    const CbHistArgs& h = a.h;
    const int nslots = cb_hist_nslots(h);
    const int R = a.c.nranks, me = a.c.rank;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const CbBundle last = h.btab[h.nbundles - 1];
    const int units = last.unit0 + nslots * (last.B >> 2) * (last.FL == 32 ? 2 : 1);
    int KS = 1;
    while (KS * 2 <= nwarp && (long long)units * (KS * 2) <= (long long)ncta * nwarp && KS * 2 <= h.nK) KS <<= 1;
    const int upb = nwarp / KS, ks = warp % KS;
    double4* red = reinterpret_cast<double4*>(sh);
    for (int ub = cta * upb; ub < units; ub += ncta * upb) {
        const int u = warp / KS < upb ? ub + warp / KS : units;
        double4 sum = make_double4(0.0, 0.0, 0.0, 0.0);
        CbBundle bd;
        int slot = 0, b4 = 0, s = 0, NS = 1;
        if (u < units) {
            int lo = 0, hi = h.nbundles - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (h.btab[mid].unit0 <= u) lo = mid; else hi = mid - 1;
            }
            bd = h.btab[lo];
            NS = bd.FL == 32 ? 2 : 1;
            int v = u - bd.unit0;
            s = v % NS; v /= NS;
            b4 = v % (bd.B >> 2);
            slot = v / (bd.B >> 2);
            const int rs = NS * 32;
            const size_t kstride = (size_t)nslots * bd.B * rs;
            const float* src = h.priv + bd.priv0 + ((size_t)slot * bd.B + b4 * 4) * rs + s * 32 + lane;
#pragma unroll 4
            for (int k = ks; k < bd.nK; k += KS) {
                const float* q = src + (size_t)k * kstride;
                const float x = __ldcg(q), y = __ldcg(q + rs), z = __ldcg(q + 2 * rs), w = __ldcg(q + 3 * rs);
                sum.x += x; sum.y += y; sum.z += z; sum.w += w;
            }
        }
        if (KS > 1) {
            red[threadIdx.x] = sum;
            __syncthreads();
            if (ks == 0)
                for (int w = 1; w < KS; ++w) {
                    const double4 t = red[(warp + w) * 32 + lane];
                    sum.x += t.x; sum.y += t.y; sum.z += t.z; sum.w += t.w;
                }
            __syncthreads();
        }
        if (u >= units || ks != 0) continue;
        float4 acc = make_float4((float)sum.x, (float)sum.y, (float)sum.z, (float)sum.w);
        if (bd.FL == 8) {                              // two replicas, one per document of a reduction
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
            acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16);
            acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
            if (lane >= 16) continue;
        }
        const int fl = lane & (bd.FL - 1);
        const int f = bd.g0 * 4 + fl;
        if (fl >= bd.gcnt * 4 || f >= h.d.F) continue;
        const int col = h.d.feat_off[f] + b4 * 4;
        if (col >= h.d.feat_off[f + 1]) continue;
        const int row = slot * 2 + (NS == 2 ? s : lane / bd.FL);
        if (R > 1) {
            int r = 0;
            while (r + 1 < R && col >= a.own_col[r + 1]) ++r;
            unsigned long long* dst = reinterpret_cast<unsigned long long*>(a.c.peer_slot[r] + (size_t)me * a.c.slot_floats)
                                      + (size_t)row * a.Wmax + (col - a.own_col[r]);
            const unsigned long long t = (unsigned long long)ll_tag << 32;
            const unsigned long long w0 = t | __float_as_uint(acc.x), w1 = t | __float_as_uint(acc.y);
            const unsigned long long w2 = t | __float_as_uint(acc.z), w3 = t | __float_as_uint(acc.w);
            asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(dst), "l"(w0), "l"(w1) : "memory");
            asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(dst + 2), "l"(w2), "l"(w3) : "memory");
        } else {
            *reinterpret_cast<float4*>(const_cast<float*>(a.s.hsrc[0]) + (size_t)row * a.Wmax + col) = acc;
        }
    }
    __syncthreads();
}

// LANES: the feature-per-lane histogram pass (two statistics, fixed point); a separate instantiation, so that neither
// path's registers and instruction lines burden the other.
template <bool LANES>
__global__ void __launch_bounds__(LANES ? CB_LANE_THREADS : 1024, 1) cb_level_fused_kernel(CbFusedArgs a) {
    extern __shared__ __align__(16) float cb_sh[];
    cg::grid_group grid = cg::this_grid();
    const int cta = blockIdx.x, ncta = gridDim.x;
    const int level = a.h.level;
    const int it = *a.s.iter_ptr;
    CbSplit* sp_arr = a.splits + (long long)it * a.depth;
    unsigned long long* ts = (a.phase_ts && cta == 0 && threadIdx.x == 0) ? a.phase_ts + level * 8 : nullptr;
    if (ts) ts[0] = cb_globaltimer();
    const int R = a.c.nranks, me = a.c.rank;
    // every block reads the level counter before the first grid barrier; block 0 advances it at the very end
    const unsigned long long hist_epoch = (R > 1) ? a.c.epoch[1] + 1 : 0ull;
    const unsigned int ll_tag = (R > 1) ? cb_ll_tag(hist_epoch) : 0u;

    // (0) leaf update with the split of the previous level: its own pass, unless the histogram pass does it
    if (!LANES && level > 0 && !a.fuse_leaf) {
        cb_update_leaf_range(a.h.d, a.leaf, sp_arr[level - 1], level - 1,
                             (long long)cta * blockDim.x + threadIdx.x, (long long)ncta * blockDim.x);
        __threadfence();
        grid.sync();
    }

    // the score noise scale only depends on the iteration: one thread per block works it out now, off the critical path
    __shared__ float s_noise_std;
    if (threadIdx.x == 0) s_noise_std = cb_noise_std(a.s);
    if (ts) ts[1] = cb_globaltimer();
    // (A) local histograms: every block dumps its shared-memory tile into its private region (no atomics)
    if (LANES) cb_lane_phase(a.h, reinterpret_cast<int*>(cb_sh), cta, ncta);
    else cb_hist_phase(a.h, cb_sh, cta, ncta);
    if (ts) ts[2] = cb_globaltimer();
    if (a.phase_ts && threadIdx.x == 0 && level == a.depth - 2) {
        unsigned int smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        a.phase_ts[a.depth * 8 + cta * 2] = cb_globaltimer();
        a.phase_ts[a.depth * 8 + cta * 2 + 1] = smid;
    }
    __threadfence();
    grid.sync();
    if (ts) ts[3] = cb_globaltimer();

    // (B) chunk reduction fused with the reduce-scatter: each 16-byte column group is summed over the chunks of
    // this rank and stored straight into the slot of the rank that owns the column (peer store over NVLink when
    // that is another GPU; every source keeps its own slot, so the owner later adds them in rank order).
    if (LANES) cb_reduce_lanes(a, cb_sh, cta, ncta, ll_tag);
    else cb_reduce_chunks(a, cta, ncta, ll_tag);
    if (R <= 1) {
        __threadfence();
        grid.sync();
    }
    // several ranks: (C) needs no barrier here, the words announce themselves and the score phase polls exactly those
    // it reads (a.s.ll_epoch is set by the host)

    if (ts) ts[4] = cb_globaltimer();
    cb_score_phase(a.s, cta, ncta, cb_sh, a.smem_floats, ts ? a.phase_ts + a.depth * 8 + 8192 + level * 4 : nullptr,
                   s_noise_std);
    __threadfence();
    grid.sync();
    if (ts) ts[5] = cb_globaltimer();

    // (D) selection: one block
    if (cta == 0) {
        cb_select_local(a.s, a.msg_local);
        __threadfence();
        __syncthreads();
        const unsigned long long* msgs[CB_MAX_RANKS];
        if (R > 1) {
            // key (two words) + mask words, each as a tagged word into every rank's mailbox; then unpack the R messages
            // that arrived here into the staging rows
            __shared__ unsigned long long s_epoch;
            if (threadIdx.x == 0) { s_epoch = a.c.epoch[0] + 1; a.c.epoch[0] = s_epoch; }
            __syncthreads();
            const unsigned long long epoch = s_epoch;
            const unsigned int tag = cb_ll_tag(epoch);
            const int parity = (int)(epoch & 1ull);
            const int nw = 2 + (((1 << level) + 31) >> 5);
            const unsigned int* src = reinterpret_cast<const unsigned int*>(a.msg_local);
            for (int idx = threadIdx.x; idx < nw * R; idx += blockDim.x) {
                const int r = idx / nw, i = idx - r * nw;
                cb_ll_store(cb_ll_box(a.c, r, parity, me) + i, src[i], tag);
            }
            for (int idx = threadIdx.x; idx < nw * R; idx += blockDim.x) {
                const int r = idx / nw, i = idx - r * nw;
                reinterpret_cast<unsigned int*>(a.msg_stage + (size_t)r * a.msg_stage_stride)[i] =
                    cb_ll_load(cb_ll_box(a.c, me, parity, r) + i, tag, a.c.timeout_ns, a.c.status, CB_TIMEOUT_MAILBOX, r);
            }
            __threadfence();
            __syncthreads();
            for (int r = 0; r < R; ++r) msgs[r] = a.msg_stage + (size_t)r * a.msg_stage_stride;
        } else {
            msgs[0] = a.msg_local;
        }
        cb_select_final(a.h.d, msgs, R, level, sp_arr + level, a.mask_out);
        if (threadIdx.x == 0) {
            *a.s.best_key = 0ull;
            if (R > 1) a.c.epoch[1] = hist_epoch;
            if (ts) ts[6] = cb_globaltimer();
        }
        if (a.h.work) {
            for (int i = threadIdx.x; i <= a.h.d.G; i += blockDim.x) a.h.work[i] = 0u;
        }
    }
}

// ---- host side ---------------------------------------------------------------------------------------
#define CB_MAX_LEVELS 16
#define CB_LANE_SEQ_DOCS 65536
struct CbFusedPlan {
    CbFusedArgs a;
    int threads;
    int max_smem;      // dynamic shared memory one block may use
    int sm_smem;       // shared memory of one SM available to two resident blocks (after their static + reserved parts)
    int sm_count;
    int max_bundle;    // widest feature-group bundle of the single-cell histogram path (0 = off)
    int fuse_leaf_update;   // 1: let the bundled histogram pass apply the previous level's split (default)
    int max_copies;    // most replicas of a histogram cell (2 for dense columns; more when one bin dominates a column,
                       // where most lanes of a warp would otherwise add to the same cell)
    std::vector<int> group_bins;     // padded bins of the widest feature of every group (empty: all groups take B)
    // per level: bundle table and work list of the bundled path, on the device (made by cb_fused_geometry)
    CbBundle* d_btab[CB_MAX_LEVELS];
    int2* d_items[CB_MAX_LEVELS];
    int* d_gchunks[CB_MAX_LEVELS];     // document chunks of every feature group (those of its bundle)
    int n_btab[CB_MAX_LEVELS], n_items[CB_MAX_LEVELS];
    int single_pass_bundle[CB_MAX_LEVELS];     // 1: one bundle holds every group in one pass (leaf update can be fused)
    // feature-per-lane path (cb_lanes.cuh)
    const uint32_t* lanes;
    const short* ldom;
    cudaStream_t lane_stream;                  // the stream the lane store was made on; the work lists go there too
    std::vector<float> group_share;            // see cb_lane_plan (empty: a bin may hold every document)
    long long seq_docs;                        // documents of a chunk from which a work item takes it through all slot passes
    int lane_smem;                             // dynamic shared memory one block of that kernel may use
    int lane_level[CB_MAX_LEVELS];             // 1: the level takes that path
    long long lane_priv[CB_MAX_LEVELS];        // floats of its private tiles
    int lane_list[CB_MAX_LEVELS];              // entries of a block's document list
    unsigned int* d_cap[CB_MAX_LEVELS];
};


CB_API CbFusedPlan* cb_fused_create(const CbData* d, const CbComm* comm, unsigned short* leaf, const float* stats, int S,
                                    int B, float* partial, float* const* local_slots, float* hbuf0, float* hbuf1,
                                    const int* own_col, int Wmax, unsigned int* mask0, unsigned int* mask1,
                                    CbSplit* splits, int depth, float l2, int score_fn, float random_strength,
                                    const double* scal, const int* iter_ptr, unsigned long long seed, float lr,
                                    unsigned long long* best_key, unsigned long long* msg_local,
                                    unsigned long long* msg_stage, int msg_stage_stride, int threads) {
    CbFusedPlan* p = new (std::nothrow) CbFusedPlan();
    if (!p) return nullptr;
    CbFusedArgs& a = p->a;
    a.h.d = *d; a.h.leaf = leaf; a.h.stats = stats; a.h.S = S; a.h.B = B; a.h.out = nullptr; a.h.priv = partial; a.h.statmax = nullptr; a.phase_ts = nullptr; a.h.nK = 0; a.h.copies = 1; a.h.work = nullptr; a.h.narrow = 0; a.h.bundle = 0;
    a.h.slot_table = nullptr; a.h.nslots_table = 0; a.h.level = 0; a.h.small_mask = mask0; a.h.slots_per_pass = 1;
    a.s.d = *d;
    if (comm) a.c = *comm; else { a.c = CbComm(); a.c.nranks = 1; a.c.rank = 0; }
    const int R = a.c.nranks;
    for (int r = 0; r < CB_MAX_RANKS; ++r) a.s.hsrc[r] = r < R ? local_slots[r] : nullptr;
    a.s.nsrc = R;
    a.s.hprev = hbuf0; a.s.hcur = hbuf1;   // swapped per level at launch
    for (int r = 0; r <= CB_MAX_RANKS; ++r) a.own_col[r] = r <= R ? own_col[r] : own_col[R];
    a.Wmax = Wmax;
    a.s.W = Wmax;
    a.s.col_base = own_col[a.c.rank];
    // owned feature range from the owned columns
    int fb = 0, fe = 0;
    // feat_off is device memory; the caller passes feature ranges through own_col only, so the
    // feature range is resolved by cb_fused_set_features().
    a.s.f_begin = fb; a.s.f_end = fe;
    a.s.level = 0; a.s.S = S; a.s.small_mask = mask0; a.s.l2 = l2; a.s.score_fn = score_fn;
    a.s.random_strength = random_strength; a.s.scal = scal; a.s.iter_ptr = iter_ptr; a.s.seed = seed;
    a.s.learning_rate = lr; a.s.best_key = best_key;
    a.leaf = leaf; a.splits = splits; a.depth = depth; a.mask_out = mask1; a.msg_local = msg_local;
    a.msg_stage = msg_stage; a.msg_stage_stride = msg_stage_stride; a.fuse_leaf = 0;
    a.h.domw = nullptr; a.h.btab = nullptr; a.h.bitems = nullptr; a.h.nbitems = 0; a.h.gchunks = nullptr;
    a.h.prev_splits = nullptr; a.h.prev_iter = iter_ptr; a.h.prev_depth = depth; a.h.leaf_rw = leaf;
    a.s.ll_epoch = R > 1 ? a.c.epoch + 1 : nullptr; a.s.ll_timeout_ns = a.c.timeout_ns; a.s.ll_status = a.c.status;
    p->threads = threads;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&p->sm_count, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&p->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // dynamic shared memory available to this kernel = opt-in maximum minus its static shared memory
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, cb_level_fused_kernel<false>) != cudaSuccess) { cudaGetLastError(); delete p; return nullptr; }
    p->max_smem -= (int)fa.sharedSizeBytes;
    cudaDeviceGetAttribute(&p->sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    p->sm_smem -= 2 * (int)fa.sharedSizeBytes;
    p->max_bundle = 0;
    p->lanes = nullptr; p->ldom = nullptr; p->lane_stream = nullptr; p->seq_docs = CB_LANE_SEQ_DOCS;
    cudaFuncAttributes fl;
    if (cudaFuncGetAttributes(&fl, cb_level_fused_kernel<true>) != cudaSuccess) { cudaGetLastError(); delete p; return nullptr; }
    p->lane_smem = p->max_smem + (int)fa.sharedSizeBytes - (int)fl.sharedSizeBytes;
    for (int l = 0; l < CB_MAX_LEVELS; ++l) { p->lane_level[l] = 0; p->lane_priv[l] = 0; p->lane_list[l] = 0; p->d_cap[l] = nullptr; }
    a.h.lanes = nullptr; a.h.ldom = nullptr; a.h.bcap = nullptr; a.h.list_q = nullptr; a.h.list_row = nullptr; a.h.list_len = 0; a.h.nbundles = 0;
    for (int l = 0; l < CB_MAX_LEVELS; ++l) { p->d_btab[l] = nullptr; p->d_items[l] = nullptr; p->d_gchunks[l] = nullptr; p->n_btab[l] = p->n_items[l] = 0; p->single_pass_bundle[l] = 0; }
    p->max_copies = 2;
    p->fuse_leaf_update = 1;
    if (cudaFuncSetAttribute(cb_level_fused_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, p->max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(cb_level_fused_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, p->lane_smem) != cudaSuccess) {
        cudaGetLastError();
        delete p;
        return nullptr;
    }
    return p;
}

// domw: one packed word per feature group (the dominant bin of each of its four features, 255 = none), or null
CB_API void cb_fused_set_dominant(CbFusedPlan* p, const unsigned int* domw) { p->a.h.domw = domw; }
CB_API void cb_fused_set_fuse_leaf(CbFusedPlan* p, int on) { p->fuse_leaf_update = on ? 1 : 0; }
CB_API void cb_fused_set_phase_ts(CbFusedPlan* p, unsigned long long* ts) { p->a.phase_ts = ts; }
CB_API void cb_fused_set_work(CbFusedPlan* p, unsigned int* work) { p->a.h.work = work; }
CB_API void cb_fused_set_narrow(CbFusedPlan* p, int narrow, int max_bundle) {
    p->a.h.narrow = narrow;
    p->max_bundle = max_bundle > 8 ? 8 : max_bundle;
}

CB_API void cb_fused_set_features(CbFusedPlan* p, int f_begin, int f_end) {
    p->a.s.f_begin = f_begin;
    p->a.s.f_end = f_end;
}

CB_API void cb_fused_destroy(CbFusedPlan* p) {
    if (!p) return;
    for (int l = 0; l < CB_MAX_LEVELS; ++l) {
        if (p->d_btab[l]) cudaFree(p->d_btab[l]);
        if (p->d_items[l]) cudaFree(p->d_items[l]);
        if (p->d_gchunks[l]) cudaFree(p->d_gchunks[l]);
        if (p->d_cap[l]) cudaFree(p->d_cap[l]);
    }
    delete p;
}

// Padded number of bins (multiple of 4) of the widest feature of every feature group, host memory.  With it the
// bundled path sizes the tile of a bundle by its own widest feature instead of the widest feature of the data set.
CB_API void cb_fused_set_group_bins(CbFusedPlan* p, const int* group_bins, int G) {
    p->group_bins.assign(group_bins, group_bins + G);
}

// Launch geometry of one level.  Returns the cooperative grid size (0 on error) and, through the pointers, the
// slots per pass, dynamic shared memory, block size, document chunks per group and cell replicas.
CB_API void cb_fused_set_max_copies(CbFusedPlan* p, int max_copies) {
    p->max_copies = max_copies >= 8 ? 8 : (max_copies >= 4 ? 4 : (max_copies >= 2 ? 2 : 1));
}

// The lane-ordered copy of the store (words the caller allocates: cb_lane_store_words) and every feature's most frequent
// bin, [4 G] on the device; call before cb_fused_geometry.
CB_API long long cb_lane_store_words(long long n, int G) {
    const long long npad = cb_lane_npad(n);
    return (G >> 3) * 8 * npad + ((G & 7) ? cb_lane_row(G & 7, 0) * npad : 0);
}
CB_API int cb_lane_store(const CbData* d, uint32_t* lanes, cudaStream_t st) {
    const long long total = (long long)((d->G + 7) >> 3) * (cb_lane_npad(d->n) >> 2) * 8;
    const long long blocks = (total + 255) / 256;
    if (blocks == 0) return 0;
    cb_lane_store_kernel<<<(int)(blocks < 148 * 32 ? blocks : 148 * 32), 256, 0, st>>>(*d, lanes);
    return (int)cudaGetLastError();
}
// (lanes == nullptr: no level takes the path)
CB_API void cb_fused_set_lanes(CbFusedPlan* p, const uint32_t* lanes, const short* ldom, cudaStream_t st) {
    p->lanes = lanes;
    p->ldom = ldom;
    p->lane_stream = st;
}
// Documents of a chunk from which a work item takes its chunk through all slot passes (call before cb_fused_geometry).
CB_API void cb_fused_set_lane_seq(CbFusedPlan* p, long long docs) { p->seq_docs = docs; }
// share[g]: see cb_lane_plan, host memory
CB_API void cb_fused_set_lane_share(CbFusedPlan* p, const float* share, int G) { p->group_share.assign(share, share + G); }
// Floats of private tiles the level needs when it takes the feature-per-lane path (0: it does not).
CB_API long long cb_fused_lane_priv(CbFusedPlan* p, int level) {
    return level < CB_MAX_LEVELS && p->lane_level[level] ? p->lane_priv[level] : 0;
}

// Document list entries (12 bytes each) of the level, all blocks, and their place.
CB_API long long cb_fused_lane_list(CbFusedPlan* p, int level) {
    return level < CB_MAX_LEVELS && p->lane_level[level] ? (long long)p->lane_list[level] * p->sm_count : 0;
}
CB_API void cb_fused_set_lane_list(CbFusedPlan* p, int2* q, unsigned int* row) {
    p->a.h.list_q = q;
    p->a.h.list_row = row;
}

// ---- feature-per-lane path: what a level does, worked out on the host from sizes alone -------------------------------
struct CbLanePlan {
    std::vector<CbBundle> bundles;
    std::vector<double> cost;          // of a bundle
    std::vector<int2> items;
    std::vector<unsigned int> cap;     // documents a lane total can receive
    std::vector<unsigned int> limit;   // documents a cell may receive
    int smem = 0, chunks = 0, list = 0;        // document list entries of a block
    long long priv = 0;                // floats of private tiles
};

// Documents one cell may receive.  The fixed-point scale is 2^31 / (documents of the fullest cell), so this is the number of
// steps a statistic's range is cut into: values much smaller than the largest one all round the same way when the steps are
// coarse (0.5 % positives: the derivative of a negative is 20 steps at 2^19 documents a cell, 320 at 2^15).  2^17 leaves
// 16383 steps and 2^15 65534; the per-group path's chunks of 2^19 documents leave 4094 per replica of a cell, and it has one
// where there are many leaves, two where there are few.  What a chunk costs is its tiles (200 KB: about 16 us to zero, write
// and add up, as much as streaming 16K documents), so the limit follows their size: between 2^15 and 2^17.
static unsigned int cb_lane_cell_limit(long long tile_bytes) {
    const double v = 65536.0 * (double)tile_bytes / 200000.0;
    return v < 32768.0 ? 32768u : (v > 131072.0 ? 131072u : (unsigned int)v);
}

// gb[g]: padded bins of the widest feature of group g; share[g]: largest share of the documents that one bin of the group
// holds, the most frequent bin of every feature left out.  False: the level takes the other path.
static bool cb_lane_plan(CbLanePlan& out, long long n, int G, const int* gb, const float* share, int level, int grid, int lane_smem,
                         bool counter, long long seq_docs) {
    // One feature group leaves three quarters of a 32-byte sector unread (10.5M x 4: 0.90 against 0.78 ms an iteration on
    // the other path; 10.5M x 8: 0.90 against 0.85, 1.2M x 8 even, 100K x 8 0.28 against 0.30, from 12 columns on faster).
    // Document and row numbers are 32 bits wide, two work strides beyond the last document included.
    if (level >= CB_MAX_LEVELS || n >= (1ll << 28) || !(G > 2 || (G == 2 && n < (1ll << 22)))) return false;
    const int nslots = level == 0 ? 1 : (1 << (level - 1));
    const int ints = lane_smem / 4 - cb_lane_extra_ints(0);
    std::vector<CbBundle>& bundles = out.bundles;
    std::vector<double>& cost = out.cost;
    bundles.clear(); cost.clear(); out.items.clear(); out.cap.clear(); out.limit.clear();
    // Cost of streaming 32 documents through a bundle: a fixed part per slot pass and a part per document taken.
    const double taken = level == 0 ? 32.0 : 15.0;
    auto shape = [&](int g, int gc, CbBundle* b) {
        int B = 4;
        for (int q = 0; q < gc; ++q) B = gb[g + q] > B ? gb[g + q] : B;
        const int FL = gc > 4 ? 32 : (gc > 2 ? 16 : 8);
        const int per = B * (FL == 32 ? 64 : 32) + 64;
        int spp = ints / per;
        if (spp < 1) return 1e30;
        if (spp > 256) spp = 256;                      // eight bits of a staged entry
        if (spp > nslots) spp = nslots;
        const int np = (nslots + spp - 1) / spp;
        spp = (nslots + np - 1) / np;
        *b = CbBundle{g, gc, B, 1, spp, np, 1, FL, 0, 0, 0};
        return np * 25.0 + taken * (FL == 32 ? 3.2 : (FL == 16 ? 2.2 : 1.2));
    };
    for (int g = 0; g < G; g += 8) {
        const int gc = G - g < 8 ? G - g : 8;
        // a row block is one bundle, or is cut into halves (quarters) where a narrower tile saves enough slot passes
        CbBundle w, h[2], t[4];
        const double cw = shape(g, gc, &w);
        std::vector<CbBundle> cut;
        std::vector<double> ccut;
        for (int half = 0; half < 2 && half * 4 < gc; ++half) {
            const int hc = gc - half * 4 < 4 ? gc - half * 4 : 4;
            const double ch = shape(g + half * 4, hc, &h[half]);
            double cq = 1e30, c0 = 0.0, c1 = 0.0;
            if (hc > 2) {
                c0 = shape(g + half * 4, 2, &t[half * 2]);
                c1 = shape(g + half * 4 + 2, hc - 2, &t[half * 2 + 1]);
                cq = c0 + c1;
            }
            if (cq < ch) {
                cut.push_back(t[half * 2]); ccut.push_back(c0);
                cut.push_back(t[half * 2 + 1]); ccut.push_back(c1);
            } else { cut.push_back(h[half]); ccut.push_back(ch); }
        }
        double sum = 0.0;
        for (double c : ccut) sum += c;
        if (cw <= sum) { bundles.push_back(w); cost.push_back(cw); }
        else for (size_t i = 0; i < cut.size(); ++i) { bundles.push_back(cut[i]); cost.push_back(ccut[i]); }
    }
    for (double c : cost) if (c >= 1e29) return false;
    const int nbun = (int)bundles.size();
    if (nbun < 1 || nbun > 0xFFFF) return false;
    int& smem = out.smem;
    smem = 0;
    for (const CbBundle& b : bundles) {
        const int need = (b.spp * b.B * (b.FL == 32 ? 64 : 32) + cb_lane_extra_ints(b.spp)) * 4;
        if (need > smem) smem = need;
    }
    // the score phase reuses the tile as scratch; one block per SM runs either way, so every warp gets some
    const int want = (CB_LANE_THREADS / 32) * CB_SCORE_WARP_FLOATS * 4;
    if (smem < want) smem = want;
    // chunks: every item about the same time, their number a whole multiple of the grid; no more chunks than steps of a
    // thread block (and at most 4096, which keeps two strides inside 32 bits)
    const long long nblk = (n + 2 * CB_LANE_THREADS - 1) / (2 * CB_LANE_THREADS);
    const int most = (int)(nblk < 1 ? 1 : (nblk < 4096 ? nblk : 4096));
    // An item takes its chunk through all slot passes (one scan, the other passes read its list), or every pass is an item of
    // its own.  The former costs a tile a pass (200 KB that a block zeroes, writes and has added up: about 20 us), the latter a
    // scan a pass (0.62 ns a document), and its items differ, because the leaves of two passes hold different numbers of
    // documents (10.5M x 28: blocks finished between 98 and 230 us).  The line is at 64K documents a chunk.  An iteration, one
    // item / items of their own: 4M x 28, 129 bins, depth 6 (27K) 0.72 / 0.64 ms; 4M x 100, 129 bins, depth 8 (54K) 2.96 /
    // 2.83; 7M x 28, 129 bins, depth 6 (47K) 0.92 / 0.87; 10.5M x 28, 129 bins (71K) depth 6 1.14 / 1.13, depth 8 2.19 / 2.30;
    // 7M x 100, 255 bins, depth 8 (95K) 5.52 / 6.90; 16M x 28, 255 bins, depth 8 (108K) 3.67 / 5.07.
    bool mixed = false;
    for (int i = 1; i < nbun; ++i) mixed = mixed || cost[i] != cost[0];
    // items of different times are handed out by a counter in two rounds, where a second tile per block is small change
    const int two = (mixed && counter) ? 2 : 1;
    const int seq = n * nbun >= seq_docs * grid * two && nslots <= 256 ? 1 : 0;      // (a list entry has eight bits for the slot)
    double W = 0.0;
    long long min_items = 0;
    bool passes = false;
    std::vector<int> per(nbun), least(nbun);           // items a chunk of the bundle takes; fewest chunks
    for (int i = 0; i < nbun; ++i) {
        bundles[i].seq = seq;
        per[i] = seq ? 1 : bundles[i].npass;
        passes = passes || per[i] > 1;
        W += cost[i];
        // chunks small enough that no cell receives more documents than it may (a lane total has a 32nd of them all)
        float sh = 1.0f / 32.0f;
        for (int q = 0; q < bundles[i].gcnt; ++q) sh = share[bundles[i].g0 + q] > sh ? share[bundles[i].g0 + q] : sh;
        out.limit.push_back(cb_lane_cell_limit((long long)nslots * bundles[i].B * (bundles[i].FL == 32 ? 64 : 32) * 4));
        const double k = (double)n * sh / (double)out.limit[i];
        least[i] = k < 1.0 ? 1 : (k > (double)most ? most : (int)k + 1);
        if (least[i] > most) least[i] = most;
        min_items += (long long)least[i] * per[i];
    }
    // About `want` items, no bundle below its fewest chunks, evened out; returns the time (us) of the longest block.
    auto cut = [&](long long want) {
        long long used = 0;
        for (int i = 0; i < nbun; ++i) {
            int k = (int)((double)want * cost[i] / per[i] / W);
            k = k < least[i] ? least[i] : (k > most ? most : k);
            bundles[i].nK = k;
            used += (long long)k * per[i];
        }
        for (;;) {
            int pick = -1;
            double worst = 0.0;
            for (int i = 0; i < nbun; ++i) {
                if (used + per[i] > want || bundles[i].nK >= most) continue;
                const double t = cost[i] / per[i] / bundles[i].nK;
                if (t > worst) { worst = t; pick = i; }
            }
            if (pick < 0) break;
            ++bundles[pick].nK;
            used += per[pick];
        }
        std::vector<std::pair<double, long long>> kinds;               // time of an item, items
        for (int i = 0; i < nbun; ++i) {
            const CbBundle& b = bundles[i];
            kinds.push_back({2.5e-5 * (double)n / b.nK * cost[i] / per[i] + 3.0 + 8.0e-5 * b.spp * b.B * (b.FL == 32 ? 256 : 128),
                             (long long)b.nK * per[i]});
        }
        std::sort(kinds.begin(), kinds.end(), std::greater<std::pair<double, long long>>());
        std::priority_queue<double, std::vector<double>, std::greater<double>> blocks;
        for (int i = 0; i < grid; ++i) blocks.push(0.0);
        double last = 0.0;
        for (const auto& kind : kinds)
            for (long long i = 0; i < kind.second; ++i) {
                const double t = blocks.top() + kind.first;
                blocks.pop();
                blocks.push(t);
                last = t > last ? t : last;
            }
        return last;
    };
    long long T = (long long)grid * (seq ? two : 1);
    while (T < min_items) T += grid;
    double time = cut(T);
    // Slot passes come in whole multiples: 86 passes of one bundle leave 62 SMs idle (1.2M x 28, 255 bins, level 9: 670 us).
    // Cut finer where that fills the SMs better.
    if (passes && counter && T == grid) {
        long long finest = T;
        for (long long t = 2 * T; t <= 4 * T; t += T) {
            const double u = cut(t);
            if (u < 0.9 * time) { time = u; finest = t; }
        }
        cut(finest);
        T = finest;
    }
    int unit = 0;
    int& best = out.chunks;
    long long& priv = out.priv;
    best = 1; priv = 0; out.list = 0;
    out.cap.resize(nbun);
    for (int i = 0; i < nbun; ++i) {
        CbBundle& b = bundles[i];
        if (b.nK > best) best = b.nK;
        const int NS = b.FL == 32 ? 2 : 1;
        b.unit0 = unit;
        b.priv0 = priv;
        unit += nslots * (b.B >> 2) * NS;
        priv += (long long)b.nK * nslots * b.B * NS * 32;
        // an item lists its documents for its own later passes, so a block needs room for one chunk
        const int docs = (int)((nblk + b.nK - 1) / b.nK) * (2 * CB_LANE_THREADS);
        if (b.seq && b.npass > 1 && docs > out.list) out.list = docs;
        // documents one lane total can receive
        out.cap[i] = (unsigned int)(((nblk + b.nK - 1) / b.nK) * (2 * CB_LANE_THREADS / 32) + 1);
    }
    std::vector<int2>& items = out.items;
    std::vector<int> order(nbun);
    for (int i = 0; i < nbun; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return cost[x] / per[x] / bundles[x].nK > cost[y] / per[y] / bundles[y].nK; });
    for (int k = 0; k < best; ++k)
        for (int bi : order)
            if (k < bundles[bi].nK)
                for (int ps = 0; ps < per[bi]; ++ps) items.push_back(make_int2(bi | (ps << 16), k));
    return true;
}

// Device memory of the path for a tree of `depth` levels: the second copy of the store, the private tiles and the document
// lists of the level with the most.  0: no level takes it.
CB_API long long cb_lane_bytes(long long n, int G, const int* group_bins, const float* share, int depth, int grid, int lane_smem) {
    long long priv = 0, list = 0;
    bool any = false;
    for (int level = 0; level < depth; ++level) {
        CbLanePlan lp;
        if (!cb_lane_plan(lp, n, G, group_bins, share, level, grid, lane_smem, true, CB_LANE_SEQ_DOCS)) continue;
        any = true;
        priv = lp.priv > priv ? lp.priv : priv;
        list = lp.list > list ? lp.list : list;
    }
    return any ? 4 * (cb_lane_store_words(n, G) + priv) + 12 * list * grid : 0;
}
CB_API long long cb_fused_lane_bytes(CbFusedPlan* p, int depth) {
    const CbData& d = p->a.h.d;
    std::vector<int> gb(p->group_bins);
    if (gb.empty()) gb.assign(d.G, p->a.h.B);
    if (p->group_share.empty()) return 0;
    return cb_lane_bytes(d.n, d.G, gb.data(), p->group_share.data(), depth, p->sm_count, p->lane_smem);
}

// The same from sizes alone: document chunks and feature groups of every bundle; returns their number (0: the level takes the
// other path).
CB_API int cb_lane_plan_query(long long n, int G, const int* group_bins, const float* share, int level, int grid, int lane_smem,
                              int max_bundles, int* chunks, int* groups) {
    CbLanePlan lp;
    if (!cb_lane_plan(lp, n, G, group_bins, share, level, grid, lane_smem, true, CB_LANE_SEQ_DOCS)) return 0;
    for (int i = 0; i < (int)lp.bundles.size() && i < max_bundles; ++i) {
        chunks[i] = lp.bundles[i].nK; groups[i] = lp.bundles[i].gcnt;
    }
    return (int)lp.bundles.size();
}

// Feature-per-lane geometry of one level: grid size, 0 = take the other path, -1 = error.
static int cb_fused_lane_geometry(CbFusedPlan* p, int level, int* slots_per_pass, int* smem_bytes, int* threads, int* chunks,
                                  int* copies, int* bundle) {
    const CbData& d = p->a.h.d;
    const int grid = p->sm_count;                      // one block per SM
    std::vector<int> gb(p->group_bins);
    if (gb.empty()) gb.assign(d.G, p->a.h.B);
    std::vector<float> share(p->group_share);
    if (share.empty()) share.assign(d.G, 1.0f);
    cudaStream_t st = p->lane_stream;
    CbLanePlan lp;
    for (int round = 0;; ++round) {
        if (!cb_lane_plan(lp, d.n, d.G, gb.data(), share.data(), level, grid, p->lane_smem, p->a.h.work != nullptr, p->seq_docs)) return 0;
        int occ = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cb_level_fused_kernel<true>, CB_LANE_THREADS, lp.smem) != cudaSuccess) { cudaGetLastError(); return -1; }
        if (occ < 1) return 0;
        const int nbun = (int)lp.bundles.size();
        if (p->d_btab[level]) { cudaFree(p->d_btab[level]); p->d_btab[level] = nullptr; }
        if (p->d_items[level]) { cudaFree(p->d_items[level]); p->d_items[level] = nullptr; }
        if (p->d_cap[level]) { cudaFree(p->d_cap[level]); p->d_cap[level] = nullptr; }
        if (cudaMalloc(&p->d_btab[level], (size_t)nbun * sizeof(CbBundle)) != cudaSuccess ||
            cudaMalloc(&p->d_items[level], lp.items.size() * sizeof(int2)) != cudaSuccess ||
            cudaMalloc(&p->d_cap[level], (size_t)nbun * sizeof(unsigned int)) != cudaSuccess) { cudaGetLastError(); return -1; }
        cudaMemcpyAsync(p->d_btab[level], lp.bundles.data(), (size_t)nbun * sizeof(CbBundle), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(p->d_items[level], lp.items.data(), lp.items.size() * sizeof(int2), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(p->d_cap[level], lp.cap.data(), (size_t)nbun * sizeof(unsigned int), cudaMemcpyHostToDevice, st);
        cb_lane_cap_kernel<<<grid, CB_LANE_THREADS, 256 * 32 * 4, st>>>(d, p->lanes, p->ldom, p->d_btab[level], p->d_items[level],
                                                                        (int)lp.items.size(), p->d_cap[level]);
        if (cudaGetLastError() != cudaSuccess) return -1;
        // The shares come from a sample of the rows.  Where chunks are so large that a cell could receive more documents than
        // it may, the count decides: too many in one bin, and the bundle is cut finer.
        bool large = false, again = false;
        for (int i = 0; i < nbun; ++i) large = large || lp.cap[i] > lp.limit[i] / 32;
        if (!large || round == 3) break;
        std::vector<unsigned int> got(nbun);
        if (cudaMemcpyAsync(got.data(), p->d_cap[level], (size_t)nbun * sizeof(unsigned int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) { cudaGetLastError(); return -1; }
        for (int i = 0; i < nbun; ++i) {
            if (got[i] <= lp.limit[i] + lp.limit[i] / 8) continue;
            const float seen = (float)((double)got[i] * lp.bundles[i].nK / (double)d.n);
            for (int q = 0; q < lp.bundles[i].gcnt; ++q) {
                float& s = share[lp.bundles[i].g0 + q];
                if (seen > s) { s = seen; again = true; }
            }
        }
        if (!again) break;
    }
    p->n_btab[level] = (int)lp.bundles.size();
    p->n_items[level] = (int)lp.items.size();
    p->lane_level[level] = 1;
    p->lane_priv[level] = lp.priv;
    p->lane_list[level] = lp.list;
    *slots_per_pass = lp.bundles[0].spp;
    *smem_bytes = lp.smem;
    *threads = CB_LANE_THREADS;
    *chunks = lp.chunks;
    *copies = 1;
    *bundle = lp.bundles[0].gcnt;
    return grid;
}

CB_API int cb_fused_geometry(CbFusedPlan* p, int level, int* slots_per_pass, int* smem_bytes, int* threads, int* chunks,
                             int* copies, int* bundle) {
    const int nslots = level == 0 ? 1 : (1 << (level - 1));
    const bool narrow = p->a.h.statmax && p->a.h.S == 2 && p->a.h.narrow;
    const int G = p->a.h.d.G;
    const long long n = p->a.h.d.n;
    if (level < CB_MAX_LEVELS) {
        p->lane_level[level] = 0;
        if (p->lanes && narrow) {
            const int grid = cb_fused_lane_geometry(p, level, slots_per_pass, smem_bytes, threads, chunks, copies, bundle);
            if (grid != 0) return grid > 0 ? grid : 0;
        }
    }
    int thr = p->threads, spp = nslots, C = 1, gpc = 0, smem = 0;
    std::vector<CbBundle> bundles;
    if (narrow && p->max_bundle > 0) {
        // Bundled single-cell path: a block accumulates the groups of one bundle at once.  Tile of a bundle =
        // slots * groups * 8 * B * C ints with B the padded bins of its widest feature, ring = warps * 64 * (3 + groups)
        // words.  Consecutive groups of similar width (within a factor of two) form a run; a run is cut into the fewest
        // bundles whose tiles hold every slot, evened out (7 groups as 4 + 3 rather than 5 + 2); when not even one group
        // holds all slots the group takes several passes over the slots.  Then the cells are replicated while room is left.
        // One 1024-thread block per SM: measured a few percent faster than two 512-thread blocks at every level (one
        // tile instead of two leaves room for wider bundles and replicas) and it balances better.
        const bool skip = p->a.h.domw != nullptr;       // dominant-bin skipping: 256 bytes of slot totals per slot
        const int budget = p->max_smem;
        thr = 1024;
        auto gb = [&](int g) { return p->group_bins.empty() ? p->a.h.B : p->group_bins[g]; };
        auto need = [&](int slots, int gc, int Bb, int Cc) {
            return slots * gc * 8 * Bb * 4 * Cc + (thr / 32) * 64 * (3 + gc) * 4 + 16 + (skip ? slots * 256 : 0);
        };
        int max_copies = p->max_copies;
        if (const char* e = getenv("CB200_MAX_COPIES")) { const int v = atoi(e); if (v == 1 || v == 2 || v == 4 || v == 8) max_copies = v; }
        int g = 0;
        while (g < G) {
            int lo_b = gb(g), hi_b = gb(g), run = 1;
            while (g + run < G) {
                const int b2 = gb(g + run);
                const int lo2 = b2 < lo_b ? b2 : lo_b, hi2 = b2 > hi_b ? b2 : hi_b;
                if (hi2 > 2 * lo2) break;
                lo_b = lo2; hi_b = hi2; ++run;
            }
            int fitg = 0;
            while (fitg < run && fitg < p->max_bundle && need(nslots, fitg + 1, hi_b, 1) <= budget) ++fitg;
            if (fitg < 1) {
                for (int q = 0; q < run; ++q) {
                    const int Bb = gb(g + q);
                    int s1 = (budget - need(0, 1, Bb, 1)) / (8 * Bb * 4 + (skip ? 256 : 0));
                    if (s1 < 1) return 0;
                    const int np = (nslots + s1 - 1) / s1;
                    s1 = (nslots + np - 1) / np;
                    bundles.push_back(CbBundle{g + q, 1, Bb, 1, s1, np, 1});
                }
            } else {
                const int nbr = (run + fitg - 1) / fitg;
                int at = g;
                for (int q = 0; q < nbr; ++q) {
                    const int cnt = (run - (at - g) + (nbr - q) - 1) / (nbr - q);
                    int Bb = 4;
                    for (int k = 0; k < cnt; ++k) Bb = gb(at + k) > Bb ? gb(at + k) : Bb;
                    bundles.push_back(CbBundle{at, cnt, Bb, 1, nslots, 1, 1});
                    at += cnt;
                }
            }
            g += run;
        }
        // Replicas: columns of few bins put many lanes of a warp on the same cell whatever the data look like (32 lanes
        // over 16 bins), so their bundles take up to 8 replicas; measured on 4.5M x 52 columns (13 floats, 39 CTR columns
        // of 16 bins), depth 8: 7.4 ms per tree against 9.8 ms with 2 replicas.
        int narrow_copies = 8;
        if (const char* e = getenv("CB200_NARROW_COPIES")) { const int v = atoi(e); if (v == 1 || v == 2 || v == 4 || v == 8) narrow_copies = v; }
        for (CbBundle& b : bundles) {
            const int mc = b.B <= 32 ? (narrow_copies > max_copies ? narrow_copies : max_copies) : max_copies;
            while (b.C < mc && need(b.spp, b.gcnt, b.B, 2 * b.C) <= budget) b.C *= 2;
            const int nb_ = need(b.spp, b.gcnt, b.B, b.C);
            if (nb_ > smem) smem = nb_;
        }
        spp = bundles[0].spp; C = bundles[0].C; gpc = bundles[0].gcnt;
    } else {
        const bool narrow_cells = p->a.h.statmax && p->a.h.narrow;      // one int32 per cell, any number of statistics
        const int per_slot = p->a.h.S * 4 * p->a.h.B * 4 * ((p->a.h.statmax && !narrow_cells) ? 2 : 1);
        const bool ring = p->a.h.statmax && p->a.h.S == 2;      // per-warp compaction rings (16 bytes x 64 entries)
        int ring_bytes = ring ? (thr / 32) * 64 * 16 + 16 : 0;
        int budget = p->max_smem - ring_bytes;
        if (spp * per_slot > budget / 2) {
            // one 1024-thread block per SM when the tile needs more than half of the shared memory
            thr = 1024;
            ring_bytes = ring ? (thr / 32) * 64 * 16 + 16 : 0;
            budget = p->max_smem - ring_bytes;
        }
        if (spp * per_slot > budget) spp = budget / per_slot;
        if (spp < 1) return 0;
        // replicate the cells while two blocks per SM still fit (fewer bank / address collisions per atomic)
        if (ring && thr == p->threads) {
            while (C < 8 && 2 * (spp * per_slot * (C * 2) + ring_bytes) <= p->max_smem) C *= 2;
        }
        smem = spp * per_slot * C + ring_bytes;
    }
    // the score phase reuses the tile as scratch: CB_SCORE_WARP_FLOATS floats per scoring warp, at least 8 warps' worth
    // (a small tile -- few bins, one slot -- would otherwise leave it without a single warp)
    {
        const int want = (thr / 32 < 8 ? thr / 32 : 8) * CB_SCORE_WARP_FLOATS * 4;
        if (smem < want) smem = want;
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cb_level_fused_kernel<false>, thr, smem) != cudaSuccess) { cudaGetLastError(); return 0; }
    if (occ < 1) return 0;
    if (occ > 4) occ = 4;
    const int grid = occ * p->sm_count;
    // document chunks per work unit (group or bundle): at least what the grid offers and what the 2^19-documents-per-
    // tile cap needs; among a few candidates take the one that fills the last round of blocks best
    const int by_docs = (int)((n + (1 << 19) - 1) >> 19);
    int best = 1;
    if (bundles.empty()) {
        const int units = G;
        const int by_grid = grid >= units ? grid / units : 1;
        const int lo = by_grid > by_docs ? by_grid : by_docs;
        best = lo;
        double best_eff = 0.0;
        for (int k = lo; k < lo + 8; ++k) {
            const long long items = (long long)units * k;
            const long long rounds = (items + grid - 1) / grid;
            const double eff = (double)items / (double)(rounds * grid);
            if (eff > best_eff + 0.02) { best_eff = eff; best = k; }
        }
    } else {
        if (level >= CB_MAX_LEVELS) return 0;
        // Every bundle is cut into its own number of document chunks so that all work items take about the same time
        // and their number is a whole multiple of the grid.  Cost of an item per document it streams: a fixed part (leaf
        // index, two statistics, compaction) worth 2.8 groups plus one unit per group of the bundle (measured on 4.5M
        // x 52 columns, depth 8: a one-group item took 0.49 of the time of a five-group item over the same documents).
        const int nbun = (int)bundles.size();
        std::vector<double> cost(nbun);
        std::vector<int> nk(nbun);
        double W = 0.0;
        long long min_items = 0;
        for (int i = 0; i < nbun; ++i) {
            cost[i] = 2.8 + bundles[i].gcnt;
            W += cost[i] * bundles[i].npass;
            min_items += (long long)bundles[i].npass * by_docs;
        }
        // bundles of different shapes: the cost model is rough (bin collisions depend on the data), so the work is cut
        // into two rounds of items handed out by a counter, which bounds the imbalance by half an item's time (measured
        // on the same data: 7.2 ms per tree with one round, 7.1 with two, 7.8 with four -- every item zeroes and dumps a tile)
        bool mixed = false;
        for (int i = 1; i < nbun; ++i)
            if (bundles[i].B != bundles[0].B || bundles[i].npass != bundles[0].npass || bundles[i].C != bundles[0].C) mixed = true;
        int rounds = (mixed && p->a.h.work) ? 2 : 1;
        if (const char* e = getenv("CB200_ITEM_ROUNDS")) { const int v = atoi(e); if (v >= 1 && v <= 16) rounds = v; }
        long long T = (long long)grid * rounds;
        while (T < min_items) T += grid;
        long long used = 0;
        for (int i = 0; i < nbun; ++i) {
            int k = (int)((double)T * cost[i] / W);
            if (k < by_docs) k = by_docs;
            if (k < 1) k = 1;
            nk[i] = k;
            used += (long long)k * bundles[i].npass;
        }
        for (;;) {
            int pick = -1;
            double worst = 0.0;
            for (int i = 0; i < nbun; ++i) {
                if (used + bundles[i].npass > T) continue;
                const double t = cost[i] / nk[i];
                if (t > worst) { worst = t; pick = i; }
            }
            if (pick < 0) break;
            ++nk[pick];
            used += bundles[pick].npass;
        }
        // work list: chunk-major, so that blocks running side by side stream the same documents (their leaf indices and
        // statistics then come from L2); the wider bundles of a chunk first
        std::vector<int> order(nbun);
        for (int i = 0; i < nbun; ++i) order[i] = i;
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] / nk[x] > cost[y] / nk[y]; });
        std::vector<int2> items;
        std::vector<int> gchunks(G, 1);
        for (int i = 0; i < nbun; ++i) {
            bundles[i].nK = nk[i];
            if (nk[i] > best) best = nk[i];
            for (int q = 0; q < bundles[i].gcnt; ++q) gchunks[bundles[i].g0 + q] = nk[i];
        }
        items.reserve((size_t)used);
        for (int k = 0; k < best; ++k)
            for (int bi : order)
                if (k < nk[bi])
                    for (int ps = 0; ps < bundles[bi].npass; ++ps) items.push_back(make_int2(bi | (ps << 16), k));
        if (p->d_btab[level]) { cudaFree(p->d_btab[level]); p->d_btab[level] = nullptr; }
        if (p->d_items[level]) { cudaFree(p->d_items[level]); p->d_items[level] = nullptr; }
        if (p->d_gchunks[level]) { cudaFree(p->d_gchunks[level]); p->d_gchunks[level] = nullptr; }
        if (cudaMalloc(&p->d_btab[level], bundles.size() * sizeof(CbBundle)) != cudaSuccess ||
            cudaMalloc(&p->d_items[level], items.size() * sizeof(int2)) != cudaSuccess ||
            cudaMalloc(&p->d_gchunks[level], (size_t)G * sizeof(int)) != cudaSuccess) { cudaGetLastError(); return 0; }
        cudaMemcpy(p->d_btab[level], bundles.data(), bundles.size() * sizeof(CbBundle), cudaMemcpyHostToDevice);
        cudaMemcpy(p->d_items[level], items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice);
        cudaMemcpy(p->d_gchunks[level], gchunks.data(), (size_t)G * sizeof(int), cudaMemcpyHostToDevice);
        p->n_btab[level] = nbun;
        p->n_items[level] = (int)items.size();
        p->single_pass_bundle[level] = (nbun == 1 && bundles[0].npass == 1 && bundles[0].gcnt >= G) ? 1 : 0;
    }
    *slots_per_pass = spp;
    *smem_bytes = smem;
    *threads = thr;
    *chunks = best;
    *copies = C;
    *bundle = gpc;
    return grid;
}

CB_API void cb_fused_set_priv(CbFusedPlan* p, float* priv, const float* statmax) { p->a.h.priv = priv; p->a.h.statmax = statmax; }

CB_API int cb_fused_launch(CbFusedPlan* p, int level, float* hprev, float* hcur, const unsigned int* mask_in,
                           unsigned int* mask_out, int grid, int slots_per_pass, int smem_bytes, int threads,
                           int chunks, int copies, int bundle, cudaStream_t st) {
    CbFusedArgs a = p->a;
    a.h.nK = chunks; a.h.copies = copies; a.h.bundle = bundle;
    a.h.level = level; a.h.small_mask = mask_in; a.h.slots_per_pass = slots_per_pass;
    a.s.level = level; a.s.small_mask = mask_in; a.s.hprev = hprev; a.s.hcur = hcur;
    a.mask_out = mask_out;
    a.smem_floats = smem_bytes / 4;
    // the bundled histogram pass can apply the previous level's split itself (see CbHistArgs::prev_split)
    // ... when one bundle holds every feature group: then the split feature's bin word is already in registers and each
    // document is streamed by exactly one block.  With several bundles each of them would have to fetch that word as
    // well, which costs more than the separate pass (measured at 10.5M x 28, level 5, 4 bundles: +86 us against 18 us).
    const bool table = bundle > 0 && level < CB_MAX_LEVELS && p->d_btab[level] != nullptr;
    const bool lanes = level < CB_MAX_LEVELS && p->lane_level[level];
    a.h.lanes = lanes ? p->lanes : nullptr; a.h.ldom = p->ldom; a.h.bcap = lanes ? p->d_cap[level] : nullptr;
    a.h.list_len = lanes ? p->lane_list[level] : 0;
    a.h.nbundles = table ? p->n_btab[level] : 0;
    a.h.btab = table ? p->d_btab[level] : nullptr;
    a.h.bitems = table ? p->d_items[level] : nullptr;
    a.h.nbitems = table ? p->n_items[level] : 0;
    a.h.gchunks = table ? p->d_gchunks[level] : nullptr;
    const bool whole = table ? p->single_pass_bundle[level] != 0 : bundle >= a.h.d.G;
    a.fuse_leaf = (level > 0 && whole && a.h.statmax && a.h.S == 2 && a.h.narrow && p->fuse_leaf_update) ? 1 : 0;
    if (lanes) a.fuse_leaf = 1;            // that path always reads the split column next to the leaf index
    a.h.prev_splits = a.fuse_leaf ? a.splits : nullptr;
    void* args[] = {&a};
    void* kernel = lanes ? (void*)cb_level_fused_kernel<true> : (void*)cb_level_fused_kernel<false>;
    cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args,
                                                (size_t)smem_bytes, st);
    return (int)e;
}
