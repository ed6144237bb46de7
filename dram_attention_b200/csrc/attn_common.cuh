// Pieces shared by the decode-attention kernels (float32 on CUDA cores, 16-bit
// types on tensor cores): launch geometry, the parameter block, the unit plan and
// the final merge of the per-CTA partials.
#pragma once

#include "da_common.cuh"

namespace da {

constexpr int kAttnWarps = 12;         // warps per CTA (16-bit types): one CTA fills an SM
constexpr int kUnitTokens = 16;
constexpr int kCounterBytes = 1024;
constexpr int kAttnSms = 148;
constexpr int kAttnMaxSplits = 148;
constexpr int kAttnMaxRows = 16;       // query rows (tokens x GQA group) of one KV head that the workspaces are sized for
constexpr int kAttnWideRows = 32;      // ... and the most that a launch takes (16-bit types)
constexpr int kRoundUnits = 32;        // units a warp plans at a time (one per lane)

// CTAs per head ("splits").  Every CTA of every launch fills an SM on its own (12 warps, nearly all of the shared
// memory): the loop of a warp is a chain of dependent instructions, so an SM wants all the warps it can hold, and one
// large CTA leaves a third of the partial rows of three small ones to the final merge, which adds them with three
// times the threads.  The merge ends every step: with 4-warp CTAs it took 3.2 to 5.6 us (one batch of loads is
// a round trip of 0.9 us, and there were up to six), with 12-warp CTAs 1.9 to 2.6 us.
//
// Phase 1 runs beside the selection kernels, whose CTAs need a whole SM each: it has at most 116 CTAs, so that
// wherever the hardware places them 32 of the 148 SMs stay empty.  Phase 2 covers the few slots the LRU update
// could evict, on what phase 1 and the update's CTAs (one per head) leave.  The caps on CTAs per head keep the merge
// short: of 4 query rows of 128 channels a thread has at most 16 partials of phase 1 (two batches) and two of phase 2, of 8
// rows (one group of threads instead of three) of three heads 38 and 6.  The single launch also keeps at least two units
// per warp.
constexpr int kAttnPhase1Ctas = 116;
constexpr int kAttnPhase1MaxPerHead = 48;
constexpr int kAttnPhase2MaxPerHead = 6;

__host__ __device__ inline int attn_splits(int n_kv_heads) {
    const int s = kAttnSms / n_kv_heads;
    return s < 1 ? 1 : s;
}

// what the workspace of the single launch has room for (part of the ABI; at least attn_splits)
__host__ __device__ inline int attn_reserved_splits(int n_kv_heads) {
    const int s = 3 * kAttnSms / n_kv_heads;
    return s > kAttnMaxSplits ? kAttnMaxSplits : (s < 1 ? 1 : s);
}

__host__ __device__ inline int attn_splits_phase1(int n_kv_heads) {
    int s = kAttnPhase1Ctas / n_kv_heads;
    if (s > kAttnPhase1MaxPerHead) s = kAttnPhase1MaxPerHead;
    if (s < 1) s = 1;
    return s;
}

__host__ __device__ inline int attn_splits_phase2(int n_kv_heads) {
    int s = (kAttnSms - n_kv_heads * (attn_splits_phase1(n_kv_heads) + 1)) / n_kv_heads;
    if (s > kAttnPhase2MaxPerHead) s = kAttnPhase2MaxPerHead;
    if (s < 1) s = 1;
    return s;
}

constexpr int kAttnMaxPeers = 16;

struct AttnParams {
    // KV-head sharding: the CTA that merges a head also sends the head's output rows to every rank's gather
    // buffer (see gather.cu for the layout and the tag); null when the caller gathers itself
    // (the pointers travel in the kernel's parameters, so that the store loop at the end of a merge has no
    // dependent load in it; peer_world == 0: nothing is sent)
    uint2 *peer_buf[kAttnMaxPeers];
    const int32_t *peer_seq;
    int peer_rank, peer_world, peer_words;   // words (4 bytes of payload each) per rank
    const unsigned char *q;        // (s_total, n_kv_heads * rep, D)
    const unsigned char *prefix;
    long long prefix_head_stride;  // elements
    int n_prefix_tokens;
    unsigned char *local_k, *local_v;
    long long local_tok_stride, local_head_stride;  // elements
    int local_capacity;
    const unsigned char *new_k, *new_v;   // (s_total, n_kv_heads, D)
    const int32_t *start_pos_dev;
    int start_pos_host;
    int dram_tokens;
    unsigned char *out;            // (s_total, n_kv_heads * rep, D)
    float *lse_out;                // (s_total, n_kv_heads * rep) or null
    float *partials;
    unsigned int *counters;
    int32_t *status;
    float scale_log2;
    // optional: pages that da_lru_update just assigned to slots are read from DRAM (pinned
    // host memory) by the warp that owns the unit, and written through to the slot
    const unsigned char *dram;       // (n_kv_heads, n_dram_pages, page_tokens, 2, D) or null
    long long dram_head_stride;      // elements
    const int32_t *slot_source;      // (n_kv_heads, n_slots): DRAM page to read instead, or -1
    int n_slots;
    int page_tokens;                 // multiple of 16 when slot_source is set
    // optional: two launches per step.  Phase 1 attends over the local window and the slots
    // outside the eviction front (it runs beside selection and LRU update); phase 2 attends over
    // the front after the update; the CTA of either launch that finishes last merges both.  The
    // front is order[h][0 .. n_evictable[h]) of the copy flip[h] names.  redo[h] != 0 (set by the
    // LRU update when it had to evict a slot outside the front): phase 2 covers the whole head
    // and the merge leaves out the rows of phase 1.
    int phase;                       // 0: one launch over everything
    const int32_t *order;            // [2][n_kv_heads][n_slots]
    const int32_t *n_evictable;      // [2][n_kv_heads]
    int32_t *flip;                   // [n_kv_heads]
    const int32_t *redo;             // [n_kv_heads]
    int part_rows;                   // partials per head in the workspace (two launches: one more than CTAs, if it has room)
    int part_offset;                 // first row this launch writes
    int ticket_target;               // CTAs of a head that take a ticket before the merge
    int splits1;                     // rows of phase 1 (first in the workspace)
    int n_kv_heads;
    int rep;
    int head_dim;
    // query tokens: the call has s_total of them (appended at consecutive positions); this
    // launch computes tokens [q_tok0, q_tok0 + n_q), i.e. n_q * rep query rows per KV head
    int s_total, q_tok0, n_q;
};

// Units of a head this launch covers.
struct LaunchUnits {
    int units_slots;      // units from the slot table
    int units_local;      // units from the local window
    const int32_t *order; // slot order to walk (null: slot-table tokens in place)
    int ups;              // units per slot page
};

// The words of the eviction queue's state a launch plans from: read together, early (see the kernel body).
struct FrontWords {
    int flip, nf0, nf1;
};
__device__ __forceinline__ FrontWords load_front(const AttnParams &p, int h) {
    FrontWords f = {0, 0, 0};
    if (p.phase != 0) {
        f.nf0 = p.n_evictable[h];
        f.nf1 = p.n_evictable[p.n_kv_heads + h];
        f.flip = p.flip[h];
    }
    return f;
}

// `redo`: the LRU update had to evict beyond the front (second launch only).
__device__ __forceinline__ LaunchUnits launch_units(const AttnParams &p, int h, int n_local, bool redo,
                                                    const FrontWords &fw) {
    LaunchUnits lu;
    lu.order = nullptr;
    lu.ups = p.phase != 0 ? p.page_tokens / kUnitTokens : 1;
    bool local = true;
    if (p.phase == 0) {
        lu.units_slots = (p.n_prefix_tokens + kUnitTokens - 1) / kUnitTokens;
    } else {
        // (the front sizes of both queue copies were read beside the flip word, not after it)
        const int cur = fw.flip & 1;
        const int32_t *order = p.order + ((size_t)cur * p.n_kv_heads + h) * p.n_slots;
        const int n_ev = min(max(cur ? fw.nf1 : fw.nf0, 0), p.n_slots);
        if (p.phase == 1) {
            lu.units_slots = (p.n_slots - n_ev) * lu.ups;
            lu.order = order;
        } else if (redo) {
            lu.units_slots = p.n_slots * lu.ups;   // the whole head, slots in place
        } else {
            lu.units_slots = n_ev * lu.ups;
            lu.order = order;
            local = false;
        }
    }
    lu.units_local = local ? (n_local + kUnitTokens - 1) / kUnitTokens : 0;
    return lu;
}

// One entry of a warp's plan table (shared memory, in the order the warp visits its units):
//   x, y  global address of the unit's first token (slot table, or the DRAM page to read instead)
//   z     slot-table units: first token inside the head's slot table (>= 0);
//         local-window units: -1 - first token of the unit in the local window
//   w     DRAM page the unit is read from (it is then written through to its slot), or -1
// A round covers the warp's units at positions round * 32 .. round * 32 + n_round - 1; lane i plans
// unit i.  Planning has two halves, so that the second launch of a step can do the first before
// the LRU update has finished: plan_base() needs only the eviction queue as it was BEFORE the
// update, plan_commit() the marks the update leaves (which slots must be read from DRAM).

// Place in the eviction queue of the k-th slot a launch walks: phase 2 from the front, phase 1 from the back, so that
// neither has to know how long the front is before it reads the queue.
__device__ __forceinline__ int queue_place(const AttnParams &p, int k) { return p.phase == 1 ? p.n_slots - 1 - k : k; }

// The slots of the first round's units out of both copies of the queue, read before it is known which one is current.
struct FirstSlots {
    int copy0, copy1;
};
__device__ __forceinline__ FirstSlots load_first_slots(const AttnParams &p, int h, int worker, int n_workers, int lane) {
    FirstSlots f = {0, 0};
    if (p.phase != 0) {
        const int at = queue_place(p, (worker + lane * n_workers) / (p.page_tokens / kUnitTokens));
        if (at >= 0 && at < p.n_slots) {
            f.copy0 = p.order[(size_t)h * p.n_slots + at];
            f.copy1 = p.order[((size_t)p.n_kv_heads + h) * p.n_slots + at];
        }
    }
    return f;
}

// First slot-table token of lane's unit of this round, or -1 (a local-window unit, or none).  `first` (round 0): the
// slot of that unit in the queue.
__device__ __forceinline__ int plan_base(const AttnParams &p, const LaunchUnits &lu, int worker, int n_workers,
                                         int lane, int round, int total_my, int first = 0) {
    const int n_round = min(kRoundUnits, total_my - round * kRoundUnits);
    const int u = worker + (round * kRoundUnits + lane) * n_workers;
    int base = -1;
    if (lane < n_round && u < lu.units_slots) {
        base = u * kUnitTokens;
        if (lu.order) {
            int slot = round == 0 ? first : lu.order[queue_place(p, u / lu.ups)];
            slot = min(max(slot, 0), p.n_slots - 1);
            base = slot * p.page_tokens + (u % lu.ups) * kUnitTokens;
        }
    }
    return base;
}

// DRAM page lane's unit has to be read from, or -1.
__device__ __forceinline__ int plan_source(const AttnParams &p, int h, int base) {
    if (base < 0 || !p.slot_source || p.phase == 1) return -1;
    return p.slot_source[(size_t)h * p.n_slots + base / p.page_tokens];
}

// Writes the round's table.  Units that have to come from DRAM are visited first, so that their
// host-link latency overlaps everything else the warp does.  Returns n_round.
__device__ __forceinline__ int plan_commit(const AttnParams &p, const LaunchUnits &lu, int h, int worker,
                                           int n_workers, int lane, int round, int total_my, int base, int src,
                                           uint4 *tab, size_t elem_bytes) {
    const int n_round = min(kRoundUnits, total_my - round * kRoundUnits);
    const int u = worker + (round * kRoundUnits + lane) * n_workers;
    const bool valid = lane < n_round;
    const unsigned fresh = __ballot_sync(DA_FULL_MASK, valid && src >= 0);
    if (valid) {
        const int before = __popc(fresh & ((1u << lane) - 1));
        const int pos = src >= 0 ? before : __popc(fresh) + (lane - before);
        uint4 e;
        unsigned long long addr = 0;
        if (base >= 0) {
            const size_t tok_bytes = (size_t)2 * p.head_dim * elem_bytes;
            const unsigned char *a =
                src < 0 ? p.prefix + (size_t)h * p.prefix_head_stride * elem_bytes + (size_t)base * tok_bytes
                        : p.dram + (size_t)h * p.dram_head_stride * elem_bytes +
                              ((size_t)src * p.page_tokens + base % p.page_tokens) * tok_bytes;
            addr = (unsigned long long)a;
            e.z = (unsigned)base;
        } else {
            e.z = (unsigned)(-1 - (u - lu.units_slots) * kUnitTokens);
        }
        e.x = (unsigned)(addr & 0xffffffffull);
        e.y = (unsigned)(addr >> 32);
        e.w = (unsigned)src;
        tab[pos] = e;
    }
    __syncwarp();
    return n_round;
}

// Floats per partial row: acc[D], max, l, padded to a multiple of 4 so that rows can
// be read with 128-bit loads.
template <int D> struct PartialRow { static constexpr int kWidth = D + 4; };

// Running softmax merge of (max, l, four accumulator columns); log2 domain.  Every product and sum is spelled out, so that
// the same operands give the same bits wherever this is compiled in.
struct MergeAcc {
    float m, l;
    float4 a;
};
__device__ __forceinline__ MergeAcc merge_nothing() { return {-INFINITY, 0.f, make_float4(0.f, 0.f, 0.f, 0.f)}; }
__device__ __forceinline__ void merge_into(MergeAcc &x, float m, float l, const float4 &v) {
    const float mn = fmaxf(x.m, m);
    const float ms = (mn == -INFINITY) ? 0.f : mn;
    const float wx = fast_exp2(x.m - ms), wv = fast_exp2(m - ms);
    x.m = mn;
    x.l = fmaf(x.l, wx, __fmul_rn(l, wv));
    x.a.x = fmaf(x.a.x, wx, __fmul_rn(v.x, wv));
    x.a.y = fmaf(x.a.y, wx, __fmul_rn(v.y, wv));
    x.a.z = fmaf(x.a.z, wx, __fmul_rn(v.z, wv));
    x.a.w = fmaf(x.a.w, wx, __fmul_rn(v.w, wv));
}

// What a CTA adds up once its ticket is taken: nothing, phase 1's partials into one (phase 2 is still at work), or the
// head's output from all partials, or from phase 2's and the one that phase 1's were merged into.
enum { kMergeNothing, kMergePhase1, kMergeAll, kMergeRest };

// Partials of every `step`-th CTA from s0 on, requested together (the last one again for places behind the end).
template <int BATCH> struct PartialBatch {
    float4 v[BATCH];
    float2 w[BATCH];
    __device__ __forceinline__ void request(const float *col, const float *ml, size_t cta_stride, int s0, int step, int hi) {
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int s = min(s0 + i * step, hi - 1);
            v[i] = __ldcg(reinterpret_cast<const float4 *>(col + (size_t)s * cta_stride));
            w[i] = __ldcg(reinterpret_cast<const float2 *>(ml + (size_t)s * cta_stride));
        }
    }
    // The batch's own maximum first, so that its exponentials do not wait for one another.
    __device__ __forceinline__ void fold_into(MergeAcc &x, int s0, int step, int hi, bool skip) {
        float mb = x.m;
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            if (skip || s0 + i * step >= hi) w[i].x = -INFINITY;
            mb = fmaxf(mb, w[i].x);
        }
        const float ms = (mb == -INFINITY) ? 0.f : mb;
        const float wx = fast_exp2(x.m - ms);
        x.m = mb;
        x.l = __fmul_rn(x.l, wx);
        x.a.x = __fmul_rn(x.a.x, wx);
        x.a.y = __fmul_rn(x.a.y, wx);
        x.a.z = __fmul_rn(x.a.z, wx);
        x.a.w = __fmul_rn(x.a.w, wx);
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            if (w[i].x == -INFINITY) continue;   // (a CTA without units: its rows are zeros)
            const float wv = fast_exp2(w[i].x - ms);
            x.l = fmaf(w[i].y, wv, x.l);
            x.a.x = fmaf(v[i].x, wv, x.a.x);
            x.a.y = fmaf(v[i].y, wv, x.a.y);
            x.a.z = fmaf(v[i].z, wv, x.a.z);
            x.a.w = fmaf(v[i].w, wv, x.a.w);
        }
    }
};

template <int BATCH>
__device__ __forceinline__ void fold_partials(MergeAcc &x, const float *col, const float *ml, size_t cta_stride, int lo, int step,
                                              int hi, bool skip) {
    for (int s0 = lo; s0 < hi; s0 += step * BATCH) {
        PartialBatch<BATCH> b;
        b.request(col, ml, cta_stride, s0, step, hi);
        b.fold_into(x, s0, step, hi, skip);
    }
}

// Merge of the per-CTA partials of one head by one CTA of THREADS threads.  A CTA's partial = `rows` rows
// of (acc[D] already weighted to the row's max, max, l); the partials of consecutive CTAs are contiguous in the
// workspace.  It is on the critical path of every step and bound by latency alone, so it is one round trip to
// L2 wherever the registers allow: a thread owns four columns of a row for every G-th CTA (G = how many
// times the row-columns fit into the CTA), requests BATCH partials together with their (max, l) pairs, and
// folds them in registers; the G groups meet in shared memory.  (Staging the rows in shared memory in two
// halves took one round trip per half: 3.7 us for 22 partials of 4 rows, 5.9 us for 55.)
// With two launches phase 1's partials and phase 2's are always added up apart and the two sums put together at the
// end: the output's bits do not depend on which launch was through first, i.e. on whether phase 1's own last CTA has
// done its part already (kMergeRest) or not (kMergeAll).  A head that phase 2 redid leaves phase 1's partials out.
// With kMergeBatchFew partials per thread or less a short batch: the long one asks for the last partial again and
// again (four resident 13K layers 78.3 / 74.0 us).  With two launches the long one is no longer than 9, and one piece of
// code serves every case: it runs once or twice per head and layer, on an SM that seldom has it at hand, so its size
// counts as much as another round trip.  us for three odd 77K layers (38 partials of 8 rows in phase 1) / four 128K layers:
// long batch of 18, 12, 9: 84 / 167, 83 / 166, 81.5 / 165.4; with every case's code apart 85 / 166; a batch of 9 in kernels
// that hold no other launch's merge 77 / 165.8 (and four resident 13K layers 73.8 instead of 75.2).
constexpr int kMergeBatch = 18;
constexpr int kMergeBatchTwo = 9;
constexpr int kMergeBatchFew = 6;

// TWO: the kernel is one of two launches.
template <typename T, int D, int THREADS, int BATCH, bool TWO>
__device__ __forceinline__ void merge_partials_by(const AttnParams &p, int h, int rows, int todo, unsigned char *smem) {
    const bool with1 = !TWO || todo != kMergeRest;        // add up phase 1's (a single launch's) partials
    const bool with2 = TWO && todo != kMergePhase1;       // ... phase 2's, requested ahead of a short batch of phase 1's
    constexpr bool ahead2 = TWO && BATCH <= kMergeBatchFew;
    constexpr int PW = PartialRow<D>::kWidth;
    constexpr int VPR = D / 4;          // float4 per accumulator row
    const int tid = threadIdx.x;
    const int32_t peer_step = p.peer_world > 0 ? __ldcg(p.peer_seq) : 0;   // (needed at the very end: read now)
    const bool skip = with2 && __ldcg(p.redo + h) != 0;
    const int n1 = TWO ? p.splits1 : p.ticket_target, n = p.ticket_target;
    const float *hp = p.partials + ((size_t)h * p.part_rows * rows) * PW;
    float *merged1 = p.partials + ((size_t)(h * p.part_rows + n) * rows) * PW;   // phase 1's, once merged
    const size_t cta_stride = (size_t)rows * PW;
    const int items = rows * VPR;
    const int groups = max(THREADS / items, 1);
    float4 *sh_a = reinterpret_cast<float4 *>(smem);                    // [2][groups - 1][items]
    float2 *sh_ml = reinterpret_cast<float2 *>(sh_a + 2 * THREADS);     // [2][groups - 1][items]
    const int g = groups > 1 ? tid / items : 0;

    for (int e0 = 0; e0 < items; e0 += THREADS) {
        const int e = groups > 1 ? tid % items : e0 + tid;
        const bool mine = e < items && g < groups;
        const size_t at = (size_t)(e / VPR) * PW + 4 * (e % VPR), at_ml = (size_t)(e / VPR) * PW + D;
        MergeAcc x1 = merge_nothing(), x2 = merge_nothing();
        if (mine) {
            const float *col = hp + at, *ml = hp + at_ml;
            PartialBatch<ahead2 ? kMergeBatchFew : 1> b2;
            if (ahead2 && with2) b2.request(col, ml, cta_stride, n1 + g, groups, n);
            if (with1) {
                fold_partials<BATCH>(x1, col, ml, cta_stride, g, groups, n1, skip);
            } else if (g == 0) {
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(merged1 + at));   // (set out before `skip` is there)
                const float2 w = __ldcg(reinterpret_cast<const float2 *>(merged1 + at_ml));
                if (!skip) x1 = {w.x, w.y, v};
            }
            if (ahead2 && with2) b2.fold_into(x2, n1 + g, groups, n, false);
            if (with2)
                fold_partials<kMergeBatchFew>(x2, col, ml, cta_stride, n1 + g + (ahead2 ? groups * kMergeBatchFew : 0), groups, n, false);
        }
        if (groups > 1) {
            const int half = (groups - 1) * items;
            if (mine && g > 0) {
                const int at_sh = (g - 1) * items + e;
                if (with1) {
                    sh_a[at_sh] = x1.a;
                    sh_ml[at_sh] = make_float2(x1.m, x1.l);
                }
                if (with2) {
                    sh_a[half + at_sh] = x2.a;
                    sh_ml[half + at_sh] = make_float2(x2.m, x2.l);
                }
            }
            __syncthreads();
            if (mine && g == 0) {
                for (int k = 0; k < groups - 1; ++k) {
                    const int at_sh = k * items + e;
                    if (with1) merge_into(x1, sh_ml[at_sh].x, sh_ml[at_sh].y, sh_a[at_sh]);
                    if (with2) merge_into(x2, sh_ml[half + at_sh].x, sh_ml[half + at_sh].y, sh_a[half + at_sh]);
                }
            }
        }
        if (!mine || g != 0) continue;
        const int r = e / VPR, c4 = e % VPR;
        if (TWO && todo == kMergePhase1) {
            *reinterpret_cast<float4 *>(merged1 + at) = x1.a;
            if (c4 == 0) *reinterpret_cast<float2 *>(merged1 + at_ml) = make_float2(x1.m, x1.l);
            continue;
        }
        if (with2) {
            merge_into(x2, x1.m, x1.l, x1.a);
            x1 = x2;
        }
        const float inv = x1.l > 0.f ? 1.f / x1.l : 0.f;
        // row r = (query token, head of the group)
        const int tok = p.q_tok0 + r / p.rep;
        const size_t orow = (size_t)tok * p.n_kv_heads * p.rep + (size_t)h * p.rep + r % p.rep;
        union { T t[4]; uint32_t w[sizeof(T)]; } o;   // four elements as whole words (2 or 4 of them)
        o.t[0] = from_float<T>(x1.a.x * inv);
        o.t[1] = from_float<T>(x1.a.y * inv);
        o.t[2] = from_float<T>(x1.a.z * inv);
        o.t[3] = from_float<T>(x1.a.w * inv);
        T *dst = reinterpret_cast<T *>(p.out) + orow * D + 4 * c4;
        if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4 *>(dst) = make_uint4(o.w[0], o.w[1], o.w[2], o.w[3]);
        else *reinterpret_cast<uint2 *>(dst) = make_uint2(o.w[0], o.w[1]);
        if (c4 == 0 && p.lse_out)
            p.lse_out[orow] = ((x1.m == -INFINITY ? 0.f : x1.m) + log2f(x1.l)) * 0.6931471805599453f;
        if (p.peer_world > 0) {
            // these four values as payload words {payload, tag} into slot (seq & 1) of every rank's buffer,
            // at this rank's place (one query token per call: orow is the head row)
            const int32_t sq = peer_step;
            const uint32_t tag = (uint32_t)(sq + 1);
            constexpr int NW = (int)sizeof(T);
            const size_t word0 = (size_t)(sq & 1) * p.peer_world * p.peer_words + (size_t)p.peer_rank * p.peer_words +
                                 (orow * D + 4 * c4) * sizeof(T) / 4;
#pragma unroll
            for (int gp = 0; gp < kAttnMaxPeers; ++gp) {
                if (gp < p.peer_world) {
                    uint2 *pd = p.peer_buf[gp] + word0;
#pragma unroll
                    for (int i = 0; i < NW; ++i) st_word_sys(pd + i, o.w[i], tag);
                }
            }
        }
    }
}

template <typename T, int D, int THREADS, bool TWO>
__device__ __forceinline__ void merge_partials(const AttnParams &p, int h, int rows, int todo, unsigned char *smem) {
    constexpr int LONG = TWO ? kMergeBatchTwo : kMergeBatch;
    const int groups = max(THREADS / (rows * (D / 4)), 1);
    const int n1 = TWO ? p.splits1 : p.ticket_target;
    if ((TWO && todo == kMergeRest) || n1 <= kMergeBatchFew * groups)
        merge_partials_by<T, D, THREADS, kMergeBatchFew, TWO>(p, h, rows, todo, smem);
    else
        merge_partials_by<T, D, THREADS, LONG, TWO>(p, h, rows, todo, smem);
}

// 16-bit element types: tensor-core kernel (attn_mma.cu).
cudaError_t launch_attention_mma(const AttnParams &p, int n_kv_heads, int head_dim, int dtype, int splits,
                                 cudaStream_t stream);

}  // namespace da
