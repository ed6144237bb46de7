// One generate call as one library call: every launch of the step, on one or two streams, enqueued from native
// code.  Enqueued one by one from an interpreted caller the launches, stream switches and events of a step took
// about 110 us of host time, three times what the GPU needs for them.

#include <new>

#include "da_common.cuh"

namespace da {

struct Fork {
    cudaStream_t side;
    cudaEvent_t started, joined;
};

static int push_peers(const da_generate_args &a) {
    if (!a.peer_buffers) return 0;
    return da_decode_attention_push_next(reinterpret_cast<void *const *>(a.peer_buffers), a.peer_seq,
                                         (int)a.peer_rank, (int)a.peer_world, (int)a.peer_bytes);
}

static int attention_plain(const da_generate_args &a) {
    if (const int rc = push_peers(a)) return rc;
    return da_decode_attention_tokens(a.q, (int)a.n_q_tokens, a.slots, a.slots_head_stride, (int)a.n_prefix_tokens,
                                      a.local_k, a.local_v, a.local_token_stride, a.local_head_stride,
                                      (int)a.local_capacity, a.new_k, a.new_v, a.start_pos_dev,
                                      (int)a.start_pos_host, (int)a.dram_tokens, a.out, nullptr, a.workspace,
                                      (size_t)a.workspace_bytes, a.status, (int)a.n_kv_heads, (int)a.rep,
                                      (int)a.head_dim, (int)a.dtype, a.stream);
}

static int attention_fetch(const da_generate_args &a) {
    if (const int rc = push_peers(a)) return rc;
    return da_decode_attention_fetch(a.q, a.slots, a.slots_head_stride, (int)a.n_slots, (int)a.page_size, a.dram_pages,
                                     (int)a.n_dram_pages, a.slot_source, a.local_k, a.local_v, a.local_token_stride,
                                     a.local_head_stride, (int)a.local_capacity, a.new_k, a.new_v, a.start_pos_dev,
                                     (int)a.start_pos_host, (int)a.dram_tokens, a.out, nullptr, a.workspace,
                                     (size_t)a.workspace_bytes, a.status, (int)a.n_kv_heads, (int)a.rep,
                                     (int)a.head_dim, (int)a.dtype, a.stream);
}

static int attention_phase(const da_generate_args &a, int phase, cudaStream_t stream) {
    if (const int rc = push_peers(a)) return rc;
    return da_decode_attention_phased(phase, a.evict_queue, a.front_count, a.split_flip, a.split_redo,
                                      (int)a.phase1_ctas, (int)a.phase2_ctas, a.q, a.slots, a.slots_head_stride,
                                      (int)a.n_slots, (int)a.page_size, a.dram_pages, (int)a.n_dram_pages,
                                      a.slot_source, a.local_k, a.local_v, a.local_token_stride, a.local_head_stride,
                                      (int)a.local_capacity, a.new_k, a.new_v, a.start_pos_dev, (int)a.start_pos_host,
                                      (int)a.dram_tokens, a.out, nullptr, a.workspace, (size_t)a.workspace_bytes,
                                      a.status, (int)a.n_kv_heads, (int)a.rep, (int)a.head_dim, (int)a.dtype, stream);
}

static int select_pages(const da_generate_args &a, int sm_budget) {
    return da_topk_pages_wide(a.scores, a.page_list, (int)a.n_q_tokens, (int)a.n_kv_heads, (int)a.rep,
                              (int)a.n_dram_pages, (int)a.top_k, sm_budget, a.stream);
}

static int update_tables(const da_generate_args &a, int advance, bool inline_fetch) {
    const int list_len = (int)(a.n_q_tokens * a.rep * a.top_k);
    return da_lru_update(a.page_list, list_len, a.dram_to_slot, (int)a.n_dram_pages, a.slot_to_dram, a.access_time,
                         (int)a.n_slots, a.step, (int)a.n_kv_heads, a.miss_pages, a.miss_slots, a.n_miss, a.slot_source,
                         a.evict_queue, a.front_count, a.split_flip, a.split_redo, (int)a.split_cap, advance,
                         inline_fetch ? a.dram_pages : nullptr, inline_fetch ? a.slots : nullptr,
                         (size_t)a.page_bytes, inline_fetch ? (int)a.inline_fetch_max : 0, a.lru_status, a.stream);
}

}  // namespace da

extern "C" int da_fork_create(void **fork) {
    if (!fork) return DA_ERR_NULL;
    da::Fork *f = new (std::nothrow) da::Fork();
    if (!f) return (int)cudaErrorMemoryAllocation;
    cudaError_t e = cudaStreamCreateWithFlags(&f->side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&f->started, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&f->joined, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        da_fork_destroy(f);
        return (int)e;
    }
    *fork = f;
    return 0;
}

extern "C" void da_fork_destroy(void *fork) {
    da::Fork *f = static_cast<da::Fork *>(fork);
    if (!f) return;
    if (f->started) cudaEventDestroy(f->started);
    if (f->joined) cudaEventDestroy(f->joined);
    if (f->side) cudaStreamDestroy(f->side);
    delete f;
}

extern "C" int da_generate(const da_generate_args *args) {
    if (!args) return DA_ERR_NULL;
    const da_generate_args &a = *args;
    int rc;
    if (a.layout == DA_LAYOUT_RESIDENT) return da::attention_plain(a);
    if (a.layout < 0 || a.layout > DA_LAYOUT_OVERLAPPED) return DA_ERR_SHAPE;
    cudaStream_t main = static_cast<cudaStream_t>(a.stream);
    da::Fork *f = static_cast<da::Fork *>(a.fork);
    const bool two = a.layout == DA_LAYOUT_OVERLAPPED;
    if (two && !f) return DA_ERR_NULL;
    const bool early = two && a.fork_before_score != 0;
    rc = da::score_pages(a.q, a.summaries, a.scores, (int)a.n_q_tokens, (int)a.n_kv_heads, (int)a.rep,
                         (int)a.n_dram_pages, (int)a.head_dim, (int)a.dtype, 1, main, early ? f->started : nullptr);
    if (rc) return rc;
    if (!two) {
        if ((rc = da::select_pages(a, 0)) != 0) return rc;
        if (a.layout == DA_LAYOUT_FETCH_IN_ATTENTION) {
            if ((rc = da::update_tables(a, 1 | 2, true)) != 0) return rc;
            return da::attention_fetch(a);
        }
        if ((rc = da::update_tables(a, 1, false)) != 0) return rc;
        rc = da_fetch_pages(a.dram_pages, a.slots, a.miss_pages, a.miss_slots, a.n_miss,
                            (int)(a.n_q_tokens * a.rep * a.top_k), (int)a.n_kv_heads, (int)a.n_dram_pages, (int)a.n_slots,
                            (size_t)a.page_bytes, a.stream);
        return rc ? rc : da::attention_plain(a);
    }
    // { score -> select -> LRU update -> attention phase 2 }  ||  attention phase 1
    cudaError_t e;
    int budget = (int)a.selection_sm_budget;
    if (budget <= 0) {
        const int ctas1 = a.phase1_ctas > 0 ? (int)a.phase1_ctas : da_decode_attention_phase1_ctas((int)a.n_kv_heads);
        budget = 148 - (int)a.n_kv_heads * ctas1;
        if (budget < 1) budget = 1;
    }
    if (!early && (e = cudaEventRecord(f->started, main)) != cudaSuccess) return (int)e;
    const da::AheadOfStream ahead(main);   // selection, update and phase 2
    if ((rc = da::select_pages(a, budget)) != 0) return rc;
    if ((e = cudaStreamWaitEvent(f->side, f->started, 0)) != cudaSuccess) return (int)e;
    const int rc1 = da::attention_phase(a, 1, f->side);
    rc = rc1;
    if (rc == 0) rc = da::update_tables(a, 2, true);
    // phase 2 needs the update, not phase 1: whichever of the two launches finishes last merges
    if (rc == 0) rc = da::attention_phase(a, 2, main);
    // The fork's stream is joined whatever became of the launches: phase 1 reads the caller's tensors, and a capture ends
    // only with all its streams joined.
    if ((e = cudaEventRecord(f->joined, f->side)) == cudaSuccess) e = cudaStreamWaitEvent(main, f->joined, 0);
    // Phase 1 without its phase 2 leaves its tickets in the workspace, which the next call would count as its own.
    if (rc != 0 && rc1 == 0 && e == cudaSuccess)
        e = cudaMemsetAsync(a.workspace, 0, (size_t)a.n_kv_heads * sizeof(unsigned int), main);
    return rc != 0 ? rc : (int)e;
}
