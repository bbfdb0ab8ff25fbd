/* C interface of the host runtime (cache manager and scheduler), loaded from
 * Python with ctypes.  Handles are opaque pointers; every function returns a
 * status (>= 0 fine, < 0 an error named beside it in the C++ headers). */
#pragma once
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

void* srlm_cache_create(int max_requests, int n_groups, const int* kinds, const int* page_sizes,
                        const int* num_pages, const int* windows, const int* keep_first);
void srlm_cache_destroy(void* cache);
int srlm_cache_open(void* cache);
int srlm_cache_close(void* cache, int slot);
int srlm_cache_reserve(void* cache, int slot, int new_len);
int srlm_cache_fit_tokens(void* cache, int slot, int want_len);
int srlm_cache_commit(void* cache, int slot, int new_len);
int srlm_cache_truncate(void* cache, int slot, int len);
int srlm_cache_length(void* cache, int slot);
int srlm_cache_reserved(void* cache, int slot);
int srlm_cache_generation(void* cache, int slot);
int srlm_cache_table(void* cache, int group, int slot, int32_t* out, int cap);
int srlm_cache_free_pages(void* cache, int group);
int srlm_cache_audit(void* cache);
/* The same for the n entries of a step at once.  look: lengths and generations (-1 where there is none).
 * reserve_many: n, all or nothing; else the first entry without pages, as its index, or as -1 - index where the
 * arguments are invalid (what the call took is given back).  commit_many: n, or the index of the first invalid entry. */
void srlm_cache_look(void* cache, int n, const int32_t* slots, int32_t* lengths, int32_t* generations);
int srlm_cache_reserve_many(void* cache, int n, const int32_t* slots, const int32_t* starts, const int32_t* new_lens);
int srlm_cache_commit_many(void* cache, int n, const int32_t* slots, const int32_t* new_lens);
/* A step's layout: positions, entry of every token, offsets of the entries' tokens, context lengths; and for a group the
 * entries' block tables (`pages` columns, zeros behind what a slot holds) and the flat cache row of every token.
 * lay_out_pages: 0, or 1 + the entry whose slot holds more than `pages` pages or is not open. */
void srlm_lay_out_tokens(int n, const int32_t* starts, const int32_t* q_lens, int32_t* positions, int32_t* entry_of_token,
                         int32_t* cu_q, int32_t* kv_lens);
int srlm_cache_lay_out_pages(void* cache, int group, int n, const int32_t* slots, const int32_t* starts,
                             const int32_t* q_lens, int page_size, int pages, int32_t* tables, int32_t* kv_slot);
/* out[i]: the uniform number in [0, 1) of draw indices[i] of a request with seeds[i] (24 bits, a function of the two alone). */
void srlm_sampling_uniforms(int n, const uint64_t* seeds, const uint64_t* indices, float* out);
void srlm_cache_reuse_counts(void* cache, int64_t* taken, int64_t* reused);

void* srlm_sched_create(void* cache, int max_active, int queue_capacity, int prefill_chunk,
                        int max_batch_tokens, int max_context);
void srlm_sched_destroy(void* sched);
int srlm_sched_submit(void* sched, int64_t id, int prompt_len, int max_new);
/* entries: 5 int64 per entry (id, slot, start, count, want_logits); returns the entry count,
 * writes the number of preempted ids to *n_preempted (ids in `preempted`, cap each). */
int srlm_sched_plan(void* sched, int64_t* entries, int cap, int64_t* preempted, int* n_preempted);
int srlm_sched_advance(void* sched, int64_t id, int count);
int srlm_sched_rollback(void* sched, int64_t id);
int srlm_sched_append_token(void* sched, int64_t id);
int srlm_sched_retract_token(void* sched, int64_t id);
int srlm_sched_finish(void* sched, int64_t id);
int srlm_sched_has_work(void* sched);
/* out[9]: submitted rejected completed preempted steps batched_tokens generated_tokens active queued */
void srlm_sched_counters(void* sched, int64_t* out);

#ifdef __cplusplus
}
#endif
