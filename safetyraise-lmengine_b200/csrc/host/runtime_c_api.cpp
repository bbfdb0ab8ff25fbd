#include "runtime_c_api.h"

#include <vector>

#include "cache_manager.hpp"
#include "scheduler.hpp"

using srlm::CacheManager;
using srlm::Scheduler;

extern "C" {

void* srlm_cache_create(int max_requests, int n_groups, const int* kinds, const int* page_sizes,
                        const int* num_pages, const int* windows, const int* keep_first) {
  if (max_requests <= 0 || n_groups < 0) return nullptr;
  std::vector<srlm::GroupSpec> groups;
  for (int g = 0; g < n_groups; ++g) {
    if (page_sizes[g] <= 0 || num_pages[g] <= 0) return nullptr;
    if (kinds[g] == srlm::GROUP_WINDOW && (windows[g] <= 0 || keep_first[g] < 0)) return nullptr;
    groups.push_back(srlm::GroupSpec{kinds[g], page_sizes[g], num_pages[g], windows[g], keep_first[g]});
  }
  return new CacheManager(max_requests, groups);
}
void srlm_cache_destroy(void* c) { delete static_cast<CacheManager*>(c); }
int srlm_cache_open(void* c) { return static_cast<CacheManager*>(c)->open_request(); }
int srlm_cache_close(void* c, int slot) { return static_cast<CacheManager*>(c)->close_request(slot); }
int srlm_cache_reserve(void* c, int slot, int n) { return static_cast<CacheManager*>(c)->reserve(slot, n); }
int srlm_cache_fit_tokens(void* c, int slot, int n) { return static_cast<CacheManager*>(c)->fit_tokens(slot, n); }
int srlm_cache_commit(void* c, int slot, int n) { return static_cast<CacheManager*>(c)->commit(slot, n); }
int srlm_cache_truncate(void* c, int slot, int n) { return static_cast<CacheManager*>(c)->truncate(slot, n); }
int srlm_cache_length(void* c, int slot) { return static_cast<CacheManager*>(c)->length(slot); }
int srlm_cache_reserved(void* c, int slot) { return static_cast<CacheManager*>(c)->reserved_tokens(slot); }
int srlm_cache_generation(void* c, int slot) { return static_cast<CacheManager*>(c)->generation(slot); }
int srlm_cache_table(void* c, int group, int slot, int32_t* out, int cap) {
  return static_cast<CacheManager*>(c)->table(group, slot, out, cap);
}
int srlm_cache_free_pages(void* c, int group) { return static_cast<CacheManager*>(c)->free_pages(group); }
int srlm_cache_audit(void* c) { return static_cast<CacheManager*>(c)->audit(); }
static uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
void srlm_sampling_uniforms(int n, const uint64_t* seeds, const uint64_t* indices, float* out) {
  for (int i = 0; i < n; ++i) {
    const uint64_t bits = splitmix64(splitmix64(seeds[i]) ^ (indices[i] + 1) * 0xD1B54A32D192ED03ull);
    out[i] = static_cast<float>(bits >> 40) * (1.0f / (1 << 24));
  }
}
void srlm_cache_reuse_counts(void* c, int64_t* taken, int64_t* reused) {
  *taken = static_cast<CacheManager*>(c)->pages_taken_total();
  *reused = static_cast<CacheManager*>(c)->pages_reused_total();
}

void srlm_cache_look(void* c, int n, const int32_t* slots, int32_t* lengths, int32_t* generations) {
  const CacheManager* m = static_cast<CacheManager*>(c);
  for (int i = 0; i < n; ++i) {
    lengths[i] = m->length(slots[i]);
    generations[i] = m->generation(slots[i]);
  }
}
int srlm_cache_reserve_many(void* c, int n, const int32_t* slots, const int32_t* starts, const int32_t* new_lens) {
  CacheManager* m = static_cast<CacheManager*>(c);
  for (int i = 0; i < n; ++i) {
    const int r = m->reserve(slots[i], new_lens[i]);
    if (r == 1) continue;
    for (int j = 0; j < i; ++j) m->truncate(slots[j], starts[j]);
    return r == 0 ? i : -1 - i;
  }
  return n;
}
int srlm_cache_commit_many(void* c, int n, const int32_t* slots, const int32_t* new_lens) {
  for (int i = 0; i < n; ++i)
    if (static_cast<CacheManager*>(c)->commit(slots[i], new_lens[i]) != 0) return i;
  return n;
}
void srlm_lay_out_tokens(int n, const int32_t* starts, const int32_t* q_lens, int32_t* positions, int32_t* entry_of_token,
                         int32_t* cu_q, int32_t* kv_lens) {
  int t = 0;
  cu_q[0] = 0;
  for (int e = 0; e < n; ++e) {
    for (int j = 0; j < q_lens[e]; ++j, ++t) {
      positions[t] = starts[e] + j;
      entry_of_token[t] = e;
    }
    cu_q[e + 1] = t;
    kv_lens[e] = starts[e] + q_lens[e];
  }
}
int srlm_cache_lay_out_pages(void* c, int group, int n, const int32_t* slots, const int32_t* starts,
                             const int32_t* q_lens, int page_size, int pages, int32_t* tables, int32_t* kv_slot) {
  const CacheManager* m = static_cast<CacheManager*>(c);
  int t = 0;
  for (int e = 0; e < n; ++e) {
    int32_t* row = tables + static_cast<int64_t>(e) * pages;
    const int held = m->table(group, slots[e], row, pages);
    if (held < 0 || held > pages) return 1 + e;
    for (int i = held; i < pages; ++i) row[i] = 0;
    for (int j = 0; j < q_lens[e]; ++j, ++t) {
      const int p = starts[e] + j;
      kv_slot[t] = row[p / page_size] * page_size + p % page_size;
    }
  }
  return 0;
}

void* srlm_sched_create(void* cache, int max_active, int queue_capacity, int prefill_chunk,
                        int max_batch_tokens, int max_context) {
  if (!cache || max_active <= 0 || queue_capacity <= 0 || prefill_chunk <= 0 ||
      max_batch_tokens <= 0 || max_context <= 0)
    return nullptr;
  srlm::SchedulerConfig cfg{max_active, queue_capacity, prefill_chunk, max_batch_tokens, max_context};
  return new Scheduler(cfg, static_cast<CacheManager*>(cache));
}
void srlm_sched_destroy(void* s) { delete static_cast<Scheduler*>(s); }
int srlm_sched_submit(void* s, int64_t id, int prompt_len, int max_new) {
  return static_cast<Scheduler*>(s)->submit(id, prompt_len, max_new);
}
int srlm_sched_plan(void* s, int64_t* entries, int cap, int64_t* preempted, int* n_preempted) {
  std::vector<srlm::PlanEntry> out;
  std::vector<int64_t> pre;
  static_cast<Scheduler*>(s)->plan(&out, &pre);
  int n = 0;
  for (const srlm::PlanEntry& e : out) {
    if (n >= cap) break;
    int64_t* row = entries + 5 * n++;
    row[0] = e.id; row[1] = e.slot; row[2] = e.start; row[3] = e.count; row[4] = e.want_logits;
  }
  int np = 0;
  for (int64_t id : pre) if (np < cap) preempted[np++] = id;
  *n_preempted = np;
  return n;
}
int srlm_sched_advance(void* s, int64_t id, int count) { return static_cast<Scheduler*>(s)->advance(id, count); }
int srlm_sched_rollback(void* s, int64_t id) { return static_cast<Scheduler*>(s)->rollback(id); }
int srlm_sched_append_token(void* s, int64_t id) { return static_cast<Scheduler*>(s)->append_token(id); }
int srlm_sched_retract_token(void* s, int64_t id) { return static_cast<Scheduler*>(s)->retract_token(id); }
int srlm_sched_finish(void* s, int64_t id) { return static_cast<Scheduler*>(s)->finish(id); }
int srlm_sched_has_work(void* s) { return static_cast<Scheduler*>(s)->has_work() ? 1 : 0; }
void srlm_sched_counters(void* s, int64_t* out) {
  srlm::Counters c = static_cast<Scheduler*>(s)->counters();
  out[0] = c.submitted; out[1] = c.rejected; out[2] = c.completed; out[3] = c.preempted;
  out[4] = c.steps; out[5] = c.batched_tokens; out[6] = c.generated_tokens;
  out[7] = c.active; out[8] = c.queued;
}

}  // extern "C"
