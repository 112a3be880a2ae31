// gtk_api.cu -- the C ABI declared in include/gputok_b200.h.
//
// One handle = one device, one stream, one merge table in HBM and a set of
// grow-only arenas (device and pinned host), so a call allocates nothing once
// the arenas have reached the working size.  The reference allocates and
// frees five device buffers inside every call (gputok_binding.cu:906-910,
// 981-986), which its own profile shows to be 70-95 % of the API time.
#include "../../include/gputok_b200.h"

#include <cuda_runtime.h>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "gtk_crew.hpp"
#include "gtk_device.cuh"
#include "gtk_table.hpp"

namespace {

thread_local std::string g_global_error;

struct CudaFail {
  std::string what;
};

#define GTK_CUDA(expr)                                                                              \
  do {                                                                                              \
    cudaError_t e__ = (expr);                                                                       \
    if (e__ != cudaSuccess) {                                                                       \
      throw CudaFail{std::string(#expr) + ": " + cudaGetErrorString(e__)};                          \
    }                                                                                               \
  } while (0)

// grow-only device / pinned-host buffers
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  void reserve(size_t bytes)
  {
    if (bytes <= cap) return;
    if (p) GTK_CUDA(cudaFree(p));
    p = nullptr;
    cap = 0;
    size_t want = std::max(bytes + bytes / 4, size_t(4096));
    GTK_CUDA(cudaMalloc(&p, want));
    cap = want;
  }
  void release()
  {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
  template <class T>
  T* as() const { return static_cast<T*>(p); }
};

struct PinBuf {
  void* p = nullptr;
  size_t cap = 0;
  void reserve(size_t bytes)
  {
    if (bytes <= cap) return;
    if (p) GTK_CUDA(cudaFreeHost(p));
    p = nullptr;
    cap = 0;
    size_t want = std::max(bytes + bytes / 4, size_t(4096));
    GTK_CUDA(cudaHostAlloc(&p, want, cudaHostAllocDefault));
    cap = want;
  }
  // page-locked memory that kernels write directly (dp = the address as the device sees it)
  void* dp = nullptr;
  void reserve_mapped(size_t bytes)
  {
    if (bytes <= cap && dp) return;
    if (p) GTK_CUDA(cudaFreeHost(p));
    p = dp = nullptr;
    cap = 0;
    size_t want = std::max(bytes, size_t(4096));
    GTK_CUDA(cudaHostAlloc(&p, want, cudaHostAllocMapped));
    GTK_CUDA(cudaHostGetDevicePointer(&dp, p, 0));
    cap = want;
  }
  void release()
  {
    if (p) cudaFreeHost(p);
    p = dp = nullptr;
    cap = 0;
  }
  template <class T>
  T* as() const { return static_cast<T*>(p); }
};

// Page-locked result buffers that callers have taken over (gtk_result_take) come back here when they are done with them.
// Shared by the handle and by the results that are still out, so either may go first.  Bounded: at most kMaxTaken
// results are out (further takes are refused and the caller copies), at most kMaxSpare buffers wait to be used again.
struct ResultPool {
  static constexpr int kMaxTaken = 4, kMaxSpare = 6;
  static constexpr size_t kMaxTakenBytes = size_t(1) << 30, kMaxSpareBytes = size_t(512) << 20;
  std::mutex mu;
  std::vector<PinBuf> spare;
  int taken = 0;
  size_t taken_bytes = 0, spare_bytes = 0;
  bool closed = false;  // the handle is gone

  ResultPool() { spare.reserve(size_t(kMaxSpare)); }  // give_back allocates nothing: it ends gtk_result_release
  ~ResultPool()
  {
    for (PinBuf& b : spare) b.release();
  }
  // a buffer of at least `bytes`: the one in hand, else the smallest spare one that does, else a new one
  void reserve(PinBuf& buf, size_t bytes)
  {
    if (buf.p && bytes <= buf.cap) return;
    {
      std::lock_guard<std::mutex> lock(mu);
      size_t best = spare.size();
      for (size_t i = 0; i < spare.size(); ++i)
        if (spare[i].cap >= bytes && (best == spare.size() || spare[i].cap < spare[best].cap)) best = i;
      if (best < spare.size()) {
        std::swap(buf, spare[best]);
        spare_bytes += spare[best].cap - buf.cap;
        if (!spare[best].p) spare.erase(spare.begin() + long(best));
        return;
      }
    }
    buf.reserve(bytes);
  }
  void give_back(PinBuf& buf)
  {
    if (!buf.p) return;
    std::lock_guard<std::mutex> lock(mu);
    if (closed || int(spare.size()) >= kMaxSpare || spare_bytes + buf.cap > kMaxSpareBytes) {
      buf.release();
      return;
    }
    spare_bytes += buf.cap;
    spare.push_back(buf);
    buf = PinBuf();
  }
};

}  // namespace

// A result that its caller has taken over.
struct gtk_taken {
  std::shared_ptr<ResultPool> pool;
  PinBuf bufs[3];
  size_t bytes = 0;
};

// Buffers of one in-flight slice of a large host batch (kSliceArenas sets rotate).
constexpr int kSliceArenas = 4;
struct SliceArena {
  DevBuf text_chunk_base, chunk_off, chunk_cnt, scan_sums, counters, totals;
  PinBuf h_totals;  // mapped: written by a kernel
  cudaEvent_t ev[6] = {};          // stage timing
  cudaEvent_t ev_in = nullptr;     // slice text is in HBM
  cudaEvent_t ev_front = nullptr;  // totals of the slice are on the host
  cudaEvent_t ev_packed = nullptr; // ids of the slice are packed
  cudaEvent_t ev_out = nullptr;    // results of the slice are on the host
  void release()
  {
    for (DevBuf* b : {&text_chunk_base, &chunk_off, &chunk_cnt, &scan_sums, &counters, &totals})
      b->release();
    h_totals.release();
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
    for (cudaEvent_t* e : {&ev_in, &ev_front, &ev_packed, &ev_out})
      if (*e) cudaEventDestroy(*e);
  }
};

struct gtk_tokenizer {
  std::unique_ptr<gtk::HostTable> table;
  int chunk_tokens = 2048;
  int max_iters = 50;
  int device = -1;
  int sm_count = 0;
  int opt_grid = 0, base_grid = 0, localmin_grid = 0, wide_grid = 0;
  int base_block = 0;  // threads per CTA of the one-CTA-per-chunk kernel, 0 = from the chunk size
  bool stage_timing = false;  // events between the stages of a batch that runs in one piece (gtk_set_stage_timing)
  float front_ms = -1.f;      // chunker + merge + scans of the last such batch when timed as one interval
  bool wide = false;  // ids or ranks beyond 16 bits: every GPU mode runs the 32-bit one-CTA-per-chunk kernel
  cudaStream_t stream = nullptr;      // stream in use
  cudaStream_t own_stream = nullptr;  // created by gtk_create
  cudaEvent_t ev[6] = {};
  std::mutex mu;
  mutable std::string last_error;

  // table in HBM
  DevBuf d_bpi;
  DevBuf d_slots, d_overflow, d_bpr, d_mor, d_sor, d_adj, d_b2i, d_short_words, d_long_words, d_learned_words, d_low_map, d_wide_slots;
  DevBuf d_staging32, d_seg_scratch32;  // 32-bit kernel
  int id_space = GTK_IDS_REFERENCE;
  gtk::DeviceTable dtab{};
  gtk::DeviceTable call_tab{};  // what the kernels of the present call get: dtab, or with a long table of the call's own

  // arenas
  DevBuf d_bytes, d_text_off, d_text_chunk_base, d_chunk_off, d_tile_chunk0, d_staging, d_unit_first, d_unit_cnt,
      d_chunk_cnt, d_tile_info, d_chunk_rel, d_text_rel, d_group_base, d_chunk_id_off, d_text_id_off, d_out_ids, d_seg_scratch, d_scan_sums,
      d_totals;  // d_totals also holds the counters and group counts (plan_batch)
  PinBuf h_ids, h_text_id_off, h_chunk_id_off, h_totals;
  // sliced host batches: offsets of all slices, moved once per batch
  DevBuf d_piece_off, d_piece_id_off, d_chunk_id_all;
  PinBuf h_piece_off, h_piece_id_off, h_chunk_id_all;
  // small batches: input and results live in mapped page-locked memory, one kernel per call
  uint8_t* small_in_h = nullptr;   // [text offsets | bytes]
  uint8_t* small_in_d = nullptr;
  uint8_t* small_out_h = nullptr;  // [totals | text id offsets | chunk id offsets | ids]
  uint8_t* small_out_d = nullptr;
  bool result_is_small = false;
  // batches below the slicing threshold: one arena [text id offsets | chunk id offsets | ids] on both sides
  DevBuf d_out_pack;
  PinBuf h_out_pack;
  bool result_is_packed = false;
  bool ids_apart = false;  // of a packed result: the ids are in h_ids
  std::shared_ptr<ResultPool> pool = std::make_shared<ResultPool>();
  bool result_is_taken = false;
  const int32_t* view_ids = nullptr;
  const int64_t *view_text = nullptr, *view_chunk = nullptr;
  PinBuf* result_bufs[3] = {nullptr, nullptr, nullptr};  // what the last result lives in, as far as it can be taken over
  size_t pack_text_bytes = 0, pack_chunk_bytes = 0;
  const uint8_t* pack_base = nullptr;  // h_out_pack, or the mapped block below behind its 64-byte header
  // batches of up to 1 MiB: a kernel writes the results into this mapped block and the host polls its header
  PinBuf h_mid;
  PinBuf h_out;                // results of encode_host_tiles, offsets of encode_host_pieces
  DevBuf d_piece_ids;          // ids in front of every piece
  PinBuf h_gather;             // strings of gtk_encode_strings, back to back
  mutable gtk::Crew crew;
  PinBuf h_marks;              // completion mark and id count of every piece
  std::vector<cudaEvent_t> piece_ev;
  double ids_per_byte = 0.4;  // room for ids that they start with; grows with the texts it meets
  int64_t mid_seq = 0;
  // zeroed counters, scanned chunk counts and, when it is short, the text travel in one copy (encode_host_tiles)
  PinBuf h_fast_in;
  DevBuf d_fast_in;
  int64_t small_seq = 0;  // calls of the small-batch kernel so far (the kernel echoes it as its completion mark)
  // sliced host path: copy streams and two slice arenas
  cudaStream_t in_stream = nullptr, out_stream = nullptr, pack_stream = nullptr;
  SliceArena slice[kSliceArenas];
  // host-side result of gtk_encode_cpu
  std::vector<int32_t> cpu_ids;
  std::vector<int64_t> cpu_text_off, cpu_chunk_off;
  bool result_is_cpu = false;
  int64_t res_n_ids = 0, res_n_chunks = 0, res_n_texts = 0;
  float stage_ms[5] = {0, 0, 0, 0, 0};
  int32_t last_launches = 0;

  int fail(int code, const std::string& msg) const
  {
    last_error = msg;
    return code;
  }
};

namespace {

// What a failing call does last: its copies and kernels may still be reading the caller's text or the handle's buffers.
void settle(gtk_tokenizer* h)
{
  for (cudaStream_t s : {h->in_stream, h->stream, h->pack_stream, h->out_stream})
    if (s) cudaStreamSynchronize(s);
}

int out_of_memory(const gtk_tokenizer* h) { return h->fail(GTK_ERR_MEMORY, "out of memory"); }  // short enough to need none

void upload(DevBuf& buf, const void* src, size_t bytes, cudaStream_t s)
{
  buf.reserve(bytes);
  GTK_CUDA(cudaMemcpyAsync(buf.p, src, bytes, cudaMemcpyHostToDevice, s));
}

void upload_table(gtk_tokenizer* h)
{
  const gtk::HostTable& t = *h->table;
  upload(h->d_slots, t.pair_buckets.data(), t.pair_buckets.size() * sizeof(gtk::PairBucket), h->stream);
  if (!t.pair_overflow.empty())
    upload(h->d_overflow, t.pair_overflow.data(), t.pair_overflow.size() * sizeof(gtk::PairSlot), h->stream);
  upload(h->d_bpr, t.byte_pair_rank.data(), t.byte_pair_rank.size() * sizeof(uint16_t), h->stream);
  upload(h->d_bpi, t.byte_pair_info.data(), t.byte_pair_info.size() * sizeof(uint16_t), h->stream);
  upload(h->d_mor, t.merged_of_rank.data(), t.merged_of_rank.size() * sizeof(uint32_t), h->stream);
  upload(h->d_sor, t.same_of_rank.data(), t.same_of_rank.size(), h->stream);
  uint32_t adj[2048];  // the device's layout: [v / 32][u]
  for (int u = 0; u < 256; ++u)
    for (int v = 0; v < 8; ++v) adj[v * 256 + u] = t.adj[u * 8 + v];
  upload(h->d_adj, adj, sizeof(adj), h->stream);
  upload(h->d_b2i, t.byte_to_id, sizeof(t.byte_to_id), h->stream);
  upload(h->d_low_map, t.gpt2_low_id, sizeof(t.gpt2_low_id), h->stream);
  upload(h->d_short_words, t.short_words.data(), t.short_words.size() * sizeof(gtk::ShortWord), h->stream);
  upload(h->d_long_words, t.long_words.data(), t.long_words.size() * sizeof(gtk::LongWord), h->stream);
  if (h->wide) upload(h->d_wide_slots, t.slots.data(), t.slots.size() * sizeof(gtk::HashSlot), h->stream);
  GTK_CUDA(cudaStreamSynchronize(h->stream));
  h->dtab.pair_buckets = h->d_slots.as<uint4>();
  h->dtab.pair_overflow = t.pair_overflow.empty() ? nullptr : h->d_overflow.as<uint2>();
  h->dtab.pair_overflow_mask = t.pair_overflow.empty() ? 0u : uint32_t(t.pair_overflow.size() - 1);
  h->dtab.byte_pair_rank = h->d_bpr.as<uint16_t>();
  h->dtab.byte_pair_info = h->d_bpi.as<uint16_t>();
  h->dtab.merged_of_rank = h->d_mor.as<uint32_t>();
  h->dtab.same_of_rank = h->d_sor.as<uint8_t>();
  h->dtab.adj = h->d_adj.as<uint32_t>();
  h->dtab.byte_to_id = h->d_b2i.as<uint16_t>();
  h->dtab.short_words = h->d_short_words.as<uint2>();
  h->dtab.long_words = h->d_long_words.as<uint4>();
  h->dtab.learn = 0;
  h->dtab.wide_slots = h->wide ? h->d_wide_slots.as<uint4>() : nullptr;
  h->dtab.wide_log2 = t.log2_capacity;
  h->dtab.wide_max_probe = t.max_probe;
  h->dtab.monotone = t.monotone ? 1 : 0;
  h->dtab.merged_is_256_plus_rank = t.merged_is_256_plus_rank ? 1 : 0;
  h->dtab.byte_ids_identity = t.byte_ids_identity ? 1 : 0;
}

// From this size on the tile kernel works on a copy of the long-string table and adds the segments it merges, so that a
// word that is not in the vocabulary is merged once in a batch and looked up from then on.  Every call starts from the
// vocabulary's own strings.  Where the line lies: the copy (8 MiB within L2, 3 us) and the first tiles, all of which miss
// and add at once, have to be earned back.  English-like text of 4 / 8 / 16 / 64 MiB: 115 / 144 / 193 / 452 us with,
// 101 / 141 / 204 / 588 us without; the sample novel 104 / 139 / 168 / 386 against 109 / 151 / 203 / 561 us.
constexpr int64_t kLearnMinBytes = int64_t(12) << 20;

void begin_call(gtk_tokenizer* h, int mode, int64_t n_bytes)
{
  h->call_tab = h->dtab;
  if (h->wide || mode != GTK_MODE_OPT || n_bytes < kLearnMinBytes) return;
  h->d_learned_words.reserve(h->table->long_words.size() * sizeof(gtk::LongWord));
  h->call_tab.long_words = h->d_learned_words.as<uint4>();
  h->call_tab.learn      = 1;  // begin_tiles sets it up
}

// Upper bound on the number of chunks without touching the device: every text
// contributes its full chunks plus at most one partial chunk.
int64_t chunk_upper_bound(int64_t n_bytes, int64_t n_texts, int chunk_tokens)
{
  return n_bytes / chunk_tokens + n_texts + 1;
}

struct Plan {
  gtk::EncodeBuffers b{};
  int64_t chunk_cap = 0;
};

// Which kernels a batch is planned for: each has arrays of its own.
enum class Kernels { tiles, chunks, small };

// Size the arenas for a batch and fill the kernel argument block.
Plan plan_batch(gtk_tokenizer* h, Kernels kernels, const uint8_t* d_bytes, int64_t n_bytes, const int64_t* d_text_off,
                int64_t n_texts, int32_t* d_out_ids, int64_t out_capacity, int64_t* d_chunk_id_off,
                bool want_text_id_off)
{
  Plan p;
  gtk::EncodeBuffers& b = p.b;
  const int64_t chunk_cap = chunk_upper_bound(n_bytes, n_texts, h->chunk_tokens);
  const int64_t n_tiles = (n_bytes + gtk::kTile - 1) / gtk::kTile;
  p.chunk_cap = chunk_cap;
  h->d_text_chunk_base.reserve(size_t(n_texts + 1) * 8);
  if (kernels == Kernels::tiles) {
    h->d_tile_info.reserve(size_t(n_tiles + 1) * sizeof(gtk::TileInfo));
    h->d_chunk_rel.reserve(size_t(chunk_cap + 1) * 4);
    h->d_text_rel.reserve(size_t(n_texts + 1) * 4);
    h->d_group_base.reserve(size_t(n_tiles / gtk::kTileGroup + 2) * 8);
    h->d_unit_first.reserve(size_t(n_tiles + 1) * 8);
    h->d_unit_cnt.reserve(size_t(n_tiles + 1) * 4);
  } else {
    h->d_chunk_off.reserve(size_t(chunk_cap + 1) * 8);
    h->d_chunk_cnt.reserve(size_t(chunk_cap + 1) * 4);
    h->d_tile_chunk0.reserve(size_t(gtk::kSmallMaxBytes / gtk::kTile + 1) * 4);
  }
  if (kernels != Kernels::small) h->d_staging.reserve(size_t(n_bytes + 16) * 2);
  if (!d_chunk_id_off) {
    h->d_chunk_id_off.reserve(size_t(chunk_cap + 1) * 8);
    d_chunk_id_off = h->d_chunk_id_off.as<int64_t>();
  }
  if (want_text_id_off) h->d_text_id_off.reserve(size_t(n_texts + 1) * 8);
  const int64_t scan_items = std::max<int64_t>(std::max(chunk_cap, n_tiles), n_texts);
  h->d_scan_sums.reserve(size_t(scan_items / 4096 + 2) * 8);
  // [0] n_chunks, [1] n_ids as int64, then the 16 int32 counters (one copy brings both) and the group counts
  h->d_totals.reserve(80 + size_t(n_tiles / gtk::kTileGroup + 1) * 4);
  // workspace for segments / chunks that do not fit in shared memory
  const int64_t longest = std::min<int64_t>(h->chunk_tokens, n_bytes);
  int64_t scratch_tokens = 0;
  if (longest > gtk::kHalo) scratch_tokens = (longest + 63) & ~int64_t(63);
  const int ctas = std::max(h->opt_grid, std::max(h->base_grid, h->localmin_grid));
  if (scratch_tokens && !h->wide) h->d_seg_scratch.reserve(size_t(ctas) * 2 * size_t(scratch_tokens) * 2);
  if (h->wide) {
    h->d_staging32.reserve(size_t(n_bytes + 16) * 4);
    if (scratch_tokens) h->d_seg_scratch32.reserve(size_t(h->wide_grid) * 2 * size_t(scratch_tokens) * 4);
  }

  b.bytes = d_bytes;
  b.n_bytes = n_bytes;
  b.text_off = d_text_off;
  b.n_texts = n_texts;
  b.chunk_bytes = h->chunk_tokens;
  b.text_chunk_base = h->d_text_chunk_base.as<int64_t>();
  b.chunk_off = h->d_chunk_off.as<int64_t>();
  b.chunk_cap = chunk_cap;
  b.tile_chunk0 = h->d_tile_chunk0.as<int32_t>();
  b.n_tiles = n_tiles;
  b.staging = h->d_staging.as<uint16_t>();
  b.unit_first = h->d_unit_first.as<int64_t>();
  b.unit_cnt = h->d_unit_cnt.as<int32_t>();
  b.chunk_cnt = h->d_chunk_cnt.as<int32_t>();
  b.tile_info = h->d_tile_info.as<gtk::TileInfo>();
  b.chunk_rel = h->d_chunk_rel.as<int32_t>();
  b.text_rel = h->d_text_rel.as<int32_t>();
  b.group_base = h->d_group_base.as<int64_t>();
  b.chunk_id_off = d_chunk_id_off;
  b.text_id_off = want_text_id_off ? h->d_text_id_off.as<int64_t>() : nullptr;
  b.out_ids = d_out_ids;
  b.out_capacity = out_capacity;
  b.seg_scratch = (scratch_tokens && !h->wide) ? h->d_seg_scratch.as<uint16_t>() : nullptr;
  b.seg_scratch32 = (scratch_tokens && h->wide) ? h->d_seg_scratch32.as<uint32_t>() : nullptr;
  b.staging32 = h->wide ? h->d_staging32.as<int32_t>() : nullptr;
  b.seg_scratch_tokens = scratch_tokens;
  b.scan_block_sums = h->d_scan_sums.as<int64_t>();
  b.totals = h->d_totals.as<int64_t>();
  b.counters = reinterpret_cast<int32_t*>(b.totals + 2);
  b.group_cnt = b.counters + 16;
  b.ticket = b.counters;
  b.tile_hi = n_tiles;
  b.low_id_map = (h->id_space == GTK_IDS_GPT2) ? h->d_low_map.as<uint16_t>() : nullptr;
  return p;
}

const char* status_text(int s)
{
  switch (s) {
    case gtk::kStatusLongQueueOverflow: return "long-segment queue overflow";
    case gtk::kStatusScratchTooSmall: return "segment workspace too small";
    case gtk::kStatusBadSegment: return "merge pass made no progress";
    case gtk::kStatusBadOffsets: return "chunk offsets outside the text";
    default: return "unknown kernel status";
  }
}

// The kernels that work chunk by chunk (GTK_MODE_BASE, GTK_MODE_LOCALMIN, tables beyond 16 bits).
// Chunker -> merge -> scans.  Leaves totals (n_chunks, n_ids) and the status
// word in the pinned totals buffer; the caller synchronises and then packs.
// n_chunks, n_ids and the status word to the host: totals and counters are adjacent in the handle's own arena
void copy_totals(gtk_tokenizer* h, const gtk::EncodeBuffers& b, int64_t* pinned_totals, cudaStream_t s)
{
  int64_t* ht = pinned_totals ? pinned_totals : h->h_totals.as<int64_t>();
  if (reinterpret_cast<const int64_t*>(b.counters) == b.totals + 2) {
    GTK_CUDA(cudaMemcpyAsync(ht, b.totals, 32, cudaMemcpyDeviceToHost, s));
  } else {
    GTK_CUDA(cudaMemcpyAsync(ht, b.totals, 16, cudaMemcpyDeviceToHost, s));
    GTK_CUDA(cudaMemcpyAsync(ht + 2, b.counters, 16, cudaMemcpyDeviceToHost, s));
  }
}

// chained: the pack follows on the same stream without a host round trip, so that one event pair around both
// times the pipeline when the stages are not timed one by one.
void run_front(gtk_tokenizer* h, const gtk::EncodeBuffers& b, int mode, int* launches, cudaEvent_t* ev = nullptr,
               int64_t* pinned_totals = nullptr, int64_t* mapped_totals = nullptr, bool chained = false)
{
  cudaStream_t s = h->stream;
  const bool stages = ev != nullptr || h->stage_timing;  // sliced batches always time their stages
  if (!ev) ev = h->ev;
  if (!gtk::chunker_resets_counters(b)) {
    GTK_CUDA(cudaMemsetAsync(b.counters, 0, 64, s));
    GTK_CUDA(cudaMemsetAsync(b.chunk_cnt, 0, size_t(b.chunk_cap + 1) * 4, s));
  }
  GTK_CUDA(cudaEventRecord(ev[0], s));
  *launches += gtk::launch_chunker(b, s);
  if (stages) GTK_CUDA(cudaEventRecord(ev[1], s));
  if (h->wide) *launches += gtk::launch_merge_wide(b, h->dtab, h->wide_grid, s);
  else if (mode == GTK_MODE_BASE) *launches += gtk::launch_merge_base(b, h->dtab, h->base_grid, h->base_block, s);
  else *launches += gtk::launch_merge_localmin(b, h->dtab, h->localmin_grid, h->max_iters, s);
  if (stages) GTK_CUDA(cudaEventRecord(ev[2], s));
  *launches += gtk::launch_output_scans(b, s);
  if (stages || !chained) GTK_CUDA(cudaEventRecord(ev[3], s));
  GTK_CUDA(cudaGetLastError());
  if (mapped_totals) {  // one small kernel writes the four words into mapped host memory: no copy-engine round trips
    *launches += gtk::launch_publish_totals(b, mapped_totals, s);
    return;
  }
  if (chained) return;  // the totals travel behind the pack (run_pack), which does not have to wait for them
  copy_totals(h, b, pinned_totals, s);
}

void run_pack(gtk_tokenizer* h, const gtk::EncodeBuffers& b, int* launches, cudaEvent_t* ev = nullptr,
              cudaStream_t on = nullptr, bool chained = false, bool totals_by_copy = true)
{
  cudaStream_t s = on ? on : h->stream;
  const bool stages = ev != nullptr || h->stage_timing;
  if (!ev) ev = h->ev;
  if (stages || !chained) GTK_CUDA(cudaEventRecord(ev[5], s));
  if (h->wide) *launches += gtk::launch_pack_wide(b, h->sm_count * 8, s);
  else *launches += gtk::launch_pack_chunks(b, h->sm_count * 8, s);
  GTK_CUDA(cudaEventRecord(ev[4], s));
  GTK_CUDA(cudaGetLastError());
  if (chained && totals_by_copy) copy_totals(h, b, nullptr, s);
}

// What comes in front of the tile kernel: reset, scan of the texts, tile records.
void begin_tiles(gtk_tokenizer* h, const gtk::EncodeBuffers& b, int* launches)
{
  const bool learned = h->call_tab.learn != 0;
  *launches += gtk::launch_begin_batch(b, h->dtab.long_words, learned ? h->call_tab.long_words : nullptr, h->stream);
  *launches += gtk::launch_scan_texts(b, learned, h->stream) + gtk::launch_tile_info(b, h->stream);
}

// All kernels of a batch in GTK_MODE_OPT.  `ready`: counters, group counts, scanned chunk counts and tile records are in place already.  The pack kernel publishes the totals (see
// launch_pack_tiles).  The events between the stages are recorded when they are asked for.
void run_tiles(gtk_tokenizer* h, const gtk::EncodeBuffers& b, bool ready, int64_t* publish, int64_t seq, int* launches)
{
  cudaStream_t s    = h->stream;
  const bool stages = h->stage_timing;
  cudaEvent_t* ev   = h->ev;
  if (stages) GTK_CUDA(cudaEventRecord(ev[0], s));
  if (!ready) begin_tiles(h, b, launches);
  if (stages) GTK_CUDA(cudaEventRecord(ev[1], s));
  *launches += gtk::launch_merge_opt(b, h->call_tab, h->opt_grid, s);
  if (stages) GTK_CUDA(cudaEventRecord(ev[2], s));
  const int scanned = ready ? 0 : gtk::launch_scan_groups(b, s);
  if (stages)
    for (int i : {3, 5}) GTK_CUDA(cudaEventRecord(ev[i], s));
  *launches += scanned + gtk::launch_pack_tiles(b, h->sm_count, scanned != 0, publish, seq, s);
  if (stages) GTK_CUDA(cudaEventRecord(ev[4], s));
  GTK_CUDA(cudaGetLastError());
}

// Adds the stage times of one pipeline run (one batch, or one slice) to h->stage_ms.  The events must have
// completed and must not have been recorded again since: the sliced path therefore reads the front events
// of a slice as soon as its front has finished (its arena's events are recorded again for a later slice
// soon after) and the pack events when its ids have arrived.
void collect_front_times(gtk_tokenizer* h, cudaEvent_t* ev = nullptr)
{
  const bool stages = ev != nullptr || h->stage_timing;
  if (!ev) ev = h->ev;
  float ms = 0;
  if (!stages) {  // chunker, merge and scans as one interval
    GTK_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[3]));
    h->front_ms = ms;
    return;
  }
  h->front_ms = -1.f;
  for (int i = 0; i < 3; ++i) {
    GTK_CUDA(cudaEventElapsedTime(&ms, ev[i], ev[i + 1]));
    h->stage_ms[i] += ms;
  }
}

void collect_pack_time(gtk_tokenizer* h, cudaEvent_t* ev = nullptr)
{
  if (!ev) ev = h->ev;
  float ms = 0;
  GTK_CUDA(cudaEventElapsedTime(&ms, ev[5], ev[4]));
  // the pipeline time excludes the host round trip between scans and pack
  if (h->front_ms >= 0.f) {
    h->stage_ms[4] = h->front_ms + ms;
    return;
  }
  h->stage_ms[3] += ms;
  h->stage_ms[4] = h->stage_ms[0] + h->stage_ms[1] + h->stage_ms[2] + h->stage_ms[3];
}

void collect_stage_times(gtk_tokenizer* h, bool chained = false)
{
  if (chained && !h->stage_timing) {  // one event pair around the whole pipeline
    GTK_CUDA(cudaEventElapsedTime(&h->stage_ms[4], h->ev[0], h->ev[4]));
    return;
  }
  collect_front_times(h);
  collect_pack_time(h);
}


// ------------------------------------------------------------------------------------------------
// Large host batches: cut the batch into slices of whole chunks and overlap, per slice, the
// host->device copy, the kernel pipeline and the device->host copy of the results on three
// streams.  A slice is an independent sub-batch (its pieces are texts or chunk-aligned parts of a
// text), so the per-chunk results are exactly those of the unsliced batch.
// ------------------------------------------------------------------------------------------------
const char* const kWideNoLocalmin =
    "the local-minimum mode is not offered for merge tables with ids >= 65535 or ranks >= 65534";
// smaller batches take the single-shot path; from 8 MiB on the overlap of a few slices (6 + 2 MiB at the least) wins:
// 8 / 16 / 23 MiB in 0.50 / 0.88 / 1.11 ms against 0.56 / 0.97 / 1.33 ms unsliced
constexpr int64_t kSliceThresholdBytes = int64_t(8) << 20;
constexpr int64_t kSliceTargetBytes    = int64_t(24) << 20;  // measured best of 16..40 MiB on config 2 (256 MiB)

struct SlicePlan {
  int64_t byte_lo = 0, byte_hi = 0;
  std::vector<int64_t> piece_off;    // [P+1], relative to byte_lo
  std::vector<int64_t> first_text;   // [P]: text index if the piece starts a text, else -1
};

// Size of the slice that starts at byte `lo` of a batch of `total` bytes: full-size slices in the middle,
// smaller ones at both ends (a quarter, then half; for batches of two full slices and more an eighth first), because
// the first slice's upload and kernels and the last slice's download are the part of the call that nothing overlaps.
int64_t slice_target(int64_t lo, int64_t total, int64_t full)
{
  if (total >= 2 * full) {  // large batches: three steps at both ends, an eighth, a quarter, a half (256 MiB: 8.03 against 8.11 ms)
    const int64_t e = full / 8, rem = total - lo;
    int64_t t = (lo < e) ? e : (lo < 3 * e) ? 2 * e : (lo < 7 * e) ? 4 * e : full;
    if (rem <= e) t = rem;
    else if (rem <= 3 * e) t = std::min(t, rem - e);
    else if (rem <= 7 * e) t = std::min(t, rem - 3 * e);
    else if (rem <= 7 * e + full) t = std::min(t, std::max(rem - 7 * e, e));
    return std::max<int64_t>(t, 1);
  }
  const int64_t q = full / 4, rem = total - lo;
  int64_t t = (lo < q) ? q : (lo < 3 * q) ? 2 * q : full;
  if (rem <= q) t = rem;
  else if (rem <= 3 * q) t = std::min(t, rem - q);
  else if (rem <= 3 * q + full) t = std::min(t, std::max(rem - 3 * q, q));
  return std::max<int64_t>(t, 1);
}

std::vector<SlicePlan> plan_slices(const int64_t* text_off, int64_t n_texts, int chunk, int64_t full)
{
  const int64_t total = n_texts > 0 ? text_off[n_texts] : 0;
  int64_t target = slice_target(0, total, full);
  std::vector<SlicePlan> out;
  SlicePlan cur;
  cur.piece_off.push_back(0);
  auto close = [&](int64_t at) {
    cur.byte_hi = at;
    out.push_back(std::move(cur));
    cur = SlicePlan();
    cur.byte_lo = at;
    cur.piece_off.push_back(0);
    target = slice_target(at, total, full);
  };
  for (int64_t t = 0; t < n_texts; ++t) {
    int64_t pos = text_off[t];
    const int64_t end = text_off[t + 1];
    bool first = true;
    do {
      const int64_t used = pos - cur.byte_lo;
      int64_t take = end - pos;
      if (used + take > target && take > 0) {
        const int64_t room_chunks = (target - used) / chunk;
        if (room_chunks <= 0 && used > 0) {  // slice is full: start a new one and retry
          close(pos);
          continue;
        }
        take = std::min<int64_t>(take, std::max<int64_t>(room_chunks, 1) * chunk);
      }
      cur.piece_off.push_back(pos + take - cur.byte_lo);
      cur.first_text.push_back(first ? t : -1);
      first = false;
      pos += take;
      if (pos - cur.byte_lo >= target) close(pos);
    } while (pos < end);
  }
  if (cur.piece_off.size() > 1) close(text_off[n_texts]);
  return out;
}

void slice_arena_prepare(gtk_tokenizer* h, SliceArena& a, int64_t max_bytes, int64_t max_pieces)
{
  const int64_t chunk_cap = chunk_upper_bound(max_bytes, max_pieces, h->chunk_tokens);
  a.text_chunk_base.reserve(size_t(max_pieces + 1) * 8);
  a.chunk_off.reserve(size_t(chunk_cap + 1) * 8);
  a.chunk_cnt.reserve(size_t(chunk_cap + 1) * 4);
  a.scan_sums.reserve(size_t(std::max(chunk_cap, max_pieces) / 4096 + 2) * 8);
  a.counters.reserve(64);
  a.totals.reserve(64);
  a.h_totals.reserve_mapped(64);
  for (auto& e : a.ev)
    if (!e) GTK_CUDA(cudaEventCreate(&e));
  for (cudaEvent_t* e : {&a.ev_in, &a.ev_front, &a.ev_packed, &a.ev_out})
    if (!*e) GTK_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
}

// Device offset of slice i inside the batch-wide byte / staging / id buffers: 16-element aligned
// (vector loads) and spaced so that neighbouring slices never share an element.
inline int64_t slice_dev_offset(const SlicePlan& sp, int index) { return (sp.byte_lo + 16 * int64_t(index) + 15) & ~int64_t(15); }

gtk::EncodeBuffers slice_buffers(gtk_tokenizer* h, SliceArena& a, const SlicePlan& sp, int index, int64_t max_bytes)
{
  gtk::EncodeBuffers b{};
  const int64_t dev_off = slice_dev_offset(sp, index);
  const int64_t n_bytes = sp.byte_hi - sp.byte_lo;
  const int64_t pieces  = int64_t(sp.piece_off.size()) - 1;
  b.bytes = h->d_bytes.as<uint8_t>() + dev_off;
  b.n_bytes = n_bytes;
  b.text_off = nullptr;  // the three offset arrays are set by the caller (batch-wide buffers)
  b.n_texts = pieces;
  b.chunk_bytes = h->chunk_tokens;
  b.text_chunk_base = a.text_chunk_base.as<int64_t>();
  b.chunk_off = a.chunk_off.as<int64_t>();
  b.chunk_cap = chunk_upper_bound(n_bytes, pieces, h->chunk_tokens);
  b.n_tiles = (n_bytes + gtk::kTile - 1) / gtk::kTile;
  b.staging = h->d_staging.as<uint16_t>() + dev_off;
  b.chunk_cnt = a.chunk_cnt.as<int32_t>();
  b.chunk_id_off = nullptr;
  b.text_id_off = nullptr;
  b.out_ids = h->d_out_ids.as<int32_t>() + dev_off;  // worst case one id per byte: slices never overlap
  b.out_capacity = n_bytes;
  const int64_t longest = std::min<int64_t>(h->chunk_tokens, n_bytes);
  const int64_t scratch_tokens = longest > gtk::kHalo ? ((longest + 63) & ~int64_t(63)) : 0;
  b.seg_scratch = (scratch_tokens && !h->wide) ? h->d_seg_scratch.as<uint16_t>() : nullptr;
  b.seg_scratch32 = (scratch_tokens && h->wide) ? h->d_seg_scratch32.as<uint32_t>() : nullptr;
  b.staging32 = h->wide ? h->d_staging32.as<int32_t>() + dev_off : nullptr;
  b.seg_scratch_tokens = scratch_tokens;
  b.scan_block_sums = a.scan_sums.as<int64_t>();
  b.counters = a.counters.as<int32_t>();
  b.totals = a.totals.as<int64_t>();
  b.low_id_map = (h->id_space == GTK_IDS_GPT2) ? h->d_low_map.as<uint16_t>() : nullptr;
  return b;
}


int encode_host_sliced(gtk_tokenizer* h, int mode, const uint8_t* bytes, const int64_t* text_offsets,
                       int64_t n_texts, int64_t n_bytes, float* kernel_ms)
{
  const std::vector<SlicePlan> slices = plan_slices(text_offsets, n_texts, h->chunk_tokens, kSliceTargetBytes);
  const int ns     = int(slices.size());
  const size_t nsz = size_t(ns);
  // Offsets travel once per batch, not once per slice: the piece offsets of all slices go up in one copy
  // before the first slice, the per-piece and per-chunk id offsets of all slices come back in two copies
  // after the last one.  Slice i owns entries [piece_at[i], piece_at[i+1]) and [chunk_at[i], chunk_at[i+1]).
  std::vector<int64_t> piece_at(nsz + 1, 0), chunk_at(nsz + 1, 0);
  int64_t max_bytes = 0, max_pieces = 0;
  for (int i = 0; i < ns; ++i) {
    const SlicePlan& sp  = slices[size_t(i)];
    const int64_t pieces = int64_t(sp.piece_off.size()) - 1;
    max_bytes  = std::max(max_bytes, sp.byte_hi - sp.byte_lo);
    max_pieces = std::max(max_pieces, pieces);
    piece_at[size_t(i) + 1] = piece_at[size_t(i)] + pieces + 1;
    chunk_at[size_t(i) + 1] = chunk_at[size_t(i)] + chunk_upper_bound(sp.byte_hi - sp.byte_lo, pieces, h->chunk_tokens) + 1;
  }
  const int64_t total_pieces = piece_at[nsz] - ns;
  // everything is sized before the first copy is issued: nothing may be reallocated in flight
  const size_t span = size_t(n_bytes) + 16 * size_t(ns) + 64;  // slices sit at 16-aligned, disjoint offsets
  h->d_bytes.reserve(span);
  h->d_staging.reserve(span * 2);
  h->d_out_ids.reserve(span * 4);
  {
    const int64_t longest = std::min<int64_t>(h->chunk_tokens, max_bytes);
    if (h->wide) {
      h->d_staging32.reserve(span * 4);
      if (longest > gtk::kHalo)
        h->d_seg_scratch32.reserve(size_t(h->wide_grid) * 2 * size_t((longest + 63) & ~int64_t(63)) * 4);
    } else if (longest > gtk::kHalo)
      h->d_seg_scratch.reserve(size_t(std::max(h->opt_grid, std::max(h->base_grid, h->localmin_grid))) * 2 * size_t((longest + 63) & ~int64_t(63)) * 2);
  }
  h->d_piece_off.reserve(size_t(piece_at[nsz]) * 8);
  h->d_piece_id_off.reserve(size_t(piece_at[nsz]) * 8);
  h->d_chunk_id_all.reserve(size_t(chunk_at[nsz]) * 8);
  h->h_piece_off.reserve(size_t(piece_at[nsz]) * 8);
  h->h_piece_id_off.reserve(size_t(piece_at[nsz]) * 8);
  h->h_chunk_id_all.reserve(size_t(chunk_at[nsz]) * 8);
  h->pool->reserve(h->h_text_id_off, size_t(n_texts + 1) * 8);
  h->pool->reserve(h->h_chunk_id_off, size_t(chunk_upper_bound(n_bytes, total_pieces, h->chunk_tokens) + 2) * 8);
  h->pool->reserve(h->h_ids, size_t(n_bytes) * 2);  // grown below if the batch yields more than one id per two bytes
  if (!h->in_stream) GTK_CUDA(cudaStreamCreateWithFlags(&h->in_stream, cudaStreamNonBlocking));
  if (!h->out_stream) GTK_CUDA(cudaStreamCreateWithFlags(&h->out_stream, cudaStreamNonBlocking));
  if (!h->pack_stream) GTK_CUDA(cudaStreamCreateWithFlags(&h->pack_stream, cudaStreamNonBlocking));
  for (auto& a : h->slice) slice_arena_prepare(h, a, max_bytes, max_pieces);
  GTK_CUDA(cudaStreamSynchronize(h->stream));

  for (int i = 0; i < ns; ++i) {
    const SlicePlan& sp = slices[size_t(i)];
    std::memcpy(h->h_piece_off.as<int64_t>() + piece_at[size_t(i)], sp.piece_off.data(), sp.piece_off.size() * 8);
  }
  GTK_CUDA(cudaMemcpyAsync(h->d_piece_off.p, h->h_piece_off.p, size_t(piece_at[nsz]) * 8, cudaMemcpyHostToDevice,
                           h->in_stream));

  std::vector<gtk::EncodeBuffers> bufs(nsz);
  std::vector<int64_t> sl_c(nsz), sl_r(nsz), sl_cbase(nsz);
  int launches = 0;
  int64_t R = 0, Cbase = 0;

  auto issue_front = [&](int i) {
    SliceArena& a = h->slice[i % kSliceArenas];
    const SlicePlan& sp = slices[size_t(i)];
    GTK_CUDA(cudaMemcpyAsync(h->d_bytes.as<uint8_t>() + slice_dev_offset(sp, i), bytes + sp.byte_lo, size_t(sp.byte_hi - sp.byte_lo),
                             cudaMemcpyHostToDevice, h->in_stream));
    GTK_CUDA(cudaEventRecord(a.ev_in, h->in_stream));
    GTK_CUDA(cudaStreamWaitEvent(h->stream, a.ev_in, 0));
    if (i >= kSliceArenas) GTK_CUDA(cudaStreamWaitEvent(h->stream, a.ev_out, 0));  // its previous slice has left this arena
    gtk::EncodeBuffers& b = bufs[size_t(i)];
    b = slice_buffers(h, a, sp, i, max_bytes);
    b.text_off     = h->d_piece_off.as<int64_t>() + piece_at[size_t(i)];
    b.text_id_off  = h->d_piece_id_off.as<int64_t>() + piece_at[size_t(i)];
    b.chunk_id_off = h->d_chunk_id_all.as<int64_t>() + chunk_at[size_t(i)];
    // the result words reach the host through mapped memory
    run_front(h, b, mode, &launches, a.ev, nullptr, static_cast<int64_t*>(a.h_totals.dp));
    GTK_CUDA(cudaEventRecord(a.ev_front, h->stream));
  };
  auto finish = [&](int i) {  // the ids of slice i are on the host
    SliceArena& a = h->slice[i % kSliceArenas];
    GTK_CUDA(cudaEventSynchronize(a.ev_out));
    collect_pack_time(h, a.ev);
  };
  auto sync_all = [&] {
    cudaStreamSynchronize(h->in_stream);
    cudaStreamSynchronize(h->stream);
    cudaStreamSynchronize(h->pack_stream);
    cudaStreamSynchronize(h->out_stream);
  };

  constexpr int kAhead = kSliceArenas - 1;  // fronts queued ahead of the slice being packed
  for (int i = 0; i < std::min(ns, kAhead); ++i) issue_front(i);
  for (int i = 0; i < ns; ++i) {
    SliceArena& a = h->slice[i % kSliceArenas];
    if (i >= 2) finish(i - 2);
    GTK_CUDA(cudaEventSynchronize(a.ev_front));
    collect_front_times(h, a.ev);
    const int64_t* ht = a.h_totals.as<int64_t>();
    const int64_t C = ht[0], N = ht[1];
    const int status = reinterpret_cast<const int32_t*>(ht + 2)[1];
    if (status != gtk::kStatusOk) {
      sync_all();
      return h->fail(GTK_ERR_KERNEL, status_text(status));
    }
    if (size_t(R + N + 1) * 4 > h->h_ids.cap) {  // grow the pinned id buffer, keeping what has arrived
      GTK_CUDA(cudaStreamSynchronize(h->out_stream));
      PinBuf bigger;
      bigger.reserve(std::max(size_t(R + N + 1) * 4 * 2, h->h_ids.cap * 2));
      std::memcpy(bigger.p, h->h_ids.p, size_t(R) * 4);
      h->h_ids.release();
      h->h_ids = bigger;
    }
    // the pack runs on a stream of its own: the compute stream already holds the fronts of later slices
    GTK_CUDA(cudaStreamWaitEvent(h->pack_stream, a.ev_front, 0));
    run_pack(h, bufs[size_t(i)], &launches, a.ev, h->pack_stream);
    GTK_CUDA(cudaEventRecord(a.ev_packed, h->pack_stream));
    GTK_CUDA(cudaStreamWaitEvent(h->out_stream, a.ev_packed, 0));
    GTK_CUDA(cudaMemcpyAsync(h->h_ids.as<int32_t>() + R, bufs[size_t(i)].out_ids, size_t(N) * 4, cudaMemcpyDeviceToHost,
                             h->out_stream));
    GTK_CUDA(cudaEventRecord(a.ev_out, h->out_stream));
    sl_c[size_t(i)]     = C;
    sl_r[size_t(i)]     = R;
    sl_cbase[size_t(i)] = Cbase;
    R += N;
    Cbase += C;
    if (i + kAhead < ns) issue_front(i + kAhead);
  }
  // offsets of all slices in two copies behind the last ids
  GTK_CUDA(cudaMemcpyAsync(h->h_piece_id_off.p, h->d_piece_id_off.p, size_t(piece_at[nsz]) * 8, cudaMemcpyDeviceToHost,
                           h->out_stream));
  GTK_CUDA(cudaMemcpyAsync(h->h_chunk_id_all.p, h->d_chunk_id_all.p, size_t(chunk_at[nsz]) * 8, cudaMemcpyDeviceToHost,
                           h->out_stream));
  for (int i = std::max(0, ns - 2); i < ns; ++i) finish(i);
  GTK_CUDA(cudaStreamSynchronize(h->out_stream));
  GTK_CUDA(cudaStreamSynchronize(h->stream));
  // per-slice offsets start at 0: add the ids that precede the slice.  A text that starts exactly where the
  // previous slice ended belongs to the slice that holds its first piece.
  int64_t* h_text  = h->h_text_id_off.as<int64_t>();
  int64_t* h_chunk = h->h_chunk_id_off.as<int64_t>();
  for (int i = 0; i < ns; ++i) {
    const SlicePlan& sp = slices[size_t(i)];
    const int64_t base  = sl_r[size_t(i)];
    const int64_t* pid  = h->h_piece_id_off.as<int64_t>() + piece_at[size_t(i)];
    for (size_t p = 0; p < sp.first_text.size(); ++p)
      if (sp.first_text[p] >= 0) h_text[sp.first_text[p]] = base + pid[p];
    const int64_t* src = h->h_chunk_id_all.as<int64_t>() + chunk_at[size_t(i)];
    int64_t* dst       = h_chunk + sl_cbase[size_t(i)];
    for (int64_t c = 0; c < sl_c[size_t(i)]; ++c) dst[c] = src[c] + base;
  }
  h_chunk[Cbase] = R;
  h_text[n_texts] = R;
  h->last_launches = launches;
  h->res_n_ids = R;
  h->res_n_chunks = Cbase;
  h->result_bufs[0] = &h->h_ids;
  h->result_bufs[1] = &h->h_text_id_off;
  h->result_bufs[2] = &h->h_chunk_id_off;
  if (kernel_ms) *kernel_ms = h->stage_ms[4];
  return GTK_OK;
}


// ------------------------------------------------------------------------------------------------
// Small host batches (latency mode): the text is copied into mapped page-locked memory, one
// single-CTA kernel reads it over PCIe and writes ids and offsets straight back into mapped
// memory; the call is one launch plus one stream synchronisation.
// ------------------------------------------------------------------------------------------------
constexpr size_t kSmallInOff    = 0;
constexpr size_t kSmallInBytes  = ((size_t(gtk::kSmallMaxTexts) + 1) * 8 + 63) & ~size_t(63);
constexpr size_t kSmallInSize   = kSmallInBytes + size_t(gtk::kSmallMaxBytes) + 64;
constexpr int64_t kSmallChunkCap = gtk::kSmallMaxBytes + gtk::kSmallMaxTexts + 2;
constexpr size_t kSmallOutTotals = 0;
constexpr size_t kSmallOutText   = 64;
constexpr size_t kSmallOutChunk  = kSmallOutText + (((size_t(gtk::kSmallMaxTexts) + 1) * 8 + 63) & ~size_t(63));
constexpr size_t kSmallOutIds    = kSmallOutChunk + (((size_t(kSmallChunkCap) + 1) * 8 + 63) & ~size_t(63));
constexpr size_t kSmallOutSize   = kSmallOutIds + size_t(gtk::kSmallMaxBytes) * 4 + 64;
// Host batches of the chunk-by-chunk modes up to this size: a kernel writes the results into a mapped block instead of two copies
// bringing them.  By kernel / by copies, 64 KiB, 256 KiB, 1, 2, 4 MiB of the novel in GTK_MODE_BASE: 111 / 126, 99 / 111, 140 / 153,
// 198 / 208, 344 / 349 us; GTK_MODE_LOCALMIN 105 / 115, 92 / 108, 147 / 162, 235 / 244, 410 / 414.  The kernel is ahead at every size
// measured, by 12 % up to 1 MiB and by 1 % at 4 MiB; the block needs five bytes of page-locked memory per byte of text, so
// it ends where the gain does.
constexpr int64_t kResultsByKernelMaxBytes = int64_t(1) << 20;
constexpr size_t kMappedResultBytes        = size_t(6) << 20;

void small_path_init(gtk_tokenizer* h)
{
  void *ih = nullptr, *oh = nullptr, *id = nullptr, *od = nullptr;
  GTK_CUDA(cudaHostAlloc(&ih, kSmallInSize, cudaHostAllocMapped));
  GTK_CUDA(cudaHostAlloc(&oh, kSmallOutSize, cudaHostAllocMapped));
  GTK_CUDA(cudaHostGetDevicePointer(&id, ih, 0));
  GTK_CUDA(cudaHostGetDevicePointer(&od, oh, 0));
  std::memset(oh, 0, 64);  // the completion mark of the result block starts at call number 0
  h->small_in_h = static_cast<uint8_t*>(ih);
  h->small_out_h = static_cast<uint8_t*>(oh);
  h->small_in_d = static_cast<uint8_t*>(id);
  h->small_out_d = static_cast<uint8_t*>(od);
}

// The mapped result block, its completion mark behind any call number that is still to come.
uint8_t* mid_block(gtk_tokenizer* h)
{
  h->pool->reserve(h->h_mid, kMappedResultBytes);
  std::memset(h->h_mid.p, 0, 64);
  return h->h_mid.as<uint8_t>();
}

// Waits for a kernel's completion mark (the call number, its last store behind a system-wide fence) in a mapped
// result block: returns as soon as the results are on the host, several microseconds before a stream
// synchronisation would.  The stream is asked now and then so that a failed launch or a fault ends the wait
// with its error.  false: the stream went idle without the mark.
bool wait_for_mark(volatile const int64_t* mark, int64_t seq, cudaStream_t s, const char* what)
{
  for (unsigned spin = 1; *mark != seq; ++spin) {
    if ((spin & 0xFFFFu) == 0u) {
      const cudaError_t q = cudaStreamQuery(s);
      if (q == cudaSuccess) return *mark == seq;
      if (q != cudaErrorNotReady) throw CudaFail{std::string(what) + ": " + cudaGetErrorString(q)};
    }
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#endif
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return true;
}

// memcpy past the caches: what is written here is read next by the copy engine, not by a core.
void copy_to_staging(uint8_t* to, const uint8_t* from, size_t n)
{
#if defined(__x86_64__)
  if (n == 0) return;
  const size_t head = std::min(n, size_t(-reinterpret_cast<uintptr_t>(to) & 15u));
  std::memcpy(to, from, head);
  size_t i = head;
  for (; i + 64 <= n; i += 64) {
    const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(from + i)), b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(from + i + 16));
    const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(from + i + 32)), d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(from + i + 48));
    _mm_stream_si128(reinterpret_cast<__m128i*>(to + i), a);
    _mm_stream_si128(reinterpret_cast<__m128i*>(to + i + 16), b);
    _mm_stream_si128(reinterpret_cast<__m128i*>(to + i + 32), c);
    _mm_stream_si128(reinterpret_cast<__m128i*>(to + i + 48), d);
  }
  std::memcpy(to + i, from + i, n - i);
  _mm_sfence();  // before the block is reported done
#else
  std::memcpy(to, from, n);
#endif
}

// The text of a call: in one buffer, or every string where it lies (gtk_encode_strings).
struct Source {
  const uint8_t* bytes;         // nullptr: strings
  const uint8_t* const* parts;  // text t is parts[t][0 .. text_offsets[t + 1] - text_offsets[t])
  const int64_t* text_offsets;
  int64_t n_texts;
  bool staged;  // goes through page-locked memory of the handle's: strings, and ordinary memory of a middling size

  void copy_texts(uint8_t* all, int64_t t, int64_t end) const  // to where they belong in the whole
  {
    for (; t < end; ++t)
      if (const size_t n = size_t(text_offsets[t + 1] - text_offsets[t])) std::memcpy(all + text_offsets[t], parts[t], n);
  }
  // the same past the caches: short ones are brought together in a block that stays in the cache first, since lines that are
  // streamed in parts cost more than a copy (5 MB in 10 000 strings 1.37 ms instead of 0.77)
  void stream_texts(uint8_t* all, int64_t t, int64_t end) const
  {
    constexpr int64_t kLong = 16 << 10;
    uint8_t block[3 * kLong];
    for (int64_t from = text_offsets[t]; t < end;) {
      int64_t have = 0, n = 0;
      for (; t < end && have < 2 * kLong && (n = text_offsets[t + 1] - text_offsets[t]) < kLong; ++t) {
        if (n) std::memcpy(block + have, parts[t], size_t(n));
        have += n;
      }
      copy_to_staging(all + from, block, size_t(have));
      from += have;
      if (t < end && n >= kLong) {
        copy_to_staging(all + from, parts[t], size_t(n));
        from += n;
        ++t;
      }
    }
  }
  void copy_all(uint8_t* to) const
  {
    if (bytes) std::memcpy(to, bytes, size_t(text_offsets[n_texts]));
    else copy_texts(to, 0, n_texts);
  }
};

// Brings a staged source together in page-locked memory, block by block and with the crew's help; ready(hi) returns the whole
// buffer once its first hi bytes are there.  Any other source is ready as it is.
class Gather {
 public:
  Gather(gtk_tokenizer* h, const Source& src) : src_(src)
  {
    if (!src.staged) return;
    const int64_t n = src.text_offsets[src.n_texts];
    h->h_gather.reserve(size_t(n));
    to_ = h->h_gather.as<uint8_t>();
    if (src.bytes) {
      for (int64_t at = kBlock; at < n; at += kBlock) end_.push_back(at);
    } else {
      first_.push_back(0);
      for (int64_t t = 1; t < src.n_texts; ++t)
        if (src.text_offsets[t] - src.text_offsets[first_.back()] >= kBlock) {
          first_.push_back(t);
          end_.push_back(src.text_offsets[t]);
        }
      first_.push_back(src.n_texts);
    }
    end_.push_back(n);
    job_.reset(new gtk::Crew::Job(h->crew, int64_t(end_.size()), [this](int64_t i) {
      const int64_t lo = i ? end_[size_t(i) - 1] : 0;
      if (src_.bytes) copy_to_staging(to_ + lo, src_.bytes + lo, size_t(end_[size_t(i)] - lo));
      else src_.stream_texts(to_, first_[size_t(i)], first_[size_t(i) + 1]);
    }));
  }
  const uint8_t* ready(int64_t hi)
  {
    if (!job_) return src_.bytes;
    while (at_ < end_.size() && (at_ ? end_[at_ - 1] : 0) < hi) job_->wait(int64_t(at_++));
    return to_;
  }

 private:
  static constexpr int64_t kBlock = 64 << 10;
  const Source src_;
  uint8_t* to_ = nullptr;
  std::vector<int64_t> end_;    // where the blocks end
  std::vector<int64_t> first_;  // strings: first text of every block
  size_t at_ = 0;
  std::unique_ptr<gtk::Crew::Job> job_;
};

// Ordinary memory from this size on is staged by the crew while the first of it is on the link already; the driver does it
// on one core.  256 KiB / 1 / 4 / 16 / 64 MiB per call: 102 / 149 / 427 / 1204 / 6740 us by the driver, 94 / 122 / 324 / 879 / 3009 staged;
// from page-locked memory 94 / 258 / 787 at 1 / 4 / 16 MiB.  (Staged with stores that go through the caches: 123 / 650 / 1156.)  The upper
// bound limits the page-locked memory that a handle keeps, not the gain: 96 and 160 MiB take 9.9 and 16.7 ms by the driver, 4.1 and
// 6.5 staged.
constexpr int64_t kStageMinBytes = int64_t(512) << 10, kStageMaxBytes = int64_t(64) << 20;

bool is_ordinary_memory(const void* p)
{
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

int encode_host_small(gtk_tokenizer* h, const Source& src, const int64_t* text_offsets, int64_t n_texts,
                      int64_t n_bytes, float* kernel_ms)
{
  std::memcpy(h->small_in_h + kSmallInOff, text_offsets, size_t(n_texts + 1) * 8);
  src.copy_all(h->small_in_h + kSmallInBytes);
  Plan p = plan_batch(h, Kernels::small, h->small_in_d + kSmallInBytes, n_bytes,
                      reinterpret_cast<const int64_t*>(h->small_in_d + kSmallInOff), n_texts,
                      reinterpret_cast<int32_t*>(h->small_out_d + kSmallOutIds), gtk::kSmallMaxBytes,
                      reinterpret_cast<int64_t*>(h->small_out_d + kSmallOutChunk), false);
  p.b.text_id_off = reinterpret_cast<int64_t*>(h->small_out_d + kSmallOutText);
  p.b.totals      = reinterpret_cast<int64_t*>(h->small_out_d + kSmallOutTotals);
  h->d_text_off.reserve((size_t(gtk::kSmallMaxTexts) + 1) * 8);
  p.b.text_off_copy = h->d_text_off.as<int64_t>();
  h->d_chunk_id_off.reserve(size_t(kSmallChunkCap + 1) * 8);
  p.b.chunk_id_mirror = h->d_chunk_id_off.as<int64_t>();
  cudaStream_t s = h->stream;
  p.b.small_seq = ++h->small_seq;
  const int launches = gtk::launch_encode_small(p.b, h->dtab, s);
  GTK_CUDA(cudaGetLastError());
  // The kernel's last store is the call number, behind a system-wide fence: polling it in the mapped result block
  // returns as soon as the results are on the host, several microseconds before a stream synchronisation would.
  // The stream is asked now and then so that a failed launch or a fault ends the wait with its error.
  volatile const int64_t* tot = reinterpret_cast<volatile const int64_t*>(h->small_out_h + kSmallOutTotals);
  if (!wait_for_mark(tot + 3, p.b.small_seq, s, "small-batch kernel"))
    return h->fail(GTK_ERR_KERNEL, "small-batch kernel ended without publishing its results");
  if (tot[2] != gtk::kStatusOk) return h->fail(GTK_ERR_KERNEL, status_text(int(tot[2])));
  h->stage_ms[1] = h->stage_ms[4] = float(double(tot[4]) * 1e-6);  // the kernel's own globaltimer span
  h->last_launches = launches;
  h->result_is_small = true;
  h->res_n_chunks = tot[0];
  h->res_n_ids = tot[1];
  if (kernel_ms) *kernel_ms = h->stage_ms[4];
  return GTK_OK;
}

// Host batches below the slicing threshold (GTK_MODE_OPT, 16-bit table): two launches.  The host scans the chunk counts of
// the texts and sends them with zeroed counters and, up to kTextInHeaderBytes, the text itself in one copy; tile kernel;
// pack kernel, which writes ids and offsets into page-locked memory and then the call number, for which the host waits.
// No chunker, no scan, no copy back, no synchronisation.
constexpr int64_t kTextInHeaderBytes = 64 << 10;
constexpr int64_t kGatherStep        = 512 << 10;  // a staged text goes up in steps of this while the rest is gathered

// The tile records of a batch, as k_tile_info makes them on the device.
void lay_tiles(const int64_t* text_off, const int64_t* chunk_base, int64_t n_texts, int64_t n_bytes, int64_t chunk,
               gtk::TileInfo* out)
{
  int64_t t = 0;  // first text that starts at or behind the tile's first byte
  for (int64_t lo = 0; lo < n_bytes; lo += gtk::kTile) {
    gtk::TileInfo& i = *out++;
    if (n_texts == 1) {
      const uint32_t past = uint32_t(lo) % uint32_t(chunk);
      const int64_t p0    = past ? chunk - past : 0;
      i = gtk::TileInfo{(lo + p0) / chunk, lo > 0, p0 < gtk::kWindow && lo + p0 < n_bytes ? int32_t(p0) : gtk::kTileNoCut,
                        gtk::kTilePlain | (lo > 0 ? gtk::kTileRunsIn : 0)};
      continue;
    }
    while (t < n_texts && text_off[t] < lo) ++t;
    const bool runs_in = t > 0 && text_off[t] > lo;
    i = gtk::TileInfo{chunk_base[t], t, gtk::kTileNoCut, runs_in ? gtk::kTileRunsIn : 0};
    if (!runs_in) continue;
    const int64_t n  = (uint32_t(lo - text_off[t - 1]) + uint32_t(chunk) - 1u) / uint32_t(chunk);
    const int64_t at = text_off[t - 1] + n * chunk;
    if (at < text_off[t]) {
      i.c0 = chunk_base[t - 1] + n;
      if (at - lo < gtk::kWindow) i.p0 = int32_t(at - lo);
    }
    if (text_off[t] >= std::min(lo + gtk::kWindow, n_bytes)) i.flags |= gtk::kTilePlain;
  }
}

int encode_host_tiles(gtk_tokenizer* h, const Source& src, const int64_t* text_offsets, int64_t n_texts, int64_t n_bytes,
                      float* kernel_ms)
{
  auto up = [](size_t x) { return (x + 63) & ~size_t(63); };
  const int64_t chunk = h->chunk_tokens, K = (n_bytes + gtk::kTile - 1) / gtk::kTile;
  const bool one = n_texts == 1, with_text = n_bytes <= kTextInHeaderBytes;
  const size_t o_off = up(16 + 64 + size_t(K / gtk::kTileGroup + 1) * 4), o_base = up(o_off + (one ? 0 : size_t(n_texts + 1) * 8));
  const size_t o_info = up(o_base + (one ? 0 : size_t(n_texts + 1) * 8)), o_text = up(o_info + size_t(K) * sizeof(gtk::TileInfo));
  const size_t header = with_text ? o_text + size_t(n_bytes) : o_text;
  h->h_fast_in.reserve(header + 32);
  h->d_fast_in.reserve(header + 32);
  uint8_t* hp = static_cast<uint8_t*>(h->h_fast_in.p);
  uint8_t* dp = h->d_fast_in.as<uint8_t>();
  cudaStream_t s = h->stream;
  if (!with_text) {
    h->d_bytes.reserve(size_t(n_bytes) + 32);
    Gather gather(h, src);
    const int64_t step = src.staged ? kGatherStep : n_bytes;
    for (int64_t lo = 0; lo < n_bytes; lo += step) {
      const int64_t hi = std::min(lo + step, n_bytes);
      GTK_CUDA(cudaMemcpyAsync(h->d_bytes.as<uint8_t>() + lo, gather.ready(hi) + lo, size_t(hi - lo), cudaMemcpyHostToDevice, s));
    }
  }
  std::memset(hp, 0, o_off);  // totals, counters, group counts
  int64_t C = 0;
  if (one) {
    C = (n_bytes + chunk - 1) / chunk;
  } else {
    std::memcpy(hp + o_off, text_offsets, size_t(n_texts + 1) * 8);
    int64_t* base = reinterpret_cast<int64_t*>(hp + o_base);
    for (int64_t t = 0; t < n_texts; ++t) {  // lengths and chunk size are below 2^31 here: 32-bit divisions
      base[t] = C;
      const uint32_t len = uint32_t(text_offsets[t + 1] - text_offsets[t]);
      C += len <= uint32_t(chunk) ? (len > 0) : (len + uint32_t(chunk) - 1u) / uint32_t(chunk);
    }
    base[n_texts] = C;
  }
  reinterpret_cast<int64_t*>(hp)[0] = C;
  lay_tiles(text_offsets, reinterpret_cast<const int64_t*>(hp + o_base), n_texts, n_bytes, chunk,
            reinterpret_cast<gtk::TileInfo*>(hp + o_info));
  if (with_text) src.copy_all(hp + o_text);
  GTK_CUDA(cudaMemcpyAsync(dp, hp, header, cudaMemcpyHostToDevice, s));

  // [64-byte header | text id offsets | chunk id offsets | ids]
  const size_t text_b = up(size_t(n_texts + 1) * 8), chunk_b = up(size_t(C + 1) * 8);
  // room for the ids: by what this handle has met so far (English has one id in three or four bytes), at most one per byte
  int64_t room = std::min<int64_t>(n_bytes, int64_t(double(n_bytes) * h->ids_per_byte) + 1024);
  begin_call(h, GTK_MODE_OPT, n_bytes);
  int launches = 0;
  Plan p;
  uint8_t* md = nullptr;
  for (int attempt = 0;; ++attempt) {
    h->pool->reserve(h->h_out, 64 + text_b + chunk_b + size_t(room) * 4);
    md = h->h_out.as<uint8_t>();  // page-locked memory has the same address on the device
    std::memset(md, 0, 64);
    p = plan_batch(h, Kernels::tiles, with_text ? dp + o_text : h->d_bytes.as<uint8_t>(), n_bytes, reinterpret_cast<int64_t*>(dp + o_off), n_texts,
                   reinterpret_cast<int32_t*>(md + 64 + text_b + chunk_b), room, reinterpret_cast<int64_t*>(md + 64 + text_b), false);
    p.b.text_id_off     = reinterpret_cast<int64_t*>(md + 64);
    p.b.totals          = reinterpret_cast<int64_t*>(dp);
    p.b.counters        = reinterpret_cast<int32_t*>(dp + 16);
    p.b.group_cnt       = p.b.counters + 16;
    p.b.ticket          = p.b.counters;
    p.b.starts_clock    = true;
    p.b.text_chunk_base = reinterpret_cast<int64_t*>(dp + o_base);
    p.b.tile_info       = reinterpret_cast<gtk::TileInfo*>(dp + o_info);
    const int64_t seq   = ++h->mid_seq;
    if (attempt == 0) {
      run_tiles(h, p.b, true, reinterpret_cast<int64_t*>(md), seq, &launches);
    } else {  // the tokens are still staged: pack them again
      GTK_CUDA(cudaMemsetAsync(p.b.counters + 8, 0, 4, s));
      launches += gtk::launch_pack_tiles(p.b, h->sm_count, false, reinterpret_cast<int64_t*>(md), seq, s);
      GTK_CUDA(cudaGetLastError());
    }
    volatile const int64_t* tot = reinterpret_cast<volatile const int64_t*>(md);
    if (!wait_for_mark(tot + 3, seq, s, "pack kernel"))
      return h->fail(GTK_ERR_KERNEL, "pack kernel ended without publishing its results");
    if (tot[2] != gtk::kStatusOk) return h->fail(GTK_ERR_KERNEL, status_text(int(tot[2])));
    if (tot[0] != C || tot[1] > n_bytes) return h->fail(GTK_ERR_KERNEL, "inconsistent totals");
    h->res_n_ids   = tot[1];
    if (attempt == 0) h->stage_ms[4] = float(double(tot[4]) * 1e-6);  // by the kernels' own clock
    if (h->res_n_ids <= room) break;
    h->ids_per_byte = std::min(1.0, 1.1 * double(h->res_n_ids) / double(n_bytes));
    room = h->res_n_ids;
  }
  if (h->stage_timing) {
    std::fill(h->stage_ms, h->stage_ms + 5, 0.f);
    GTK_CUDA(cudaEventSynchronize(h->ev[4]));
    collect_stage_times(h);
  }
  h->result_is_packed = true;
  h->pack_base        = md + 64;
  h->result_bufs[0]   = &h->h_out;
  h->pack_text_bytes  = text_b;
  h->pack_chunk_bytes = chunk_b;
  h->last_launches    = launches;
  h->res_n_chunks     = C;
  if (kernel_ms) *kernel_ms = h->stage_ms[4];
  return GTK_OK;
}

// Larger host batches (GTK_MODE_OPT, 16-bit table): the text goes up in pieces, and while a piece travels the one before it
// is in the tile and pack kernels and the ids of earlier ones are on their way back.  The pack kernel of a piece knows where
// its ids go; a mark with the id count is left in page-locked memory, where the host polls for it and then sends the ids with
// the copy engine.  (Ids written by the pack kernel itself: 3.8 instead of 3.1 ms for
// 96 MiB, since beside the next piece's tile kernel no pack CTA finds room on an SM.)  Bound by the host link, which carries
// one byte up and 1.0 .. 2.4 bytes of ids down per byte of text.
// While the link is busy every step from one stream to another takes 25 .. 55 us (commands and marks travel behind the
// text), so pieces are few: 96 MiB of the novel 2.70 ms with pieces of 2 .. 12 MiB, 2.76 with 0.5 .. 16 MiB; below 6 MiB the
// single upload of encode_host_tiles is quicker (4 MiB page-locked 256 against 281 us, 7 MiB 431 against 433, from
// ordinary memory 680 against 610).
constexpr int64_t kPiecesMinBytes = int64_t(6) << 20;
constexpr int64_t kPieceMin = int64_t(2) << 20, kPieceMax = int64_t(12) << 20;

// Ends of the pieces: small ones first and last, because the first upload and the last piece's kernels and download are what
// nothing overlaps; whole tile groups.
std::vector<int64_t> piece_ends(int64_t n_bytes)
{
  constexpr int64_t kGroup = int64_t(gtk::kTileGroup) * gtk::kTile;
  std::vector<int64_t> ends;
  for (int64_t at = 0; at < n_bytes;) {
    const int64_t left = n_bytes - at;
    int64_t take = std::max(std::min({std::max(at, kPieceMin), left / 2, kPieceMax}), kPieceMin) / kGroup * kGroup;
    if (left - take < kPieceMin / 2) take = left;
    at += take;
    ends.push_back(at);
  }
  return ends;
}

int encode_host_pieces(gtk_tokenizer* h, const Source& src, const int64_t* text_offsets, int64_t n_texts, int64_t n_bytes,
                       float* kernel_ms)
{
  auto up = [](size_t x) { return (x + 63) & ~size_t(63); };
  const int64_t chunk = h->chunk_tokens, K = (n_bytes + gtk::kTile - 1) / gtk::kTile, groups = K / gtk::kTileGroup + 1;
  int64_t C = 0;
  if (n_texts == 1) {
    C = (n_bytes + chunk - 1) / chunk;
  } else {
    for (int64_t t = 0; t < n_texts; ++t) {
      const int64_t len = text_offsets[t + 1] - text_offsets[t];
      C += len <= chunk ? (len > 0) : (len + chunk - 1) / chunk;
    }
  }
  const std::vector<int64_t> ends = piece_ends(n_bytes);
  const size_t np = ends.size();
  const size_t text_b = up(size_t(n_texts + 1) * 8), chunk_b = up(size_t(C + 1) * 8);
  // everything is sized before the first copy is issued: nothing may be reallocated in flight
  h->pool->reserve(h->h_out, text_b + chunk_b);
  h->pool->reserve(h->h_ids, std::min(size_t(n_bytes), size_t(double(n_bytes) * h->ids_per_byte) + 1024) * 4);  // grown below
  h->h_marks.reserve(np * 64);
  std::memset(h->h_marks.p, 0, np * 64);
  h->d_bytes.reserve(size_t(n_bytes) + 32);
  h->d_out_ids.reserve(size_t(n_bytes) * 4);
  if (n_texts > 1) h->d_text_off.reserve(size_t(n_texts + 1) * 8);
  h->d_totals.reserve(80 + size_t(groups) * 8);
  h->d_piece_ids.reserve((np + 1) * 8);
  for (cudaStream_t* c : {&h->in_stream, &h->pack_stream, &h->out_stream})
    if (!*c) GTK_CUDA(cudaStreamCreateWithFlags(c, cudaStreamNonBlocking));
  while (h->piece_ev.size() < np * 4) {  // per piece: uploaded; in front of, between and behind its kernels
    cudaEvent_t e;
    GTK_CUDA(cudaEventCreateWithFlags(&e, h->piece_ev.size() % 4 == 0 ? cudaEventDisableTiming : cudaEventDefault));
    h->piece_ev.push_back(e);
  }
  gtk::EncodeBuffers b = plan_batch(h, Kernels::tiles, h->d_bytes.as<uint8_t>(), n_bytes, h->d_text_off.as<int64_t>(), n_texts,
                                    h->d_out_ids.as<int32_t>(), n_bytes, nullptr, true).b;
  int32_t* tickets = b.group_cnt + groups;
  cudaStream_t s   = h->stream;
  int launches     = 0;
  begin_call(h, GTK_MODE_OPT, n_bytes);
  if (n_texts > 1) GTK_CUDA(cudaMemcpyAsync(h->d_text_off.p, text_offsets, size_t(n_texts + 1) * 8, cudaMemcpyHostToDevice, s));
  GTK_CUDA(cudaMemsetAsync(tickets, 0, np * 4, s));
  GTK_CUDA(cudaEventRecord(h->ev[0], s));
  begin_tiles(h, b, &launches);
  GTK_CUDA(cudaEventRecord(h->ev[1], s));
  GTK_CUDA(cudaGetLastError());

  Gather gather(h, src);
  int64_t have = 0;  // ids whose copy has been issued
  // the ids of piece i, once its mark is there; wait: for the mark.  false: not there yet
  auto collect = [&](size_t i, bool wait) {
    volatile const int64_t* m = h->h_marks.as<int64_t>() + 8 * i;
    if (!wait && m[3] != int64_t(i) + 1) return false;
    if (!wait_for_mark(m + 3, int64_t(i) + 1, h->pack_stream, "pack kernel"))
      throw CudaFail{"pack kernel ended without publishing its results"};
    const int64_t n = m[1];
    if (n < have || n > n_bytes) throw CudaFail{"inconsistent id count"};
    if (size_t(n) * 4 > h->h_ids.cap) {  // grow the pinned id buffer, keeping what has arrived
      h->ids_per_byte = std::min(1.0, std::max(h->ids_per_byte, 1.1 * double(n) / double(ends[i])));
      GTK_CUDA(cudaStreamSynchronize(h->out_stream));
      PinBuf bigger;
      h->pool->reserve(bigger, std::max(size_t(n), std::min(size_t(n_bytes), size_t(double(n_bytes) * h->ids_per_byte) + 1024)) * 4);
      std::memcpy(bigger.p, h->h_ids.p, size_t(have) * 4);
      h->pool->give_back(h->h_ids);
      h->h_ids = bigger;
    }
    if (n > have)
      GTK_CUDA(cudaMemcpyAsync(h->h_ids.as<int32_t>() + have, h->d_out_ids.as<int32_t>() + have, size_t(n - have) * 4,
                               cudaMemcpyDeviceToHost, h->out_stream));
    have = n;
    return true;
  };
  size_t done = 0;  // pieces collected
  for (size_t i = 0; i < np; ++i) {
    cudaEvent_t* ev  = &h->piece_ev[4 * i];
    const int64_t lo = i ? ends[i - 1] : 0;
    GTK_CUDA(cudaMemcpyAsync(h->d_bytes.as<uint8_t>() + lo, gather.ready(ends[i]) + lo, size_t(ends[i] - lo), cudaMemcpyHostToDevice, h->in_stream));
    GTK_CUDA(cudaEventRecord(ev[0], h->in_stream));
    GTK_CUDA(cudaStreamWaitEvent(s, ev[0], 0));
    // a tile may need the text to the end of its last chunk: such tiles wait for the next piece
    const bool last   = i + 1 == np;
    const int64_t own = ends[i] - gtk::kWindow - std::min(chunk, n_bytes);
    b.tile_hi         = last ? K : std::max(b.tile_lo, own / gtk::kTile / gtk::kTileGroup * gtk::kTileGroup);
    b.ticket          = tickets + i;
    b.piece_ids       = h->d_piece_ids.as<int64_t>() + i;
    GTK_CUDA(cudaEventRecord(ev[1], s));
    launches += gtk::launch_merge_opt(b, h->call_tab, h->opt_grid, s);
    GTK_CUDA(cudaEventRecord(ev[2], s));
    // a piece without a tile hands the count of the pieces in front of it on
    launches += gtk::launch_pack_tiles(b, h->sm_count, false, nullptr, 0, s);
    GTK_CUDA(cudaEventRecord(ev[3], s));
    GTK_CUDA(cudaStreamWaitEvent(h->pack_stream, ev[3], 0));
    launches += gtk::launch_publish_piece(b, h->h_marks.as<int64_t>() + 8 * i, int64_t(i) + 1, h->pack_stream);  // page-locked: same address on the device
    GTK_CUDA(cudaGetLastError());
    b.tile_lo = b.tile_hi;
    while (done < i && collect(done, false)) ++done;
  }
  while (done < np) collect(done++, true);
  GTK_CUDA(cudaMemcpyAsync(h->h_out.p, b.text_id_off, size_t(n_texts + 1) * 8, cudaMemcpyDeviceToHost, h->out_stream));
  GTK_CUDA(cudaMemcpyAsync(h->h_out.as<uint8_t>() + text_b, b.chunk_id_off, size_t(C + 1) * 8, cudaMemcpyDeviceToHost, h->out_stream));
  GTK_CUDA(cudaStreamSynchronize(h->out_stream));
  const int64_t* end = h->h_marks.as<int64_t>() + 8 * (np - 1);
  if (end[2] != gtk::kStatusOk) return h->fail(GTK_ERR_KERNEL, status_text(int(end[2])));
  if (end[0] != C) return h->fail(GTK_ERR_KERNEL, "inconsistent totals");
  GTK_CUDA(cudaEventSynchronize(h->piece_ev[4 * np - 1]));
  GTK_CUDA(cudaEventElapsedTime(&h->stage_ms[0], h->ev[0], h->ev[1]));
  for (size_t i = 0; i < np; ++i) {
    float merge = 0, pack = 0;
    GTK_CUDA(cudaEventElapsedTime(&merge, h->piece_ev[4 * i + 1], h->piece_ev[4 * i + 2]));
    GTK_CUDA(cudaEventElapsedTime(&pack, h->piece_ev[4 * i + 2], h->piece_ev[4 * i + 3]));
    h->stage_ms[1] += merge;
    h->stage_ms[3] += pack;
  }
  h->stage_ms[4]      = h->stage_ms[0] + h->stage_ms[1] + h->stage_ms[3];
  h->result_is_packed = true;
  h->ids_apart        = true;
  h->pack_base        = h->h_out.as<uint8_t>();
  h->result_bufs[0]   = &h->h_out;
  h->result_bufs[1]   = &h->h_ids;
  h->pack_text_bytes  = text_b;
  h->pack_chunk_bytes = chunk_b;
  h->last_launches    = launches;
  h->res_n_ids        = have;
  h->res_n_chunks     = C;
  if (kernel_ms) *kernel_ms = h->stage_ms[4];
  return GTK_OK;
}

// frees every device / pinned buffer, stream and event of a handle (also used when gtk_create fails half way)
void release_handle(gtk_tokenizer* h)
{
  if (h->device >= 0) {
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (DevBuf* b : {&h->d_bpi, &h->d_slots, &h->d_overflow, &h->d_bpr, &h->d_mor, &h->d_sor, &h->d_adj, &h->d_b2i, &h->d_short_words, &h->d_long_words, &h->d_learned_words, &h->d_low_map, &h->d_wide_slots, &h->d_staging32, &h->d_seg_scratch32, &h->d_bytes, &h->d_text_off,
                      &h->d_text_chunk_base, &h->d_chunk_off, &h->d_tile_chunk0, &h->d_staging, &h->d_unit_first,
                      &h->d_unit_cnt, &h->d_chunk_cnt, &h->d_tile_info, &h->d_chunk_rel, &h->d_text_rel, &h->d_group_base, &h->d_chunk_id_off, &h->d_text_id_off,
                      &h->d_out_ids, &h->d_seg_scratch, &h->d_scan_sums, &h->d_totals, &h->d_out_pack, &h->d_fast_in})
      b->release();
    for (PinBuf* b : {&h->h_ids, &h->h_text_id_off, &h->h_chunk_id_off, &h->h_totals, &h->h_piece_off, &h->h_piece_id_off, &h->h_chunk_id_all, &h->h_out_pack, &h->h_mid, &h->h_out, &h->h_gather, &h->h_marks, &h->h_fast_in}) b->release();
    for (DevBuf* b : {&h->d_piece_off, &h->d_piece_id_off, &h->d_chunk_id_all, &h->d_piece_ids}) b->release();
    if (h->small_in_h) cudaFreeHost(h->small_in_h);
    if (h->small_out_h) cudaFreeHost(h->small_out_h);
    {
      std::lock_guard<std::mutex> lock(h->pool->mu);
      h->pool->closed = true;
      for (PinBuf& b : h->pool->spare) b.release();
      h->pool->spare.clear();
    }
    for (auto& sl : h->slice) sl.release();
    if (h->in_stream) cudaStreamDestroy(h->in_stream);
    if (h->out_stream) cudaStreamDestroy(h->out_stream);
    if (h->pack_stream) cudaStreamDestroy(h->pack_stream);
    for (cudaEvent_t ev : h->piece_ev) cudaEventDestroy(ev);
    for (auto& ev : h->ev)
      if (ev) cudaEventDestroy(ev);
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
  }
}

int validate_offsets(gtk_tokenizer* h, const int64_t* text_offsets, int64_t n_texts)
{
  if (n_texts < 0) return h->fail(GTK_ERR_INVALID_ARG, "n_texts must be >= 0");
  if (n_texts > 0 && !text_offsets) return h->fail(GTK_ERR_INVALID_ARG, "text_offsets is null");
  if (n_texts > 0 && text_offsets[0] != 0) return h->fail(GTK_ERR_INVALID_ARG, "text_offsets[0] must be 0");
  for (int64_t t = 0; t < n_texts; ++t)
    if (text_offsets[t + 1] < text_offsets[t]) return h->fail(GTK_ERR_INVALID_ARG, "text_offsets must be non-decreasing");
  return GTK_OK;
}

}  // namespace

namespace gtk {
cudaError_t wait_for_word(volatile const int32_t* word, int32_t seq, cudaStream_t stream)
{
  for (unsigned spin = 1; *word != seq; ++spin) {
    if ((spin & 0xFFFFu) == 0u) {
      const cudaError_t q = cudaStreamQuery(stream);
      if (q == cudaSuccess && *word != seq) return cudaErrorUnknown;
      if (q != cudaSuccess && q != cudaErrorNotReady) return q;
    }
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#endif
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return cudaSuccess;
}

bool handle_view(gtk_tokenizer* h, HandleView* out)
{
  if (!h || !out) return false;
  out->device = h->device;
  out->sm_count = h->sm_count;
  out->stream = h->stream;
  out->table = h->dtab;
  out->wide = h->wide;
  out->low_id_map = (h->device >= 0 && h->id_space == GTK_IDS_GPT2) ? h->d_low_map.as<uint16_t>() : nullptr;
  out->pinned_words = h->device >= 0 ? h->h_totals.as<int32_t>() + 8 : nullptr;
  out->mu = &h->mu;
  out->last_error = &h->last_error;
  return true;
}
}  // namespace gtk

// ------------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------------

extern "C" {

GTK_API const char* gtk_version(void) { return "gputok_b200 0.1 (sm_100a)"; }

GTK_API const char* gtk_global_error(void) { return g_global_error.c_str(); }

GTK_API int gtk_create(const char* merges_path, int chunk_tokens, int max_iters, int device, gtk_tokenizer** out)
{
  if (!out) {
    g_global_error = "out is null";
    return GTK_ERR_INVALID_ARG;
  }
  *out = nullptr;
  if (!merges_path) {
    g_global_error = "merges_path is null";
    return GTK_ERR_INVALID_ARG;
  }
  if (chunk_tokens <= 0) {
    g_global_error = "chunk_tokens must be > 0";
    return GTK_ERR_INVALID_ARG;
  }
  if (max_iters <= 0) max_iters = 50;
  gtk_tokenizer* h = nullptr;
  try {
    h = new gtk_tokenizer();
    h->chunk_tokens = chunk_tokens;
    h->max_iters = max_iters;
    h->device = device;
    try {
      h->table.reset(new gtk::HostTable(merges_path));
    } catch (const std::runtime_error& e) {
      g_global_error = e.what();
      delete h;
      return GTK_ERR_IO;
    }
    if (device >= 0) {
      h->wide = !h->table->fits_u16;  // ids >= 65535 or ranks >= 65534: served by the 32-bit kernel
      int count = 0;
      cudaError_t e = cudaGetDeviceCount(&count);
      if (e != cudaSuccess || device >= count) {
        g_global_error = std::string("CUDA device ") + std::to_string(device) + " not available: " +
                         (e != cudaSuccess ? cudaGetErrorString(e) : "ordinal out of range");
        delete h;
        return GTK_ERR_NO_DEVICE;
      }
      GTK_CUDA(cudaSetDevice(device));
      GTK_CUDA(cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, device));
      GTK_CUDA(cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking));
      h->stream = h->own_stream;
      for (auto& ev : h->ev) GTK_CUDA(cudaEventCreate(&ev));
      upload_table(h);
      h->opt_grid = h->sm_count * std::max(1, gtk::opt_kernel_max_blocks_per_sm());
      h->base_grid = h->sm_count * std::max(1, gtk::base_kernel_max_blocks_per_sm(chunk_tokens, 0));
      h->localmin_grid = h->sm_count * std::max(1, gtk::localmin_kernel_max_blocks_per_sm());
      h->wide_grid = h->sm_count * std::max(1, gtk::wide_kernel_max_blocks_per_sm());
      h->h_totals.reserve(64);
      std::memset(h->h_totals.p, 0, 64);
      small_path_init(h);
    }
    *out = h;
    return GTK_OK;
  } catch (const CudaFail& f) {
    g_global_error = f.what;
    if (h) release_handle(h);
    delete h;
    return GTK_ERR_CUDA;
  } catch (const std::bad_alloc&) {
    g_global_error = "out of host memory";
    if (h) release_handle(h);
    delete h;
    return GTK_ERR_INVALID_ARG;
  }
}

GTK_API void gtk_destroy(gtk_tokenizer* h)
{
  if (!h) return;
  release_handle(h);
  delete h;
}

GTK_API const char* gtk_last_error(const gtk_tokenizer* h) { return h ? h->last_error.c_str() : "null handle"; }

GTK_API int gtk_table_info_get(const gtk_tokenizer* h, gtk_table_info* out)
{
  if (!h || !out) return GTK_ERR_INVALID_ARG;
  const gtk::HostTable& t = *h->table;
  out->vocab_size = int32_t(t.id_to_symbols.size());
  out->num_merges = int32_t(t.rows.size());
  out->max_rank = t.max_rank;
  out->hash_capacity = uint32_t(t.pair_buckets.size() * 4);
  out->hash_overflow_entries = t.pair_overflow_count;
  out->hash_bytes = uint32_t(t.pair_buckets.size() * sizeof(gtk::PairBucket) + t.pair_overflow.size() * sizeof(gtk::PairSlot));
  out->monotone = t.monotone;
  out->merged_is_256_plus_rank = t.merged_is_256_plus_rank;
  out->byte_ids_identity = t.byte_ids_identity;
  out->adj_bigrams = t.adj_count;
  out->chunk_tokens = h->chunk_tokens;
  out->max_iters = h->max_iters;
  out->device = h->device;
  out->sm_count = h->sm_count;
  out->whole_segment_entries = int32_t(t.word_count);
  out->whole_segment_dropped = t.word_dropped;
  return GTK_OK;
}

GTK_API int gtk_encode_device(gtk_tokenizer* h, int mode, const uint8_t* d_bytes, int64_t n_bytes,
                              const int64_t* d_text_offsets, int64_t n_texts, int32_t* d_out_ids,
                              int64_t out_capacity, int64_t* d_out_chunk_offsets, int64_t chunk_capacity,
                              int64_t* n_ids, int64_t* n_chunks, float* kernel_ms)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  if (h->device < 0) return h->fail(GTK_ERR_NO_DEVICE, "host-only handle: no GPU entry points");
  if (mode != GTK_MODE_OPT && mode != GTK_MODE_BASE && mode != GTK_MODE_LOCALMIN) return h->fail(GTK_ERR_INVALID_ARG, "unknown mode");
  if (n_bytes < 0 || n_texts < 0) return h->fail(GTK_ERR_INVALID_ARG, "negative size");
  if (n_ids) *n_ids = 0;
  if (n_chunks) *n_chunks = 0;
  if (kernel_ms) *kernel_ms = 0.f;
  h->last_launches = 0;
  std::fill(h->stage_ms, h->stage_ms + 5, 0.f);
  h->front_ms = -1.f;
  if (n_texts == 0 || n_bytes == 0) return GTK_OK;
  if (!d_bytes || !d_text_offsets || !d_out_ids) return h->fail(GTK_ERR_INVALID_ARG, "null device pointer");
  if (h->wide && mode == GTK_MODE_LOCALMIN) return h->fail(GTK_ERR_TABLE, kWideNoLocalmin);
  try {
    GTK_CUDA(cudaSetDevice(h->device));
    const int64_t need_chunks = chunk_upper_bound(n_bytes, n_texts, h->chunk_tokens);
    int64_t* chunk_dst = d_out_chunk_offsets;
    if (chunk_dst && chunk_capacity < need_chunks + 1) chunk_dst = nullptr;  // scan into the arena, copy what fits
    const bool by_tiles = mode == GTK_MODE_OPT && !h->wide;
    Plan p = plan_batch(h, by_tiles ? Kernels::tiles : Kernels::chunks, d_bytes, n_bytes, d_text_offsets, n_texts, d_out_ids,
                        out_capacity, chunk_dst, false);
    begin_call(h, mode, n_bytes);
    int launches = 0;
    if (by_tiles) {
      p.b.text_end = d_text_offsets + n_texts;
      volatile int64_t* tot = h->h_totals.as<int64_t>();
      const int64_t seq     = ++h->mid_seq;
      tot[3] = 0;  // copy_totals of an earlier call in another mode has left its chunk ticket there, which may equal the call number
      run_tiles(h, p.b, false, h->h_totals.as<int64_t>(), seq, &launches);
      if (!wait_for_mark(tot + 3, seq, h->stream, "pack kernel"))
        return h->fail(GTK_ERR_KERNEL, "pack kernel ended without publishing its results");
      const int64_t C = tot[0], N = tot[1];
      h->stage_ms[4]  = float(double(tot[4]) * 1e-6);  // by the kernels' own clock
      if (tot[2] != gtk::kStatusOk) return h->fail(GTK_ERR_KERNEL, status_text(int(tot[2])));
      if (N > out_capacity) return h->fail(GTK_ERR_CAPACITY, "d_out_ids too small: need " + std::to_string(N) + " ids");
      if (d_out_chunk_offsets && !chunk_dst) {
        if (chunk_capacity < C + 1)
          return h->fail(GTK_ERR_CAPACITY, "d_out_chunk_offsets too small: need " + std::to_string(C + 1));
        GTK_CUDA(cudaMemcpyAsync(d_out_chunk_offsets, p.b.chunk_id_off, size_t(C + 1) * 8, cudaMemcpyDeviceToDevice,
                                 h->stream));
        GTK_CUDA(cudaStreamSynchronize(h->stream));
      }
      if (h->stage_timing) {
        std::fill(h->stage_ms, h->stage_ms + 5, 0.f);
        GTK_CUDA(cudaEventSynchronize(h->ev[4]));
        collect_stage_times(h);
      }
      h->last_launches = launches;
      if (n_ids) *n_ids = N;
      if (n_chunks) *n_chunks = C;
      if (kernel_ms) *kernel_ms = h->stage_ms[4];
      return GTK_OK;
    }
    // When the chunk offsets are scanned straight into the caller's buffer (or not wanted), the pack follows
    // the front without a host round trip: the pack kernel itself never writes past out_capacity, and the
    // totals are checked once at the end.
    const bool one_sync = !d_out_chunk_offsets || chunk_dst;
    run_front(h, p.b, mode, &launches, nullptr, nullptr, nullptr, one_sync);
    if (one_sync) run_pack(h, p.b, &launches, nullptr, nullptr, true);
    GTK_CUDA(cudaStreamSynchronize(h->stream));
    const int64_t* ht = h->h_totals.as<int64_t>();
    const int64_t C = ht[0], N = ht[1];
    const int status = reinterpret_cast<const int32_t*>(ht + 2)[1];
    if (status != gtk::kStatusOk) return h->fail(GTK_ERR_KERNEL, status_text(status));
    if (N > out_capacity) return h->fail(GTK_ERR_CAPACITY, "d_out_ids too small: need " + std::to_string(N) + " ids");
    if (one_sync) {
      collect_stage_times(h, true);
      h->last_launches = launches;
      if (n_ids) *n_ids = N;
      if (n_chunks) *n_chunks = C;
      if (kernel_ms) *kernel_ms = h->stage_ms[4];
      return GTK_OK;
    }
    if (d_out_chunk_offsets && !chunk_dst) {
      if (chunk_capacity < C + 1)
        return h->fail(GTK_ERR_CAPACITY, "d_out_chunk_offsets too small: need " + std::to_string(C + 1));
      GTK_CUDA(cudaMemcpyAsync(d_out_chunk_offsets, p.b.chunk_id_off, size_t(C + 1) * 8, cudaMemcpyDeviceToDevice,
                               h->stream));
    }
    run_pack(h, p.b, &launches);
    GTK_CUDA(cudaStreamSynchronize(h->stream));
    collect_stage_times(h);
    h->last_launches = launches;
    if (n_ids) *n_ids = N;
    if (n_chunks) *n_chunks = C;
    if (kernel_ms) *kernel_ms = h->stage_ms[4];
    return GTK_OK;
  } catch (const CudaFail& f) {
    settle(h);
    return h->fail(GTK_ERR_CUDA, f.what);
  } catch (const std::bad_alloc&) {
    settle(h);
    return out_of_memory(h);
  }
}

static int encode_host(gtk_tokenizer* h, int mode, const uint8_t* bytes, const uint8_t* const* parts,
                       const int64_t* text_offsets, int64_t n_texts, float* kernel_ms)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  if (h->device < 0) return h->fail(GTK_ERR_NO_DEVICE, "host-only handle: no GPU entry points");
  if (mode != GTK_MODE_OPT && mode != GTK_MODE_BASE && mode != GTK_MODE_LOCALMIN) return h->fail(GTK_ERR_INVALID_ARG, "unknown mode");
  if (int rc = validate_offsets(h, text_offsets, n_texts)) return rc;
  if (kernel_ms) *kernel_ms = 0.f;
  h->result_is_cpu = false;
  h->result_is_small = false;
  h->result_is_packed = false;
  h->ids_apart = false;
  h->result_is_taken = false;
  h->result_bufs[0] = h->result_bufs[1] = h->result_bufs[2] = nullptr;
  h->res_n_ids = h->res_n_chunks = 0;
  h->res_n_texts = n_texts;
  h->last_launches = 0;
  std::fill(h->stage_ms, h->stage_ms + 5, 0.f);
  h->front_ms = -1.f;
  try {
    GTK_CUDA(cudaSetDevice(h->device));
    const int64_t n_bytes = n_texts ? text_offsets[n_texts] : 0;
    if (n_bytes == 0) {  // empty batch or only empty texts: ([], 0.0) in the reference
      h->pool->reserve(h->h_text_id_off, size_t(n_texts + 1) * 8);
      std::memset(h->h_text_id_off.p, 0, size_t(n_texts + 1) * 8);
      h->pool->reserve(h->h_chunk_id_off, 8);
      h->h_chunk_id_off.as<int64_t>()[0] = 0;
      return GTK_OK;
    }
    if (!bytes && !parts) return h->fail(GTK_ERR_INVALID_ARG, "bytes is null");
    const bool staged = !bytes || (n_bytes >= kStageMinBytes && n_bytes <= kStageMaxBytes && is_ordinary_memory(bytes));
    const Source src{bytes, parts, text_offsets, n_texts, staged};
    if (h->wide && mode == GTK_MODE_LOCALMIN) return h->fail(GTK_ERR_TABLE, kWideNoLocalmin);
    if (!h->wide && mode == GTK_MODE_OPT && n_bytes <= gtk::kSmallMaxBytes && n_texts <= gtk::kSmallMaxTexts)
      return encode_host_small(h, src, text_offsets, n_texts, n_bytes, kernel_ms);
    if (!h->wide && mode == GTK_MODE_OPT)
      return n_bytes >= kPiecesMinBytes ? encode_host_pieces(h, src, text_offsets, n_texts, n_bytes, kernel_ms)
                                        : encode_host_tiles(h, src, text_offsets, n_texts, n_bytes, kernel_ms);
    Gather gather(h, src);
    bytes = gather.ready(n_bytes);  // the kernels that work chunk by chunk take one buffer
    if (n_bytes >= kSliceThresholdBytes) return encode_host_sliced(h, mode, bytes, text_offsets, n_texts, n_bytes, kernel_ms);
    cudaStream_t s = h->stream;
    h->d_bytes.reserve(size_t(n_bytes) + 32);
    h->d_text_off.reserve(size_t(n_texts + 1) * 8);
    GTK_CUDA(cudaMemcpyAsync(h->d_bytes.p, bytes, size_t(n_bytes), cudaMemcpyHostToDevice, s));
    GTK_CUDA(cudaMemcpyAsync(h->d_text_off.p, text_offsets, size_t(n_texts + 1) * 8, cudaMemcpyHostToDevice, s));
    // Everything that goes back lives in one arena, [text id offsets | chunk id offsets | ids], each sized by its
    // bound (a batch of this path is below 8 MiB, so 4 bytes per input byte for the ids is little): the pack
    // follows the front without a host round trip and one copy brings the results.
    const size_t text_b  = ((size_t(n_texts) + 1) * 8 + 63) & ~size_t(63);
    const size_t chunk_b = ((size_t(chunk_upper_bound(n_bytes, n_texts, h->chunk_tokens)) + 1) * 8 + 63) & ~size_t(63);
    h->d_out_pack.reserve(text_b + chunk_b + size_t(n_bytes) * 4 + 64);
    uint8_t* dp = h->d_out_pack.as<uint8_t>();
    Plan p = plan_batch(h, Kernels::chunks, h->d_bytes.as<uint8_t>(), n_bytes, h->d_text_off.as<int64_t>(), n_texts,
                        reinterpret_cast<int32_t*>(dp + text_b + chunk_b), n_bytes,
                        reinterpret_cast<int64_t*>(dp + text_b), true);
    p.b.text_id_off = reinterpret_cast<int64_t*>(dp);
    int launches = 0;
    // Up to 1 MiB of text a kernel behind the pack writes the results into mapped host memory and the host polls
    // its completion mark: no copy of the totals, no second copy sized by them, no stream synchronisation.
    const bool by_kernel = n_bytes <= kResultsByKernelMaxBytes &&
                           64 + text_b + chunk_b + size_t(n_bytes) * 4 + 64 <= kMappedResultBytes;
    run_front(h, p.b, mode, &launches, nullptr, nullptr, nullptr, true);
    run_pack(h, p.b, &launches, nullptr, nullptr, true, !by_kernel);
    int64_t C = 0, N = 0;
    int status = gtk::kStatusOk;
    if (by_kernel) {
      const int64_t seq = ++h->mid_seq;
      uint8_t* md = mid_block(h);
      launches += gtk::launch_results_to_host(p.b, dp, md + 64, int64_t(text_b + chunk_b), reinterpret_cast<int64_t*>(md), seq, s);
      GTK_CUDA(cudaGetLastError());
      volatile const int64_t* tot = h->h_mid.as<volatile const int64_t>();
      if (!wait_for_mark(tot + 3, seq, s, "result kernel"))
        return h->fail(GTK_ERR_KERNEL, "result kernel ended without publishing its results");
      C = tot[0], N = tot[1], status = int(tot[2]);
    } else {
      GTK_CUDA(cudaStreamSynchronize(s));
      const int64_t* ht = h->h_totals.as<int64_t>();
      C = ht[0], N = ht[1];
      status = reinterpret_cast<const int32_t*>(ht + 2)[1];
    }
    if (status != gtk::kStatusOk) return h->fail(GTK_ERR_KERNEL, status_text(status));
    if (N > n_bytes) return h->fail(GTK_ERR_KERNEL, "more ids than input bytes");
    if (!by_kernel) {
      h->pool->reserve(h->h_out_pack, text_b + chunk_b + size_t(N) * 4 + 64);
      GTK_CUDA(cudaMemcpyAsync(h->h_out_pack.p, dp, text_b + chunk_b + size_t(N) * 4, cudaMemcpyDeviceToHost, s));
      GTK_CUDA(cudaStreamSynchronize(s));
    }
    collect_stage_times(h, true);
    // only now is there a result that can be looked at and taken over
    h->pack_base        = by_kernel ? h->h_mid.as<uint8_t>() + 64 : h->h_out_pack.as<uint8_t>();
    h->result_bufs[0]   = by_kernel ? &h->h_mid : &h->h_out_pack;
    h->result_is_packed = true;
    h->pack_text_bytes  = text_b;
    h->pack_chunk_bytes = chunk_b;
    h->last_launches = launches;
    h->res_n_ids = N;
    h->res_n_chunks = C;
    if (kernel_ms) *kernel_ms = h->stage_ms[4];
    return GTK_OK;
  } catch (const CudaFail& f) {
    settle(h);
    return h->fail(GTK_ERR_CUDA, f.what);
  } catch (const std::bad_alloc&) {
    settle(h);
    return out_of_memory(h);
  }
}

GTK_API int gtk_encode(gtk_tokenizer* h, int mode, const uint8_t* bytes, const int64_t* text_offsets, int64_t n_texts,
                       float* kernel_ms)
{
  return encode_host(h, mode, bytes, nullptr, text_offsets, n_texts, kernel_ms);
}

GTK_API int gtk_encode_strings(gtk_tokenizer* h, int mode, const uint8_t* const* texts, const int64_t* text_offsets,
                               int64_t n_texts, float* kernel_ms)
{
  return encode_host(h, mode, nullptr, texts, text_offsets, n_texts, kernel_ms);
}

GTK_API int gtk_encode_cpu(gtk_tokenizer* h, int rule, const uint8_t* bytes, const int64_t* text_offsets,
                           int64_t n_texts)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  if (rule != GTK_RULE_GREEDY && rule != GTK_RULE_LOCALMIN) return h->fail(GTK_ERR_INVALID_ARG, "unknown rule");
  if (int rc = validate_offsets(h, text_offsets, n_texts)) return rc;
  if (n_texts > 0 && text_offsets[n_texts] > 0 && !bytes) return h->fail(GTK_ERR_INVALID_ARG, "bytes is null");
  h->cpu_ids.clear();
  h->cpu_text_off.assign(1, 0);
  h->cpu_chunk_off.assign(1, 0);
  for (int64_t t = 0; t < n_texts; ++t) {
    const int64_t s = text_offsets[t], e = text_offsets[t + 1];
    if (rule == GTK_RULE_LOCALMIN) {
      if (e > s) {
        h->table->localmin_text(bytes + s, e - s, h->max_iters, h->cpu_ids);
        h->cpu_chunk_off.push_back(int64_t(h->cpu_ids.size()));
      }
    } else {
      for (int64_t pos = s; pos < e; pos += h->chunk_tokens) {
        const int64_t len = std::min<int64_t>(h->chunk_tokens, e - pos);
        h->table->greedy_chunk(bytes + pos, len, h->cpu_ids);
        h->cpu_chunk_off.push_back(int64_t(h->cpu_ids.size()));
      }
    }
    h->cpu_text_off.push_back(int64_t(h->cpu_ids.size()));
  }
  h->result_is_cpu = true;
  h->result_is_small = false;
  h->result_is_packed = false;
  h->ids_apart = false;
  h->result_is_taken = false;
  h->result_bufs[0] = h->result_bufs[1] = h->result_bufs[2] = nullptr;
  h->res_n_ids = int64_t(h->cpu_ids.size());
  h->res_n_chunks = int64_t(h->cpu_chunk_off.size()) - 1;
  h->res_n_texts = n_texts;
  return GTK_OK;
}

GTK_API int gtk_result_sizes(const gtk_tokenizer* h, int64_t* n_ids, int64_t* n_chunks, int64_t* n_texts)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  if (n_ids) *n_ids = h->res_n_ids;
  if (n_chunks) *n_chunks = h->res_n_chunks;
  if (n_texts) *n_texts = h->res_n_texts;
  return GTK_OK;
}

GTK_API int gtk_result_view(const gtk_tokenizer* h, const int32_t** ids, const int64_t** text_id_offsets,
                            const int64_t** chunk_id_offsets)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  if (h->result_is_taken) {
    if (ids) *ids = h->view_ids;
    if (text_id_offsets) *text_id_offsets = h->view_text;
    if (chunk_id_offsets) *chunk_id_offsets = h->view_chunk;
  } else if (h->result_is_cpu) {
    if (ids) *ids = h->cpu_ids.data();
    if (text_id_offsets) *text_id_offsets = h->cpu_text_off.data();
    if (chunk_id_offsets) *chunk_id_offsets = h->cpu_chunk_off.data();
  } else if (h->result_is_small) {
    if (ids) *ids = reinterpret_cast<const int32_t*>(h->small_out_h + kSmallOutIds);
    if (text_id_offsets) *text_id_offsets = reinterpret_cast<const int64_t*>(h->small_out_h + kSmallOutText);
    if (chunk_id_offsets) *chunk_id_offsets = reinterpret_cast<const int64_t*>(h->small_out_h + kSmallOutChunk);
  } else if (h->result_is_packed) {
    const uint8_t* base = h->pack_base;
    if (ids) *ids = h->ids_apart ? h->h_ids.as<int32_t>() : reinterpret_cast<const int32_t*>(base + h->pack_text_bytes + h->pack_chunk_bytes);
    if (text_id_offsets) *text_id_offsets = reinterpret_cast<const int64_t*>(base);
    if (chunk_id_offsets) *chunk_id_offsets = reinterpret_cast<const int64_t*>(base + h->pack_text_bytes);
  } else {
    if (ids) *ids = h->h_ids.as<int32_t>();
    if (text_id_offsets) *text_id_offsets = h->h_text_id_off.as<int64_t>();
    if (chunk_id_offsets) *chunk_id_offsets = h->h_chunk_id_off.as<int64_t>();
  }
  return GTK_OK;
}

GTK_API int gtk_result_copy(const gtk_tokenizer* h, int32_t* ids, int64_t ids_capacity, int64_t* text_id_offsets,
                            int64_t* chunk_id_offsets, int64_t chunk_capacity)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  const int32_t* src_ids;
  const int64_t *src_text, *src_chunk;
  gtk_result_view(h, &src_ids, &src_text, &src_chunk);
  if (ids) {
    if (ids_capacity < h->res_n_ids) return h->fail(GTK_ERR_CAPACITY, "ids buffer too small");
    if (h->res_n_ids) std::memcpy(ids, src_ids, size_t(h->res_n_ids) * 4);
  }
  if (text_id_offsets && src_text) std::memcpy(text_id_offsets, src_text, size_t(h->res_n_texts + 1) * 8);
  if (chunk_id_offsets) {
    if (chunk_capacity < h->res_n_chunks + 1) return h->fail(GTK_ERR_CAPACITY, "chunk offset buffer too small");
    if (src_chunk) std::memcpy(chunk_id_offsets, src_chunk, size_t(h->res_n_chunks + 1) * 8);
  }
  return GTK_OK;
}

GTK_API gtk_taken* gtk_result_take(gtk_tokenizer* h)
{
  if (!h) return nullptr;
  std::lock_guard<std::mutex> lock(h->mu);
  if (!h->result_bufs[0]) return nullptr;
  size_t bytes = 0;
  for (PinBuf* b : h->result_bufs)
    if (b) bytes += b->cap;
  std::unique_ptr<gtk_taken> t(new (std::nothrow) gtk_taken());  // in front of the count, which a failure would leave raised
  if (!t) return nullptr;
  {
    std::lock_guard<std::mutex> plock(h->pool->mu);
    if (h->pool->taken >= ResultPool::kMaxTaken || h->pool->taken_bytes + bytes > ResultPool::kMaxTakenBytes) return nullptr;
    ++h->pool->taken;
    h->pool->taken_bytes += bytes;
  }
  t->pool  = h->pool;
  t->bytes = bytes;
  // the pointers of gtk_result_view stay what they are
  const int32_t* ids;
  const int64_t *text_off, *chunk_off;
  gtk_result_view(h, &ids, &text_off, &chunk_off);
  h->view_ids = ids, h->view_text = text_off, h->view_chunk = chunk_off;
  for (int i = 0; i < 3; ++i) {
    if (h->result_bufs[i]) std::swap(t->bufs[i], *h->result_bufs[i]);
    h->result_bufs[i] = nullptr;
  }
  h->result_is_taken = true;
  return t.release();
}

GTK_API void gtk_result_release(gtk_taken* t)
{
  if (!t) return;
  {
    std::lock_guard<std::mutex> lock(t->pool->mu);
    --t->pool->taken;
    t->pool->taken_bytes -= t->bytes;
  }
  for (PinBuf& b : t->bufs) t->pool->give_back(b);
  delete t;
}

GTK_API int gtk_last_stage_ms(const gtk_tokenizer* h, float stage_ms[5], int32_t* kernel_launches)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  if (stage_ms) std::memcpy(stage_ms, h->stage_ms, sizeof(h->stage_ms));
  if (kernel_launches) *kernel_launches = h->last_launches;
  return GTK_OK;
}

GTK_API int gtk_decode(const gtk_tokenizer* h, const int32_t* ids, int64_t n_ids, uint8_t* out, int64_t out_capacity,
                       int64_t* n_out)
{
  if (!h || (n_ids > 0 && !ids)) return GTK_ERR_INVALID_ARG;
  // Long ones block by block with the crew's help: the lengths first, then every block to its place.  Whatever is not plain
  // (an unknown id, too little room) is left to the one pass that finds out what.
  constexpr int64_t kBlock = 16384;
  int64_t k = -1;
  if (n_ids >= 4 * kBlock) try {
    const int64_t nb = (n_ids + kBlock - 1) / kBlock;
    std::vector<int64_t> at(size_t(nb) + 1, 0);
    gtk::Crew::Job(h->crew, nb, [&](int64_t i) {
      at[size_t(i) + 1] = h->table->decode(ids + i * kBlock, std::min(kBlock, n_ids - i * kBlock), nullptr, 0);
    }).finish();
    bool plain = true;
    for (int64_t i = 0; i < nb; ++i) {
      plain = plain && at[size_t(i) + 1] >= 0;
      at[size_t(i) + 1] += at[size_t(i)];
    }
    plain = plain && (!out || at[size_t(nb)] <= out_capacity);
    if (plain && out)
      gtk::Crew::Job(h->crew, nb, [&](int64_t i) {
        h->table->decode(ids + i * kBlock, std::min(kBlock, n_ids - i * kBlock), out + at[size_t(i)], at[size_t(i) + 1] - at[size_t(i)]);
      }).finish();
    if (plain) k = at[size_t(nb)];
  } catch (const std::bad_alloc&) {  // the one pass needs no memory
  }
  if (k < 0) k = h->table->decode(ids, n_ids, out, out_capacity);
  if (k == -1 - n_ids) return h->fail(GTK_ERR_CAPACITY, "decode buffer too small");
  if (k < 0) return h->fail(GTK_ERR_INVALID_ARG, "id " + std::to_string(ids[-1 - k]) + " has no byte string");
  if (n_out) *n_out = k;
  return GTK_OK;
}

GTK_API int32_t gtk_token_symbols(const gtk_tokenizer* h, int32_t id, char* buf, int32_t capacity)
{
  if (!h || id < 0 || size_t(id) >= h->table->id_to_symbols.size()) return -1;
  const std::string& s = h->table->id_to_symbols[size_t(id)];
  if (buf && capacity >= int32_t(s.size())) std::memcpy(buf, s.data(), s.size());
  return int32_t(s.size());
}

GTK_API int gtk_set_stream(gtk_tokenizer* h, void* cuda_stream)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  if (h->device < 0) return h->fail(GTK_ERR_NO_DEVICE, "host-only handle: no GPU entry points");
  cudaSetDevice(h->device);
  cudaStreamSynchronize(h->stream);
  h->stream = cuda_stream ? static_cast<cudaStream_t>(cuda_stream) : h->own_stream;
  return GTK_OK;
}

GTK_API int gtk_set_stage_timing(gtk_tokenizer* h, int per_stage)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  h->stage_timing = per_stage != 0;
  return GTK_OK;
}

GTK_API int gtk_set_base_block_size(gtk_tokenizer* h, int threads)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  if (h->device < 0) return h->fail(GTK_ERR_NO_DEVICE, "host-only handle: no GPU entry points");
  if (threads != 0 && threads != 64 && threads != 128 && threads != 256 && threads != 512 && threads != 1024)
    return h->fail(GTK_ERR_INVALID_ARG, "block size must be 0 (automatic), 64, 128, 256, 512 or 1024");
  try {
    GTK_CUDA(cudaSetDevice(h->device));
    h->base_block = threads;
    h->base_grid  = h->sm_count * std::max(1, gtk::base_kernel_max_blocks_per_sm(h->chunk_tokens, threads));
    GTK_CUDA(cudaGetLastError());
  } catch (const CudaFail& f) {
    return h->fail(GTK_ERR_CUDA, f.what);
  }
  return GTK_OK;
}

GTK_API int gtk_set_id_space(gtk_tokenizer* h, int id_space)
{
  if (!h) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(h->mu);
  if (id_space != GTK_IDS_REFERENCE && id_space != GTK_IDS_GPT2) return h->fail(GTK_ERR_INVALID_ARG, "unknown id space");
  h->id_space = id_space;
  return GTK_OK;
}

GTK_API int gtk_write_token_strings(const gtk_tokenizer* h, const char* path, const int32_t* ids,
                                    const int64_t* chunk_id_offsets, int64_t n_chunks)
{
  if (!h || !path || n_chunks < 0 || (n_chunks > 0 && (!ids || !chunk_id_offsets))) return GTK_ERR_INVALID_ARG;
  FILE* f = std::fopen(path, "wb");
  if (!f) return h->fail(GTK_ERR_IO, std::string("Failed to open output file for writing: ") + path);
  const auto& sym = h->table->id_to_symbols;
  std::string line;
  for (int64_t c = 0; c < n_chunks; ++c) {
    line.clear();
    for (int64_t i = chunk_id_offsets[c]; i < chunk_id_offsets[c + 1]; ++i) {
      const int32_t id = ids[i];
      if (id < 0 || size_t(id) >= sym.size()) line += std::to_string(id);  // raw id, as the reference's fallback
      else line += sym[size_t(id)];
      if (i + 1 < chunk_id_offsets[c + 1]) line += ' ';
    }
    line += '\n';
    std::fwrite(line.data(), 1, line.size(), f);
  }
  std::fclose(f);
  return GTK_OK;
}

GTK_API void* gtk_pinned_alloc(size_t bytes)
{
  void* p = nullptr;
  if (cudaHostAlloc(&p, bytes ? bytes : 1, cudaHostAllocDefault) != cudaSuccess) return nullptr;
  return p;
}

GTK_API void gtk_pinned_free(void* p)
{
  if (p) cudaFreeHost(p);
}

}  // extern "C"
