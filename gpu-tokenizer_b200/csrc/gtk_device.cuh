// gtk_device.cuh -- device-side view of the merge table and the launchers the
// host API calls.  Kernels live in gtk_kernels.cu.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>
#include <string>

struct gtk_tokenizer;

namespace gtk {

// Tile geometry of the segment-parallel kernel: a CTA owns the segments that
// start inside TILE consecutive bytes and sees HALO more bytes so that the
// last owned segment can finish inside shared memory.
#ifndef GTK_OPT_THREADS
#define GTK_OPT_THREADS 256
#endif
constexpr int kOptThreads = GTK_OPT_THREADS;
constexpr int kTile = kOptThreads * 16;  // sixteen positions per thread
constexpr int kHalo = 256;
constexpr int kWindow = kTile + kHalo;
constexpr int kBaseThreads = 512;
constexpr int kBaseSmemTokens = 8192;  // chunks up to this length stay in shared memory in the local-minimum and allocation-free kernels
// Longest segment a single thread merges on its own; longer ones are a warp's.  A list entry has four bits for the length and the
// merge scratch room for 16 ranks per lane.  Text with many segments of 17..32 bytes (JSON records 3.0 a tile, Python source 0.7, novel
// 0.05), 256 KiB / 8 / 64 MiB a call: 62 / 138 / 719, 79 / 139 / 472 and 59 / 112 / 322 us; 73 / 159 / 724, 95 / 168 / 700 and 74 / 142 / 589 us with the
// tiles before, where a thread took up to 32 bytes.
constexpr int kThreadSegMax = 16;

// Pointers into HBM, passed by value to every kernel.
struct DeviceTable {
  const uint4* pair_buckets;       // PairBucket[65536]: four words low16(key * kPairMul) << 16 | rank, empty = all ones
  const uint2* pair_overflow;      // {key, rank} open addressing, or nullptr when no bucket overflowed
  uint32_t pair_overflow_mask;     // capacity - 1
  const uint16_t* byte_pair_rank;  // [65536]
  const uint16_t* byte_pair_info;  // [65536]: 0xFFFF cut, 0xFFFE mergeable boundary without a byte-pair rank, else rank
  const uint32_t* merged_of_rank;  // [max_rank+1]
  const uint8_t* same_of_rank;     // [max_rank+1]
  const uint32_t* adj;             // [2048]: word [v / 32][u], bit v % 32: bytes u, v stand next to each other inside a merge result
  const uint16_t* byte_to_id;      // [256]
  const uint2* short_words;        // ShortWord[1 << kShortBits]
  uint4* long_words;               // LongWord[1 << kLongBits], two uint4 each
  int learn;                       // 1: long_words is this call's own copy, merged segments may be added to it
  const uint4* wide_slots;         // tables beyond 16 bits: HashSlot[1 << wide_log2] {right, left, rank, merged id}
  uint32_t wide_log2;
  uint32_t wide_max_probe;         // longest displacement of a stored key
  int monotone;
  int merged_is_256_plus_rank;
  int byte_ids_identity;
};

// Status word written by kernels instead of trapping: 0 = fine.
enum : int {
  kStatusOk = 0,
  kStatusLongQueueOverflow = 1,
  kStatusScratchTooSmall = 2,
  kStatusBadSegment = 3,
  kStatusBadOffsets = 4,  // caller-provided chunk offsets point outside the text or decrease
};

// Chunks and texts around a tile of the tile kernel.
struct TileInfo {
  int64_t c0, t0;  // chunks and texts that start in front of it
  int32_t p0;      // position of the first chunk boundary of the text that runs into the tile, or kTileNoCut
  int32_t flags;
};
constexpr int32_t kTileNoCut  = 0x40000000;
constexpr int32_t kTilePlain  = 1;  // no text starts in the window (or there is only one): its cuts are p0 + i * chunk
constexpr int32_t kTileRunsIn = 2;  // the last of the texts in front of the tile reaches into it

struct EncodeBuffers {
  const uint8_t* bytes;      // input text, n_bytes
  int64_t n_bytes;
  const int64_t* text_off;   // [n_texts+1]
  int64_t* text_off_copy;    // small-batch kernel only: device copy of text_off when that lives in host memory
  int64_t n_texts;
  const int64_t* text_end;   // tile kernel, device-resident batches: where the last text ends, bytes behind it belong to none; nullptr = n_bytes
  int chunk_bytes;
  // chunker outputs
  int64_t* text_chunk_base;  // [n_texts+1] exclusive scan of chunks per text
  int64_t* chunk_off;        // [chunk_cap+1] start byte of each chunk, chunk_off[C] = n_bytes
  int64_t chunk_cap;         // upper bound on the number of chunks
  int32_t* tile_chunk0;      // [n_tiles] single-CTA kernel only: chunk that contains the first byte of the tile
  int64_t n_tiles;
  int64_t tile_lo, tile_hi;  // the launch works on these (all, or those of a piece that starts with a group)
  int32_t* ticket;           // tile ticket of the launch (zero at the start)
  bool starts_clock;         // the tile kernel is the first of the call: it notes the time, otherwise the launch that resets the counters has
  int64_t* piece_ids;        // nullptr, or [0] ids in front of the piece, [1] the same for the next one (pack kernel)
  // merge outputs
  uint16_t* staging;         // [n_bytes] tokens of a unit, compacted at the unit's first byte
  int64_t* unit_first;       // [n_tiles] byte position where the unit's tokens start in staging (opt mode)
  int32_t* unit_cnt;         // [n_tiles] tokens produced by the unit (opt mode)
  int32_t* chunk_cnt;        // [chunk_cap] tokens per chunk (kernels that work chunk by chunk)
  TileInfo* tile_info;       // [n_tiles] what starts where (tile kernel)
  int32_t* chunk_rel;        // [chunk_cap] ids of its tile in front of a chunk
  int32_t* text_rel;         // [n_texts] the same for the texts
  int32_t* group_cnt;        // [n_tiles / kTileGroup + 1] ids per group of tiles (zero at the start)
  int64_t* group_base;       // [n_tiles / kTileGroup + 2] the same, scanned
  // scan outputs
  int64_t* chunk_id_off;     // [chunk_cap+1] packed id offset of each chunk (caller visible)
  int64_t* text_id_off;      // [n_texts+1] or nullptr
  int64_t* chunk_id_mirror;  // single-CTA and finish kernels: device copy of chunk_id_off when that lives in host memory
  int64_t small_seq;         // small-batch kernel only: call number, written to totals[3] as the last store of the kernel
  int32_t* out_ids;
  const uint16_t* low_id_map;  // nullptr, or 256 entries: output id of every id < 256 (GPT-2 id space)
  int64_t out_capacity;
  // scratch
  uint16_t* seg_scratch;     // per-CTA workspace for segments that do not fit in shared memory
  uint32_t* seg_scratch32;   // the same for the 32-bit kernel (tables beyond 16 bits)
  int32_t* staging32;        // [n_bytes] 32-bit kernel: tokens of a chunk, compacted at the chunk's first byte
  int64_t seg_scratch_tokens;  // tokens per CTA (two arrays of this length per CTA)
  int64_t* scan_block_sums;  // workspace of the multi-block scan
  int32_t* counters;         // [0] tile ticket of whole batches, [1] status word, [2] chunk ticket, [8] CTAs done, [12..13] time the first kernel of the call began
  int64_t* totals;           // device: [0] n_chunks, [1] n_ids
};

// Launchers (all asynchronous on `stream`; return the number of kernels launched).
// resets the call's counters and group counts and, when learned is given, the learned long table to the vocabulary's; for
// medium batches without one also what launch_scan_texts does
int launch_begin_batch(const EncodeBuffers& b, const uint4* long_words, uint4* learned, cudaStream_t stream);
int launch_chunker(const EncodeBuffers& b, cudaStream_t stream);
bool chunker_resets_counters(const EncodeBuffers& b);
int launch_merge_opt(const EncodeBuffers& b, const DeviceTable& t, int grid, cudaStream_t stream);
int launch_merge_base(const EncodeBuffers& b, const DeviceTable& t, int grid, int block_threads, cudaStream_t stream);
int launch_merge_wide(const EncodeBuffers& b, const DeviceTable& t, int grid, cudaStream_t stream);
int launch_pack_wide(const EncodeBuffers& b, int grid, cudaStream_t stream);
int wide_kernel_max_blocks_per_sm();
int launch_merge_localmin(const EncodeBuffers& b, const DeviceTable& t, int grid, int max_iters, cudaStream_t stream);
int launch_output_scans(const EncodeBuffers& b, cudaStream_t stream);
// packs the ids of kernels that work chunk by chunk
int launch_pack_chunks(const EncodeBuffers& b, int grid, cudaStream_t stream);
// group_base from group_cnt for batches that are large enough for it (else nothing: returns 0)
int launch_scan_groups(const EncodeBuffers& b, cudaStream_t stream);
// tile_info from text_off and text_chunk_base
int launch_tile_info(const EncodeBuffers& b, cudaStream_t stream);
// text_chunk_base and totals[0] from text_off, for the tile kernel; nothing for one text, or when launch_begin_batch has
// done it (learned: whether that was given a learned table): returns 0
int launch_scan_texts(const EncodeBuffers& b, bool learned, cudaStream_t stream);
// What follows the tile kernel: ids back to back, offsets of chunks and texts, totals[0] and [1].  publish: where the
// host waits for the call, or nullptr: {n_chunks, n_ids, status, seq, nanoseconds since the first kernel of the call began}, seq last;
// out_ids, chunk_id_off and text_id_off may then be page-locked host memory.  Uses counters[8] (zero at the start).
int launch_pack_tiles(const EncodeBuffers& b, int sm_count, bool groups_scanned, int64_t* publish, int64_t seq, cudaStream_t stream);
// {n_chunks, ids up to the end of the piece, status, seq} to `publish` in page-locked host memory, seq last
int launch_publish_piece(const EncodeBuffers& b, int64_t* publish, int64_t seq, cudaStream_t stream);
// the device result arena of a batch into mapped host memory, then totals {n_chunks, n_ids, status} and,
// last, the call number into mapped[0..3]; uses counters[8] (zero at the start of the call)
int launch_results_to_host(const EncodeBuffers& b, const void* src, void* dst, int64_t prefix_bytes, int64_t* mapped,
                           int64_t seq, cudaStream_t stream);
// totals[0..1] and counters[0..3] to `mapped` (page-locked host memory as the device sees it), laid out as 4 x int64
int launch_publish_totals(const EncodeBuffers& b, int64_t* mapped, cudaStream_t stream);
// Whole pipeline in one single-CTA kernel for small batches; totals[0..2] receive n_chunks, n_ids, status,
// totals[4] the kernel's own duration in nanoseconds and, as the very last store, totals[3] the call number.
int launch_encode_small(const EncodeBuffers& b, const DeviceTable& t, cudaStream_t stream);
#ifndef GTK_SMALL_MAX_BYTES
#define GTK_SMALL_MAX_BYTES 8192
#endif
// 8 KiB as two tiles one after the other in one CTA 48 us, as two launches 47; 4 KiB 31 us
constexpr int64_t kSmallMaxBytes = GTK_SMALL_MAX_BYTES;
constexpr int64_t kSmallMaxTexts = 1024;
constexpr int kTileGroup = 64;  // tiles whose ids are counted together
// What the allocation-free entry point needs from a handle (defined in gtk_api.cu).
struct HandleView {
  int device;
  int sm_count;
  cudaStream_t stream;
  DeviceTable table;
  const uint16_t* low_id_map;  // nullptr, or the 256-entry remap of ids < 256 (GPT-2 id space selected)
  bool wide;                   // table beyond 16 bits (the allocation-free kernel is 16-bit only)
  int32_t* pinned_words;  // 8 ints of page-locked host memory owned by the handle
  std::mutex* mu;
  std::string* last_error;
};
bool handle_view(gtk_tokenizer* h, HandleView* out);
// waits for a kernel's last store, the call number, in page-locked memory; an error when the stream fails or goes idle without it
cudaError_t wait_for_word(volatile const int32_t* word, int32_t seq, cudaStream_t stream);

int opt_kernel_max_blocks_per_sm();
int base_kernel_max_blocks_per_sm(int chunk_bytes, int block_threads);
int localmin_kernel_max_blocks_per_sm();
int chunk_kernel_threads(int chunk_bytes, int block_threads);

}  // namespace gtk
