// gtk_tile.cuh -- the segment-parallel tokeniser of one window of text, shared by the tile kernel, the single-CTA
// small-batch kernel and the one-CTA-per-chunk kernels.  Included by gtk_kernels.cu, inside its anonymous namespace.
//
// A CTA of TH threads looks at kWin = 16 * TH + kHalo bytes and tokenises the never-merge segments that start in the
// first 16 * TH of them (sixteen positions per thread):
//   tile_cut      text -> segment-start bitmap, and every position's byte as a token
//   tile_lookup   per warp: multi-byte segments of up to 7 bytes -> table of short strings, one 64-bit load each; the rest
//                 -> table of long strings and of what this call has merged before; one or two misses are merged on the
//                 spot, more go to the CTA's list
//   tile_merge    listed misses, sorted by length, one thread each; segments beyond kThreadSegMax bytes one warp each
//   tile_emit     the start bitmap has become the bitmap of live tokens: every warp hands its own ones over in order
//
// What bounds it: latency and instruction issue together.  A tile is a chain of table loads between barriers, and the
// chip holds only as many tiles as shared memory and registers allow; HBM traffic is 1.7 bytes per input byte, a
// thirtieth of what the memory could carry.  So the layout saves shared memory (what is not used is L1 for the tables),
// barriers (six in a tile without listed misses and long segments: reset, cut, list, lookup, emit, ticket) and instructions: the boundary test is one load from an 8 KiB bit matrix (a
// 128-byte line holds the 32 right bytes of a block for 32 left bytes, so a gather over English text touches three or
// four lines), and ranks are only formed for the segments that no table knows.  Figures: see k_merge_opt.

template <int TH>
struct TileSmem {
  static constexpr int kThreads = TH;
  static constexpr int kWarps   = TH / 32;
  static constexpr int kOwn     = TH * 16;       // positions whose segments belong to the tile
  static constexpr int kWin     = kOwn + kHalo;  // positions it can see
  static constexpr int kWords   = kWin / 32;
  static constexpr int kGroups  = kWin / 16;
  static constexpr int kLong    = kOwn / (kThreadSegMax + 1) + 2;
  static constexpr int kRegion  = 272;           // places per warp in work: 256 segments, or 256 tokens and up to 7 in front
  static constexpr int kMisses  = 512;
  // a segment as it travels through the lists: start << 4 | length - 1 (2..16 bytes), 0 = nothing
  using Entry = std::conditional_t<(TH <= 256), uint16_t, uint32_t>;
  static_assert(kThreadSegMax <= 16 && (TH > 256 || kOwn <= 4096), "entries hold 12 bits of start and 4 of length");

  alignas(16) uint8_t bytes[16 + kWin + 32];  // [16 + i] = window position i
  alignas(16) uint16_t tok[kWin];             // token that starts at a position
  // one region per warp: segments to look up, list of runs or ranks of a long segment, tokens on their way out; all of it
  // (and some more, so that eight batches usually fit at once) is the scratch of the merge loop
  alignas(16) Entry work[kWarps * kRegion + (TH == 256 ? 384 : 0)];
  alignas(16) Entry miss[kMisses];            // segments that no table knows; then gs
  alignas(16) uint4 key_mask[16];             // [length - 1]: byte masks of the four key words
  uint32_t cut[kWords + 4];                   // segment starts, later live tokens; all ones behind the window
  uint16_t longq[kLong];
  int hist[16];
  int nmiss, nlong;
  int first, end;      // owned region: first owned start, end of the last owned segment
  int total;           // live tokens in it
  int over_start;      // start of a segment that runs past the window, or -1
  int no_space;        // a segment needs a workspace and there is none
  int ticket;
  int merged;          // ids of the sequence that the whole CTA has merged
  long long over_end;
  int n_tiles, tail;   // tiles that hold text, bytes of it in the last of them (tile kernel)
  long long run;       // ids written so far (kernels that walk tiles in order)

  static constexpr int kScratchBytes = int(sizeof(work));
  __device__ __forceinline__ uint16_t* region(int warp) { return reinterpret_cast<uint16_t*>(work + warp * kRegion); }
  __device__ __forceinline__ GroupScratch* gs() { return reinterpret_cast<GroupScratch*>(miss); }
  static_assert(sizeof(GroupScratch) <= sizeof(miss), "the group scratch lives in the miss list");
};

// One instance per CTA: static up to 256 threads, in dynamic shared memory beyond (48 KiB is the static limit).
// Named through a function so that out-of-line code compiles to shared-memory instructions too.
extern __shared__ __align__(16) unsigned char g_dyn_smem[];

template <int TH>
__device__ __forceinline__ TileSmem<TH>& tile_smem()
{
  if constexpr (TH <= 256) {
    __shared__ TileSmem<TH> s;
    return s;
  } else {
    return *reinterpret_cast<TileSmem<TH>*>(g_dyn_smem);
  }
}

// A window of text: position i is bytes[lo + i].
struct Span {
  const uint8_t* bytes;
  int64_t lo;
  int own_lo, own_hi;  // owned positions
  int wlen;            // the text ends in front of this position
  bool has_prev;       // the byte in front of position 0 belongs to the same text range
  bool start_here;     // position own_lo starts a segment whatever precedes it
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// the n lowest bits of a word, all of them from n = 32 on
__device__ __forceinline__ uint32_t low_bits(int n)
{
  uint32_t r;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(r) : "r"(n));
  return r;
}

// bits [lo, hi) of the 32-bit word that starts at position w0
__device__ __forceinline__ uint32_t range_mask(int w0, int lo, int hi)
{
  const int a = max(lo - w0, 0), e = min(hi - w0, 32);
  if (e <= a) return 0u;
  return (0xFFFFFFFFu << a) & (0xFFFFFFFFu >> (32 - e));
}

// first segment start strictly after window position s (the words behind the window are all ones)
template <int TH>
__device__ __forceinline__ int next_cut(const TileSmem<TH>& S, int s)
{
  int w = (s + 1) >> 5;
  if (!GTK_IN(w, S.kWords + 2, 1)) return S.kWin;
  uint32_t x = S.cut[w] & (0xFFFFFFFFu << ((s + 1) & 31));
  while (!x) {
    if (!GTK_IN(w + 1, S.kWords + 2, 2)) return S.kWin;
    x = S.cut[++w];
  }
  return w * 32 + __ffs(int(x)) - 1;
}

// The start bitmap turns into the bitmap of live tokens as segments finish: the first token of a segment is always
// live, so a finished segment adds the bits of its other live slots (`a`, relative to its start s; bit 0 is ignored).
// Only bits inside the segment change, so next_cut() of any other segment still finds the same end.
template <int TH>
__device__ __forceinline__ void mark_alive(TileSmem<TH>& S, int s, uint32_t a)
{
  a &= ~1u;
  if (!a) return;
  const int sh = s & 31;
  if (!GTK_IN((s >> 5) + 1, S.kWords + 2, 6)) return;
  atomicOr(&S.cut[s >> 5], a << sh);
  if (sh && (a >> (32 - sh))) atomicOr(&S.cut[(s >> 5) + 1], a >> (32 - sh));
}

// one warp: positions [lo, hi) become live
template <int TH>
__device__ __forceinline__ void mark_alive_range(TileSmem<TH>& S, int lo, int hi, int lane)
{
  if (hi <= lo || !GTK_IN(hi - 1, S.kWin, 7) || !GTK_IN(lo, S.kWin, 7)) return;
  for (int w = (lo >> 5) + lane; w <= ((hi - 1) >> 5); w += 32) atomicOr(&S.cut[w], range_mask(w * 32, lo, hi));
}

// Per-CTA set-up, once per kernel; the first barrier of a tile orders it before its uses.
template <int TH>
__device__ __forceinline__ void tile_setup(TileSmem<TH>& S)
{
  const int tid = threadIdx.x;
  if (tid < 4) S.cut[S.kWords + tid] = 0xFFFFFFFFu;
  if (tid < 16) {
    uint32_t m[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int nb = tid + 1 - 4 * k;  // bytes of the string in word k
      m[k] = nb >= 4 ? 0xFFFFFFFFu : nb <= 0 ? 0u : (1u << (8 * nb)) - 1u;
    }
    S.key_mask[tid] = make_uint4(m[0], m[1], m[2], m[3]);
  }
}

// Reset of the per-tile words; every thread calls it, a barrier follows.
template <int TH>
__device__ __forceinline__ void tile_reset(TileSmem<TH>& S)
{
  if (threadIdx.x < 16) S.hist[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    S.nmiss      = 0;
    S.nlong      = 0;
    S.over_start = -1;
    S.no_space   = 0;
  }
}

// ---- text -> bytes, tok and the start bitmap.  `cuts(mark)` calls mark(p) on some lanes of every warp for every further
//      start p in [0, wlen); each warp keeps those in the positions it has written itself.  Ends with a barrier. ----
template <int TH, class Cuts>
__device__ __forceinline__ void tile_cut(TileSmem<TH>& S, const Span& sp, const DeviceTable& T, Cuts cuts)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint8_t* text = sp.bytes + sp.lo;
  const bool aligned  = (reinterpret_cast<uintptr_t>(text) & 15u) == 0;
  uint16_t* cut16     = reinterpret_cast<uint16_t*>(S.cut);
  for (int g0 = warp * 32; g0 < S.kGroups; g0 += TH) {
    const int g = g0 + lane, p0 = g * 16;
    if (g0 * 16 >= sp.wlen) {  // nothing but the end of the window
      if (g < S.kGroups) cut16[g] = 0xFFFFu;
      continue;
    }
    uint4 x = make_uint4(0, 0, 0, 0);
    if (g < S.kGroups) {
      if (aligned && p0 >= sp.own_lo && p0 + 16 <= sp.wlen) {
        x = __ldg(reinterpret_cast<const uint4*>(text + p0));
      } else if (p0 < sp.wlen) {
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll 4
        for (int j = 0; j < 16; ++j) {
          const uint32_t c = (p0 + j >= sp.own_lo && p0 + j < sp.wlen) ? uint32_t(text[p0 + j]) : 0u;
          w[j >> 2] |= c << (8 * (j & 3));
        }
        x = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    uint32_t before = __shfl_up_sync(0xFFFFFFFFu, x.w, 1);
    if (lane == 0) before = (p0 > 0 || sp.has_prev) ? uint32_t(text[p0 - 1]) << 24 : 0u;
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    uint32_t acc = 0;  // bit 16 + i: the boundary in front of position i may merge
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t left = __funnelshift_r(k ? w[k - 1] : before, w[k], 24);  // byte in front of each of the four
      const uint32_t blk  = (w[k] >> 5) & 0x07070707u;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // index = block of the right byte << 8 | left byte; the upper half is the sign of a byte below 128: zero
        const uint32_t idx = prmt(left, blk, 0xCC40u + 0x1111u * uint32_t(e));
        const uint32_t row = __ldg(T.adj + idx);
        const uint32_t bit = __funnelshift_r(row, row, w[k] >> (8 * e));  // right byte & 31 selects the bit
        acc = __funnelshift_r(acc, bit, 1);
      }
    }
    uint32_t starts = ~(acc >> 16) & 0xFFFFu;
    if (p0 + 16 > sp.wlen) starts |= (p0 >= sp.wlen) ? 0xFFFFu : (0xFFFFu << (sp.wlen - p0)) & 0xFFFFu;
    if (sp.start_here && (sp.own_lo >> 4) == g) starts |= 1u << (sp.own_lo & 15);
    if (g < S.kGroups) {
      cut16[g] = uint16_t(starts);
      *reinterpret_cast<uint4*>(&S.bytes[16 + p0]) = x;
      uint4* t = reinterpret_cast<uint4*>(&S.tok[p0]);
      if (T.byte_ids_identity) {
        t[0] = make_uint4(prmt(x.x, 0u, 0x4140u), prmt(x.x, 0u, 0x4342u), prmt(x.y, 0u, 0x4140u), prmt(x.y, 0u, 0x4342u));
        t[1] = make_uint4(prmt(x.z, 0u, 0x4140u), prmt(x.z, 0u, 0x4342u), prmt(x.w, 0u, 0x4140u), prmt(x.w, 0u, 0x4342u));
      } else {
        for (int j = 0; j < 16; ++j) S.tok[p0 + j] = __ldg(T.byte_to_id + ((w[j >> 2] >> (8 * (j & 3))) & 0xFFu));
      }
    }
  }
  __syncwarp();
  cuts([&](int p) {
    if (!GTK_IN(p, S.kWin, 28)) return;
    if ((p >= S.kOwn ? 0 : p >> 9) == warp) atomicOr(&S.cut[p >> 5], 1u << (p & 31));
  });
  __syncthreads();
}

// the 16 bytes from window position `at` on
template <int TH>
__device__ __forceinline__ void window_words(const TileSmem<TH>& S, int at, uint32_t k[4])
{
  const uint32_t* wp = reinterpret_cast<const uint32_t*>(S.bytes + ((16 + at) & ~3));
  const uint32_t sh  = uint32_t(at & 3) * 8u;
  const uint32_t a0 = wp[0], a1 = wp[1], a2 = wp[2], a3 = wp[3], a4 = wp[4];
  k[0] = __funnelshift_r(a0, a1, sh);
  k[1] = __funnelshift_r(a1, a2, sh);
  k[2] = __funnelshift_r(a2, a3, sh);
  k[3] = __funnelshift_r(a3, a4, sh);
}

// A slot of the long table.  During a batch that learns, other threads fill empty slots word by word (see learn_segment):
// every word goes from zero to its final value once, and a filled slot has no zero in its last four words, so a slot that
// is seen half filled is recognised whatever order its words arrive in, and counts as empty.  A key word that has not
// arrived could only pass for the one that is looked for if that is zero too, four NUL bytes or what a string ends with:
// such strings are not looked up while the table is being added to (blank_word).
struct LongSlot {
  uint4 k, v;  // v = {meta, ids[3]}
};
__device__ __forceinline__ LongSlot load_long(const uint4* words, uint32_t slot)
{
  LongSlot s;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s.k.x), "=r"(s.k.y), "=r"(s.k.z), "=r"(s.k.w) : "l"(words + 2 * slot));
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s.v.x), "=r"(s.v.y), "=r"(s.v.z), "=r"(s.v.w) : "l"(words + 2 * slot + 1));
  return s;
}
// the same past L1, which may hold an old copy of a slot
__device__ __forceinline__ LongSlot load_long_l2(const uint4* words, uint32_t slot)
{
  LongSlot s;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s.k.x), "=r"(s.k.y), "=r"(s.k.z), "=r"(s.k.w) : "l"(words + 2 * slot));
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s.v.x), "=r"(s.v.y), "=r"(s.v.z), "=r"(s.v.w) : "l"(words + 2 * slot + 1));
  return s;
}
__device__ __forceinline__ uint32_t long_slot_of(const uint32_t k[4], uint32_t length)  // = long_slot() of the host
{
  uint32_t h = k[0] * 0x9E3779B1u ^ k[1] * 0x85EBCA77u ^ k[2] * 0xC2B2AE3Du ^ (k[3] + length) * 0x27D4EB2Fu;
  h ^= h >> 15;
  return (h * 0x2C1B3C6Du) >> (32 - kLongBits);
}
__device__ __forceinline__ bool long_matches(const LongSlot& s, const uint32_t k[4], uint32_t length)
{
  const uint32_t diff = (s.k.x ^ k[0]) | (s.k.y ^ k[1]) | (s.k.z ^ k[2]) | (s.k.w ^ k[3]) | ((s.v.x ^ length) & 31u);
  return diff == 0u && s.v.x != 0u && s.v.y != 0u && s.v.z != 0u && s.v.w != 0u;
}

__device__ __forceinline__ bool find_long(const DeviceTable& T, const uint32_t k[4], uint32_t length, LongSlot& at)
{
  const uint32_t h = long_slot_of(k, length);
  at         = load_long(T.long_words, h);
  bool found = long_matches(at, k, length);
  for (uint32_t hop = 1; !found && (at.v.x & kLongMore) && hop < kLongHops; ++hop) {
    at    = load_long(T.long_words, h ^ hop);
    found = long_matches(at, k, length);
  }
  if (T.learn && !found) {  // nothing that this SM's L1 knows of
    at    = load_long_l2(T.long_words, h);
    found = long_matches(at, k, length);
    for (uint32_t hop = 1; !found && (at.v.x & kLongMore) && hop < kLongHops; ++hop) {
      at    = load_long_l2(T.long_words, h ^ hop);
      found = long_matches(at, k, length);
    }
  }
  return found;
}

// one of the words that hold the L bytes of a key is zero
__device__ __forceinline__ bool blank_word(const uint32_t k[4], uint32_t L)
{
  return k[0] == 0u || (L > 4u && k[1] == 0u) || (L > 8u && k[2] == 0u) || (L > 12u && k[3] == 0u);
}

// Looks a listed segment up in the long table; a hit leaves its ids in tok and its live bits in the bitmap.
template <int TH>
__device__ __forceinline__ bool recall_segment(TileSmem<TH>& S, const DeviceTable& T, uint32_t ent)
{
  const uint32_t L = (ent & 15u) + 1u;
  const int s      = int(ent >> 4);
  const uint4 km   = S.key_mask[ent & 15u];
  uint32_t k[4];
  window_words(S, s, k);
  k[0] &= km.x, k[1] &= km.y, k[2] &= km.z, k[3] &= km.w;
  if (T.learn && blank_word(k, L)) return false;
  LongSlot at;
  if (!find_long(T, k, L, at)) return false;
  const uint32_t starts = at.v.x >> 16;
  S.tok[s]              = uint16_t((at.v.y & 0xFFFFu) - 1u);
  uint32_t m            = starts & (starts - 1u);
  const uint32_t id[5]  = {at.v.y >> 16, at.v.z & 0xFFFFu, at.v.z >> 16, at.v.w & 0xFFFFu, at.v.w >> 16};
#pragma unroll
  for (int e = 0; e < 5; ++e)
    if (m) {
      S.tok[s + __ffs(int(m)) - 1] = uint16_t(id[e] - 1u);
      m &= m - 1u;
    }
  mark_alive(S, s, starts);
  return true;
}

// A segment that has just been merged goes into the first empty slot of its row, if there is one.  A slot is claimed with
// its final meta word (see LongSlot for how a reader tells a slot that is still being filled); slots that are passed over
// get kLongMore.
template <int TH>
__device__ __forceinline__ void learn_segment(const TileSmem<TH>& S, uint4* words, int s, uint32_t L, uint32_t alive)
{
  if (__popc(alive) > kLongMaxIds) return;
  const uint4 km = S.key_mask[L - 1u];
  uint32_t k[4];
  window_words(S, s, k);
  k[0] &= km.x, k[1] &= km.y, k[2] &= km.z, k[3] &= km.w;
  const uint32_t h = long_slot_of(k, L), meta = L | alive << 16;
  uint32_t* slot   = nullptr;
  uint32_t taken[kLongHops];
#pragma unroll
  for (uint32_t hop = 0; hop < kLongHops; ++hop)
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(taken[hop]) : "l"(reinterpret_cast<uint32_t*>(words + 2 * (h ^ hop)) + 4));
#pragma unroll
  for (uint32_t hop = 0; hop < kLongHops; ++hop) {
    uint32_t* at = reinterpret_cast<uint32_t*>(words + 2 * (h ^ hop));
    if (slot) break;
    if (taken[hop] == 0u) taken[hop] = atomicCAS(at + 4, 0u, meta);
    if (taken[hop] == 0u) slot = at;
    else if (taken[hop] == meta) return;  // most likely this very segment, merged by another CTA meanwhile
    else if (!(taken[hop] & kLongMore)) atomicOr(at + 4, kLongMore);
  }
  if (!slot) return;
  uint32_t id[kLongMaxIds];
#pragma unroll
  for (int e = 0; e < kLongMaxIds; ++e) {
    id[e] = alive ? uint32_t(S.tok[s + __ffs(int(alive)) - 1]) + 1u : 0xFFFFu;
    alive &= alive - 1u;
  }
  *reinterpret_cast<uint4*>(slot) = make_uint4(k[0], k[1], k[2], k[3]);
  slot[5] = id[0] | id[1] << 16;
  slot[6] = id[2] | id[3] << 16;
  slot[7] = id[4] | id[5] << 16;
}

// ---- One batch of at most 32 misses, one segment per lane, merged to the end (Algorithm 1 inside the segment).
//      Ranks of the pairs, 16 bits each, in a lane-interleaved scratch: slot i of a lane in half i & 1 of word
//      (i >> 1) * 32.  slots (8 or 16, uniform) covers the longest segment.  A step merges the left-most pair of lowest
//      rank, starts the probes of the two pairs next to the new token (one 128-bit bucket load each), takes the minimum of
//      all other pairs while they are on their way, and folds the two new ranks in. ----
template <int TH>
__device__ __noinline__ void merge_batch(uint32_t ent, int slots, int scratch_word, PairTable P, const uint16_t* info,
                                         uint4* learned)
{
  TileSmem<TH>& S = tile_smem<TH>();
  const int L = int(ent & 15u) + 1;
  int s       = int(ent >> 4);
  if (!GTK_IN(s + L, S.kWin + 1, 15)) s = 0, ent = 0;
  if (!GTK_IN((scratch_word + 16 * slots) * 4, S.kScratchBytes + 1, 14)) return;
  uint32_t* scr = reinterpret_cast<uint32_t*>(S.work) + scratch_word + (threadIdx.x & 31);
  uint16_t* tok = S.tok + s;
  {
    uint32_t k[5];
    window_words(S, s, k);
    k[4] = 0;
    for (int i0 = 0; i0 < slots; i0 += 8) {
      uint32_t r[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {  // left byte << 8 | right byte of the pair in slot i0 + e
        const uint32_t idx = (e & 3) < 3 ? prmt(k[e >> 2], 0u, 0x4400u | uint32_t(e & 3) << 4 | uint32_t((e & 3) + 1))
                                         : prmt(k[e >> 2], k[(e >> 2) + 1], 0x0034u) & 0xFFFFu;
        r[e] = NONE;
        if (i0 + e + 1 < L) r[e] = __ldg(info + idx);
      }
#pragma unroll
      for (int e = 0; e < 8; e += 2) scr[((i0 + e) >> 1) * 32] = r[e] | r[e + 1] << 16;
      k[0] = k[2], k[1] = k[3], k[2] = 0;
    }
  }
  uint32_t alive = (ent != 0) ? (2u << (L - 1)) - 1u : 0u;
  auto lowest    = [&]() {
    uint32_t b = 0xFFFFFFFFu;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t x = scr[w * 32];
      b = __vimin3_u32(b, (x << 16) | uint32_t(2 * w), (x & 0xFFFF0000u) | uint32_t(2 * w + 1));
    }
    if (slots > 8) {
#pragma unroll
      for (int w = 4; w < 8; ++w) {
        const uint32_t x = scr[w * 32];
        b = __vimin3_u32(b, (x << 16) | uint32_t(2 * w), (x & 0xFFFF0000u) | uint32_t(2 * w + 1));
      }
    }
    return b;
  };
  auto set_rank = [&](int i, uint32_t v) { reinterpret_cast<uint16_t*>(scr + (i >> 1) * 32)[i & 1] = uint16_t(v); };
  uint32_t best = lowest();
  while (__any_sync(0xFFFFFFFFu, best < (SEL << 16))) {
    if (best < (SEL << 16)) {
      const int j = int(best & 0xFFFFu);
      uint32_t t  = alive & (0xFFFFFFFEu << j);
      const int q = __ffs(int(t)) - 1;  // next live slot: the right token of the pair
      if (!(GTK_IN(j, L - 1, 17) && GTK_IN(q, L, 18))) {
        best = 0xFFFFFFFFu;
        continue;
      }
      t &= t - 1;  // live slots behind the pair
      alive ^= 1u << q;
      const uint32_t left = alive & ((1u << j) - 1u);
      const uint32_t c    = P.merged_of_rank ? __ldg(P.merged_of_rank + (best >> 16)) : 256u + (best >> 16);
      const int p         = 31 - __clz(int(left));
      uint32_t key_r = 0, key_l = 0;
      uint4 vr = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu), vl = vr;
      if (t) {
        key_r = (c << 16) | uint32_t(tok[__ffs(int(t)) - 1]);
        vr    = __ldg(P.buckets + ((key_r * 0x9E3779B1u) >> 16));
      }
      if (left) {
        key_l = (uint32_t(tok[p]) << 16) | c;
        vl    = __ldg(P.buckets + ((key_l * 0x9E3779B1u) >> 16));
        set_rank(p, NONE);
      }
      tok[j] = uint16_t(c);
      set_rank(q, NONE);
      set_rank(j, NONE);
      best = lowest();  // every pair but the two new ones
      if (t) {
        const uint32_t r = resolve_rank_raw(vr, key_r, P.overflow, P.overflow_mask);
        if (r < SEL) {
          set_rank(j, r);
          best = min(best, (r << 16) | uint32_t(j));
        }
      }
      if (left) {
        const uint32_t r = resolve_rank_raw(vl, key_l, P.overflow, P.overflow_mask);
        if (r < SEL) {
          set_rank(p, r);
          best = min(best, (r << 16) | uint32_t(p));
        }
      }
    }
  }
  if (ent) {
    mark_alive(S, s, alive);
    if (learned) learn_segment(S, learned, s, uint32_t(L), alive);
  }
}

// ---- One or two misses of a warp: half a warp each, one token per lane, so that a step is a few shuffles and one table
//      load deep instead of the hundred instructions of merge_batch (a tile with one miss: 6 instead of 12 thousand cycles,
//      during which the rest of the CTA waits).  Lane i of a half holds the i-th live token, its byte offset in the segment
//      and the rank of the pair with its right neighbour.  ent: the half's segment, 0 = none. ----
template <int TH>
__device__ __noinline__ void merge_two(uint32_t ent, PairTable P, const uint16_t* info, uint4* learned)
{
  TileSmem<TH>& S = tile_smem<TH>();
  const int lane = threadIdx.x & 31, i = lane & 15;
  const int L    = int(ent & 15u) + 1;
  int s              = int(ent >> 4);
  if (!GTK_IN(s + L, S.kWin + 1, 15)) s = 0;
  int n       = ent ? L : 0;
  uint32_t t  = S.tok[s + i];
  int at      = i;
  uint32_t rk = NONE;
  if (i + 1 < n) rk = __ldg(info + ((uint32_t(S.bytes[16 + s + i]) << 8) | S.bytes[17 + s + i]));
  // the row of the long table is read while the ranks are on their way
  uint32_t k[4] = {0, 0, 0, 0}, h = 0, meta = 1;
  if (learned && ent) {
    const uint4 km = S.key_mask[L - 1];
    window_words(S, s, k);
    k[0] &= km.x, k[1] &= km.y, k[2] &= km.z, k[3] &= km.w;
    h = long_slot_of(k, uint32_t(L));
    if (i < int(kLongHops))
      asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(meta) : "l"(reinterpret_cast<uint32_t*>(learned + 2 * (h ^ uint32_t(i))) + 4));
  }
  if (i + 1 >= n) rk = NONE;
  for (;;) {
    uint32_t best = (min(rk, NONE) << 16) | uint32_t(i);
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) best = min(best, __shfl_xor_sync(0xFFFFFFFFu, best, d));
    const bool act = best < (SEL << 16);
    if (!__any_sync(0xFFFFFFFFu, act)) break;
    const int j      = int(best & 15u);
    const uint32_t c = P.merged_of_rank ? (act ? __ldg(P.merged_of_rank + (best >> 16)) : 0u) : 256u + (best >> 16);
    const uint32_t t1 = __shfl_down_sync(0xFFFFFFFFu, t, 1, 16), r1 = __shfl_down_sync(0xFFFFFFFFu, rk, 1, 16);
    const int at1     = __shfl_down_sync(0xFFFFFFFFu, at, 1, 16);
    if (act) {
      if (i > j) t = t1, at = at1, rk = r1;
      if (i == j) t = c;
      --n;
    }
    const uint32_t next = __shfl_down_sync(0xFFFFFFFFu, t, 1, 16);
    if (act && (i == j || i + 1 == j)) {
      rk = NONE;
      if (i + 1 < n) {
        const uint32_t key = (t << 16) | next;
        rk = resolve_rank(__ldg(P.buckets + ((key * 0x9E3779B1u) >> 16)), key, P.overflow, P.overflow_mask);
      }
    }
  }
  if (i < n && GTK_IN(s + at, S.kWin, 12)) S.tok[s + at] = uint16_t(t);
  uint32_t alive = i < n ? 1u << at : 0u;
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) alive |= __shfl_xor_sync(0xFFFFFFFFu, alive, d);
  if (i == 0 && ent) mark_alive(S, s, alive);
  if (learned) {
    // first empty slot of the row; if another CTA takes it first the segment is simply not learned this time
    const uint32_t want  = uint32_t(L) | alive << 16;
    const uint32_t empty = (__ballot_sync(0xFFFFFFFFu, meta == 0u) >> (lane & 16)) & 0xFFFFu;
    const bool there     = ((__ballot_sync(0xFFFFFFFFu, i < int(kLongHops) && (meta & ~kLongMore) == want) >> (lane & 16)) & 0xFFFFu) != 0u;
    const int hop        = __ffs(int(empty)) - 1;
    bool mine            = ent != 0 && hop >= 0 && hop < int(kLongHops) && !there && __popc(alive) <= kLongMaxIds;
    uint32_t* slot       = reinterpret_cast<uint32_t*>(learned + 2 * (h ^ uint32_t(max(hop, 0))));
    if (mine && i < hop && !(meta & kLongMore)) atomicOr(reinterpret_cast<uint32_t*>(learned + 2 * (h ^ uint32_t(i))) + 4, kLongMore);
    uint32_t was = 1;
    if (mine && i == 0) was = atomicCAS(slot + 4, 0u, want);
    was  = __shfl_sync(0xFFFFFFFFu, was, 0, 16);
    mine = mine && was == 0u;
    // the ids, two to a word, from the lanes that hold them
    const uint32_t mine_id = (i < n) ? t + 1u : 0xFFFFu;
    const uint32_t hi_id   = __shfl_down_sync(0xFFFFFFFFu, mine_id, 1, 16);
    if (mine && i == 0) *reinterpret_cast<uint4*>(slot) = make_uint4(k[0], k[1], k[2], k[3]);
    if (mine && (i & 1) == 0 && i < kLongMaxIds) slot[5 + (i >> 1)] = mine_id | hi_id << 16;
  }
}

// ---- A long segment is hardly ever anything but a run of one byte with a few others around it.  One warp merges it as a
//      list of (token, count) items, one per lane: a step merges either the pair inside an item, all its occurrences at
//      once (left to right, which is what Algorithm 1 does over consecutive steps when no merge exposes a lower rank), or
//      one pair across two items; it costs one round of table loads and some shuffles whatever the length of the run, where
//      the pass routine sweeps the whole segment once per merge rank.  The segment's L tokens, still its bytes, stand at s
//      and make way for the ids; list: room for 32 entries.  Returns the number of ids, or -1 when the segment has too many items (tok is then
//      unchanged).  Monotone tables only. ----
constexpr int kRunItems = 30;
constexpr int kRunKept  = 3;           // items of a result that learn_run can keep
constexpr int kRunMany  = 0x10000;     // flag on the result of merge_runs: more than that
template <int TH>
__device__ __noinline__ int merge_runs(int s, uint16_t* list, int L, const PairTable P)
{
  TileSmem<TH>& S   = tile_smem<TH>();
  uint16_t* tok     = S.tok + s;
  const int lane    = threadIdx.x & 31;
  int m             = 0;  // items
  uint32_t carry    = 0;  // last byte of the 256 before
  for (int base = 0; base < L; base += 256) {  // eight bytes per lane
    const int i0 = base + 8 * lane;
    uint32_t x0 = 0, x1 = 0;
    if (i0 < L) {
      const int at       = 16 + s + i0;
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(S.bytes + (at & ~3));
      const uint32_t sh  = uint32_t(at & 3) * 8u;
      x0 = __funnelshift_r(wp[0], wp[1], sh);
      x1 = __funnelshift_r(wp[1], wp[2], sh);
    }
    uint32_t before = __shfl_up_sync(0xFFFFFFFFu, x1, 1);
    if (lane == 0) before = carry;
    carry = __shfl_sync(0xFFFFFFFFu, x1, 31);
    const uint32_t d0 = __vcmpne4(x0, __funnelshift_l(before, x0, 8)), d1 = __vcmpne4(x1, __funnelshift_l(x0, x1, 8));
    uint32_t starts   = (((d0 & 0x01010101u) * 0x01020408u) >> 24 & 15u) | ((((d1 & 0x01010101u) * 0x01020408u) >> 20) & 0xF0u);
    if (i0 == 0) starts |= 1u;
    starts &= low_bits(max(min(L - i0, 8), 0));
    const int cnt = __popc(starts);
    int inc       = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += y;
    }
    const int total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    if (m + total > kRunItems) return -1;
    for (int at = m + inc - cnt; starts; starts &= starts - 1) list[at++] = uint16_t(i0 + __ffs(int(starts)) - 1);
    m += total;
  }
  __syncwarp();
  // tc = token << 16 | count; rank = rank of (t, t) << 16 | rank of (t, next item's token)
  const int start = lane < m ? int(list[lane]) : L;
  uint32_t tc     = uint32_t(__shfl_down_sync(0xFFFFFFFFu, start, 1) - start);
  tc              = lane < m ? uint32_t(tok[start]) << 16 | tc : 0xFFFF0000u;
  uint32_t rank   = 0xFFFFFFFFu;
  auto probe = [&](uint32_t next, bool inner, bool cross) {  // both loads leave before anything waits for them
    const uint32_t t = tc >> 16, key_i = t << 16 | t, key_c = t << 16 | next;
    uint4 vi = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu), vc = vi;
    if (inner) vi = __ldg(P.buckets + ((key_i * 0x9E3779B1u) >> 16));
    if (cross) vc = __ldg(P.buckets + ((key_c * 0x9E3779B1u) >> 16));
    if (inner) rank = (rank & 0xFFFFu) | resolve_rank(vi, key_i, P.overflow, P.overflow_mask) << 16;
    if (cross) rank = (rank & 0xFFFF0000u) | resolve_rank(vc, key_c, P.overflow, P.overflow_mask);
  };
  probe(__shfl_down_sync(0xFFFFFFFFu, tc, 1) >> 16, lane < m && (tc & 0xFFFFu) >= 2u, lane + 1 < m);
  for (int step = 0; step < 2 * L; ++step) {
    const uint32_t in = (tc & 0xFFFFu) >= 2u ? rank >> 16 : NONE, cross = rank & 0xFFFFu;
    const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, (min(in, cross) << 6) | uint32_t(lane << 1) | (in <= cross ? 0u : 1u));
    const uint32_t r    = best >> 6;
    if (r >= SEL || m > kRunItems) break;
    const int a       = int(best >> 1) & 31;
    const uint32_t c  = P.merged_of_rank ? __ldg(P.merged_of_rank + r) : 256u + r;
    const uint32_t xa = __shfl_sync(0xFFFFFFFFu, tc, a), xb = __shfl_sync(0xFFFFFFFFu, tc, a + 1);
    const uint32_t na = xa & 0xFFFFu, nb = xb & 0xFFFFu;
    // the items that take the place of item a (and a + 1)
    uint32_t y0, y1, y2 = 0;
    int k, w;
    if ((best & 1u) == 0u) {
      w  = 1;
      y0 = c << 16 | na >> 1;
      y1 = (xa & 0xFFFF0000u) | 1u;
      k  = 1 + int(na & 1u);
    } else {
      w = 2;
      const bool keep_a = na > 1u, keep_b = nb > 1u;
      const uint32_t one = c << 16 | 1u;
      y0 = keep_a ? xa - 1u : one;
      y1 = keep_a ? one : xb - 1u;
      y2 = xb - 1u;
      k  = 1 + int(keep_a) + int(keep_b);
    }
    const int from    = (lane - (k - w)) & 31;
    const uint32_t st = __shfl_sync(0xFFFFFFFFu, tc, from), sr = __shfl_sync(0xFFFFFFFFu, rank, from);
    m += k - w;
    if (lane >= a + k) tc = st, rank = sr;
    const int e = lane - a;
    if (e >= 0 && e < k) {
      tc   = e == 0 ? y0 : e == 1 ? y1 : y2;
      rank = 0xFFFFFFFFu;
    }
    if (lane >= m) tc = 0xFFFF0000u, rank = 0xFFFFFFFFu;
    const uint32_t next = __shfl_down_sync(0xFFFFFFFFu, tc, 1) >> 16;
    if (e == -1) rank |= 0xFFFFu;
    probe(next, e >= 0 && e < k && lane < m && (tc & 0xFFFFu) >= 2u, e >= -1 && e < k && lane + 1 < m);
  }
  int inc = int(tc & 0xFFFFu);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
    if (lane >= d) inc += y;
  }
  __syncwarp();
  for (int i = 0; i < m; ++i) {
    const uint32_t x = __shfl_sync(0xFFFFFFFFu, tc, i);
    const int hi = __shfl_sync(0xFFFFFFFFu, inc, i), lo = hi - int(x & 0xFFFFu);
    for (int j = lo + lane; j < hi; j += 32)
      if (GTK_IN(j, L, 13)) tok[j] = uint16_t(x >> 16);
  }
  const int len = __shfl_sync(0xFFFFFFFFu, inc, 31);
  if (lane < kRunKept) reinterpret_cast<uint32_t*>(list)[lane] = lane < m ? tc : 0xFFFF0000u;  // for learn_run
  __syncwarp();
  return m > kRunItems ? -2 - len : m > kRunKept ? len | kRunMany : len;
}

// Runs are remembered too, in a batch that learns: a long segment of up to three runs of a byte (a rule of dashes, padding in
// front of a number) that ends as up to three runs of a token.  Key: bytes, where the runs start, length, and a word that no
// text has in that place together with length code 31.  Value: token + 1 | count << 16 of each run.  A third of the time of
// merge_runs, whose code is hardly ever in the instruction cache.
constexpr uint32_t kRunCode = 31u;
template <int TH>
__device__ __forceinline__ bool run_key(const TileSmem<TH>& S, int s, int L, uint32_t k[4])
{
  if (L > 256) return false;
  const int lane = threadIdx.x & 31, i0 = 8 * lane;
  uint32_t starts = 0;
  if (i0 < L) {  // starts of runs among eight bytes, but for the first of the segment
    const int at       = 16 + s + i0;
    const uint32_t* wp = reinterpret_cast<const uint32_t*>(S.bytes + (at & ~3));
    const uint32_t sh  = uint32_t(at & 3) * 8u;
    const uint32_t x0 = __funnelshift_r(wp[0], wp[1], sh), x1 = __funnelshift_r(wp[1], wp[2], sh);
    const uint32_t d0 = __vcmpne4(x0, x0 << 8 | S.bytes[at - 1]), d1 = __vcmpne4(x1, __funnelshift_l(x0, x1, 8));
    starts = (((d0 & 0x01010101u) * 0x01020408u) >> 24 & 15u) | ((((d1 & 0x01010101u) * 0x01020408u) >> 20) & 0xF0u);
    starts &= low_bits(L - i0) & (lane == 0 ? 0xFEu : 0xFFu);
  }
  if (__reduce_add_sync(0xFFFFFFFFu, __popc(starts)) > 2) return false;
  const int p1 = int(__reduce_min_sync(0xFFFFFFFFu, starts ? uint32_t(i0 + __ffs(int(starts)) - 1) : uint32_t(L)));
  const int p2 = int(__reduce_max_sync(0xFFFFFFFFu, starts ? uint32_t(i0 + 31 - __clz(int(starts))) : 0u));
  const uint8_t* bp = S.bytes + 16 + s;
  k[0] = uint32_t(bp[0]) | uint32_t(bp[p1 < L ? p1 : 0]) << 8 | uint32_t(bp[p2]) << 16 | 1u << 24;
  k[1] = uint32_t(p1) | uint32_t(p2) << 16;  // p1 > 0
  k[2] = uint32_t(L);
  k[3] = 0x736E7572u;
  return true;
}
template <int TH>
__device__ __noinline__ int recall_run(int s, int L, const DeviceTable& T)
{
  TileSmem<TH>& S = tile_smem<TH>();
  uint32_t k[4];
  LongSlot at;
  if (!run_key(S, s, L, k)) return -1;
  // the slot may be filled just now: what the first lane has seen holds for the warp
  const bool found = find_long(T, k, kRunCode, at);
  if (!__shfl_sync(0xFFFFFFFFu, found, 0)) return -1;
  at.v.y = __shfl_sync(0xFFFFFFFFu, at.v.y, 0);
  at.v.z = __shfl_sync(0xFFFFFFFFu, at.v.z, 0);
  at.v.w = __shfl_sync(0xFFFFFFFFu, at.v.w, 0);
  const int n0 = int(at.v.y >> 16), n1 = n0 + int(at.v.z >> 16), n2 = n1 + int(at.v.w >> 16);
  for (int j = threadIdx.x & 31; j < n2; j += 32)
    if (GTK_IN(j, L, 16)) S.tok[s + j] = uint16_t(((j < n0 ? at.v.y : j < n1 ? at.v.z : at.v.w) & 0xFFFFu) - 1u);
  __syncwarp();
  return n2;
}
template <int TH>
__device__ __noinline__ void learn_run(int s, int L, const uint32_t* items, uint4* words)
{
  const int lane = threadIdx.x & 31;
  uint32_t k[4];
  if (!run_key(tile_smem<TH>(), s, L, k)) return;
  const uint32_t h = long_slot_of(k, kRunCode), want = kRunCode | (k[0] * 0x9E3779B1u ^ k[1] * 0x85EBCA77u ^ k[2]) << 16;
  uint32_t meta = 1;
  if (lane < int(kLongHops))
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(meta) : "l"(reinterpret_cast<uint32_t*>(words + 2 * (h ^ uint32_t(lane))) + 4));
  const int hop = __ffs(int(__ballot_sync(0xFFFFFFFFu, meta == 0u))) - 1;  // first empty slot of the row
  if (hop < 0 || __any_sync(0xFFFFFFFFu, (meta & ~kLongMore) == want)) return;
  uint32_t* slot = reinterpret_cast<uint32_t*>(words + 2 * (h ^ uint32_t(hop)));
  if (lane < hop && !(meta & kLongMore)) atomicOr(reinterpret_cast<uint32_t*>(words + 2 * (h ^ uint32_t(lane))) + 4, kLongMore);
  uint32_t was = 1;
  if (lane == 0) was = atomicCAS(slot + 4, 0u, want);
  if (__shfl_sync(0xFFFFFFFFu, was, 0) != 0u) return;  // taken meanwhile
  if (lane == 0) *reinterpret_cast<uint4*>(slot) = make_uint4(k[0], k[1], k[2], k[3]);
  if (lane < kRunKept) slot[5 + lane] = ((items[lane] >> 16) + 1u & 0xFFFFu) | items[lane] << 16 | (items[lane] == 0xFFFF0000u ? 0xFFFFu : 0u);
}

// ---- multi-byte segments, every warp those that start in its own 512 positions: listed, looked up in the table of short
//      strings, what is left in the table of long ones.  One or two misses are merged on the spot (a batch that learns has
//      hardly more), others join the CTA's list, as the long segments do theirs.  Ends with a barrier. ----
template <int TH>
__device__ __forceinline__ void tile_lookup(TileSmem<TH>& S, const Span& sp, const DeviceTable& T, int* status)
{
  using Entry = typename TileSmem<TH>::Entry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = lanemask_lt();
  // Everything that is read from the bitmap of starts is read in front of the barrier, because segments that are done mark
  // their tokens in it, also those that reach into the next warp's positions.
  const int base    = tid * 16;
  const uint32_t w0 = S.cut[tid >> 1], w1 = S.cut[(tid >> 1) + 1], w2 = S.cut[(tid >> 1) + 2];
  const uint32_t a  = __funnelshift_r(w0, w1, (tid & 1) * 16), a2 = __funnelshift_r(w1, w2, (tid & 1) * 16);  // 64 positions from base on
  uint32_t m = a & ~(a >> 1) & range_mask(base, sp.own_lo, sp.own_hi) & 0xFFFFu;  // starts whose next position is no start
  if (m) {  // only the last of the segments that start in sixteen positions can be a long one
    const int b = 31 - __clz(int(m));
    if (unsigned(__ffs(int(__funnelshift_r(a, a2, b + 1))) - 1) >= unsigned(kThreadSegMax)) {
      const int long_at = base + b;
      m ^= 1u << b;
      if (next_cut(S, long_at) >= S.kWin && sp.wlen == S.kWin) {
        S.over_start = long_at;
      } else {
        const int q = atomicAdd(&S.nlong, 1);
        if (q < S.kLong && GTK_IN(long_at, S.kOwn, 3)) S.longq[q] = uint16_t(long_at);
        else atomicMax(status, int(kStatusLongQueueOverflow));
      }
    }
  }
  if (warp == TileSmem<TH>::kWarps - 1 && lane == 0) {
    S.first = next_cut(S, sp.own_lo - 1);
    S.end   = min(next_cut(S, sp.own_hi - 1), sp.wlen);
  }
  __syncthreads();
  if (warp * 512 < sp.own_hi) {
    Entry* list = S.work + warp * TileSmem<TH>::kRegion;
    int tot;
    {
      const int cnt = __popc(m);
      int inc       = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= d) inc += y;
      }
      tot    = __shfl_sync(0xFFFFFFFFu, inc, 31);
      int at = inc - cnt;
      while (m) {
        const int b = __ffs(int(m)) - 1;
        m &= m - 1;
        const int len = __ffs(int(__funnelshift_r(a, a2, b + 1)));
        if (GTK_IN(at, 256, 4)) list[at] = Entry(((base + b) << 4) | (len - 1));
        ++at;
      }
    }
    __syncwarp();
    int nrest = 0;  // entries that are left, at the front of the list
    for (int r = 0; r < tot; r += 64) {  // two loads in flight per lane: 16 MiB 169 -> 150 us; four: the same
      uint32_t ent[2], p[2], k1[2];
      uint2 v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i  = r + 32 * e + lane;
        ent[e]       = i < tot ? uint32_t(list[i]) : 0u;
        const int L  = int(ent[e] & 15u) + 1;
        const int at = 16 + int(ent[e] >> 4);
        const uint32_t* wp = reinterpret_cast<const uint32_t*>(S.bytes + (at & ~3));
        const uint32_t sh  = uint32_t(at & 3) * 8u;
        const uint32_t a0 = wp[0], a1 = wp[1], a2 = wp[2];
        const uint32_t k0 = __funnelshift_r(a0, a1, sh) & low_bits(8 * L);
        k1[e] = (__funnelshift_r(a1, a2, sh) & low_bits(max(8 * L - 32, 0))) | uint32_t(L) << 24;
        p[e]  = k0 * kShortMulA;
        v[e]  = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);  // an empty place: whatever k1 is, bits 16 and 17 of the id stay set
        if (L <= kShortMaxBytes) v[e] = __ldg(T.short_words + ((p[e] ^ (k1[e] * kShortMulB)) >> (32 - kShortBits)));
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t id = v[e].y ^ (p[e] << kShortBits);
        bool left         = ent[e] != 0;
        if (left && v[e].x == k1[e] && id < 0x10000u) {
          S.tok[ent[e] >> 4] = uint16_t(id);
          left               = false;
        }
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, left);
        if (left && GTK_IN(nrest + __popc(bal & lt), 256, 5)) list[nrest + __popc(bal & lt)] = Entry(ent[e]);
        nrest += __popc(bal);
      }
    }
    __syncwarp();
    int nmiss = 0;
    for (int r = 0; r < nrest; r += 32) {
      const uint32_t ent = (r + lane < nrest) ? uint32_t(list[r + lane]) : 0u;
      const bool miss    = ent != 0 && !recall_segment(S, T, ent);
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, miss);
      if (miss && GTK_IN(nmiss + __popc(bal & lt), 256, 8)) list[nmiss + __popc(bal & lt)] = Entry(ent);
      nmiss += __popc(bal);
    }
    __syncwarp();
    if (nmiss > 2) {
      int at = 0;
      if (lane == 0) at = atomicAdd(&S.nmiss, nmiss);
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      const int room = max(min(nmiss, TileSmem<TH>::kMisses - at), 0);
      nmiss -= room;  // what finds no room there (text of nothing but misses) stays with the warp
      for (int i = lane; i < room; i += 32) S.miss[at + i] = list[nmiss + i];
    }
    for (int i = 0; i < nmiss; i += 2) {
      const int k = i + (lane >> 4);
      merge_two<TH>(k < nmiss ? uint32_t(list[k]) : 0u, pair_table(T), T.byte_pair_info, T.learn ? T.long_words : nullptr);
    }
  }
  __syncthreads();
}

// One warp merges each segment of the long list, as runs or else pass by pass with the ranks in its region; what is too
// long for that stays on the list (the others are struck off) for the whole CTA.
constexpr uint32_t kStruck = 0xFFFFu;
template <int TH>
__device__ __noinline__ void merge_long_segments(const DeviceTable& T, int* status)
{
  TileSmem<TH>& S = tile_smem<TH>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nl   = min(S.nlong, S.kLong);
  uint16_t* area = S.region(warp);
  for (int q = warp; q < nl; q += S.kWarps) {
    const int s = S.longq[q];
    const int L = next_cut(S, s) - s;
    if (!(GTK_IN(s, S.kWin, 19) && GTK_IN(s + L, S.kWin + 1, 20))) continue;
    int len = -1;
    if (T.monotone) {
      if (T.learn) len = recall_run<TH>(s, L, T);
      if (len < 0) {
        len = merge_runs<TH>(s, area, L, pair_table(T));
        if (T.learn && len >= 0 && !(len & kRunMany)) learn_run<TH>(s, L, reinterpret_cast<const uint32_t*>(area), T.long_words);
        if (len >= 0) len &= kRunMany - 1;
      }
    }
    if (len < 0) {
      // too many different tokens (len -1: from the start; else -2 - len tokens are left to go on with)
      const int left = len == -1 ? L : -2 - len;
      if (left > S.kRegion) continue;
      for (int i = lane; i < left; i += 32)
        area[i] = (i + 1 < left) ? uint16_t(probe_rank(T, S.tok[s + i], S.tok[s + i + 1])) : uint16_t(NONE);
      __syncwarp();
      len = group_merge_dense<1>(S.tok + s, area, left, T, nullptr, status);
    }
    mark_alive_range(S, s + 1, s + len, lane);
    if (lane == 0) S.longq[q] = uint16_t(kStruck);
    __syncwarp();
  }
}

// What is left of the long list: the whole CTA, in an HBM workspace (two arrays of scratch_tokens slots).
template <int TH>
__device__ __noinline__ void merge_huge_segments(uint16_t* scratch, int64_t scratch_tokens, const DeviceTable& T, int* status)
{
  TileSmem<TH>& S = tile_smem<TH>();
  const int tid = threadIdx.x;
  const int nl  = min(S.nlong, S.kLong);
  for (int q = 0; q < nl; ++q) {
    const uint32_t s = S.longq[q];
    if (s == kStruck) continue;
    const int L = next_cut(S, int(s)) - int(s);
    if (scratch == nullptr || L > scratch_tokens) {
      if (tid == 0) S.no_space = 1;
      continue;
    }
    for (int i = tid; i < L; i += TH) {
      const uint32_t u = S.bytes[16 + s + i];
      scratch[i]       = __ldg(T.byte_to_id + u);
      scratch[scratch_tokens + i] = (i + 1 < L) ? __ldg(T.byte_pair_rank + ((u << 8) | S.bytes[17 + s + i])) : uint16_t(NONE);
    }
    __syncthreads();
    const int len = group_merge<TH / 32>(scratch, scratch + scratch_tokens, L, T, S.gs(), status);
    __syncthreads();
    for (int i = tid; i < len; i += TH) S.tok[s + i] = scratch[i];
    if (tid < 32) mark_alive_range(S, int(s) + 1, int(s) + len, tid);
    __syncthreads();
  }
  __syncthreads();  // no_space: the whole CTA decides by it what comes next
}

// ---- the listed misses and the long segments.  Ends with a barrier when there are any. ----
template <int TH>
__device__ __forceinline__ void tile_merge(TileSmem<TH>& S, const DeviceTable& T, uint16_t* scratch, int64_t scratch_tokens,
                                           int* status)
{
  using Entry = typename TileSmem<TH>::Entry;
  constexpr int NW  = TileSmem<TH>::kWarps;
  constexpr int cap = TileSmem<TH>::kScratchBytes / 128;  // columns of 32 words in the scratch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n   = min(S.nmiss, S.kMisses);
  if (n > 0 && n <= 2 * NW) {  // few: two for each warp, quicker than one warp's loop over all (128-byte call 20.8 -> 19.7 us)
    const int k = 2 * warp + (lane >> 4);
    if (2 * warp < n)
      merge_two<TH>(k < n ? uint32_t(S.miss[k]) : 0u, pair_table(T), T.byte_pair_info, T.learn ? T.long_words : nullptr);
    __syncthreads();
  } else if (n > 0) {  // CTA-uniform
    Entry* ml = S.miss;
    if (n > 32) {
      // counting sort, longest first, so that the lanes of a warp work on segments of similar length
      constexpr int kPer = (TileSmem<TH>::kMisses + TH - 1) / TH;
      uint32_t e[kPer];
      int slot[kPer];
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int i = tid + k * TH;
        e[k]        = (i < n) ? uint32_t(ml[i]) : 0u;
        slot[k]     = (i < n) ? atomicAdd(&S.hist[e[k] & 15u], 1) : 0;
      }
      __syncthreads();
      const int v = (lane < 16) ? S.hist[15 - lane] : 0;
      int inc     = v;
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= d) inc += y;
      }
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int at = __shfl_sync(0xFFFFFFFFu, inc - v, 15 - int(e[k] & 15u)) + slot[k];
        if (tid + k * TH < n && GTK_IN(at, n, 9)) ml[at] = Entry(e[k]);
      }
      __syncthreads();
    }
    // Batches of 32 (at most 16); a batch needs four or eight columns of the scratch.  Every warp works out the same
    // schedule.
    const int nb = (n + 31) >> 5;
    int need     = 0;
    if (n > 32) {
      if (lane < nb) need = (ml[lane * 32] & 15u) >= 8u ? 8 : 4;
    } else {
      const uint32_t longest = __reduce_max_sync(0xFFFFFFFFu, (lane < n) ? uint32_t(ml[lane] & 15u) : 0u);
      if (lane == 0) need = longest >= 8u ? 8 : 4;
    }
    int pre = need;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, pre, d);
      if (lane >= d) pre += y;
    }
    auto run = [&](int b, int base) {  // batch b, its columns counted from column `base` of the schedule
      const int cols = __shfl_sync(0xFFFFFFFFu, need, b);
      const int col  = __shfl_sync(0xFFFFFFFFu, pre, b) - cols - base;
      const int i    = b * 32 + lane;
      merge_batch<TH>((i < n) ? uint32_t(ml[i]) : 0u, 2 * cols, col * 32, pair_table(T), T.byte_pair_info,
                      T.learn ? T.long_words : nullptr);
    };
    for (int b0 = 0; b0 < nb;) {  // one round in the usual case
      const int base    = b0 ? __shfl_sync(0xFFFFFFFFu, pre, b0 - 1) : 0;
      const uint32_t in = __ballot_sync(0xFFFFFFFFu, lane >= b0 && lane < nb && lane < b0 + 2 * NW && pre - base <= cap);
      const int cnt     = max(__popc(in), 1);
      // a warp that takes one of the longest batches takes none or one of the shortest
      if (warp < cnt) run(b0 + warp, base);
      if (2 * NW - 1 - warp < cnt) run(b0 + 2 * NW - 1 - warp, base);
      b0 += cnt;
      __syncthreads();
    }
  }
  if (S.nlong > 0) {  // CTA-uniform
    merge_long_segments<TH>(T, status);
    const bool more = S.nlong > 0 && __syncthreads_or(tid < min(S.nlong, S.kLong) && S.longq[tid] != kStruck);
    if (more) merge_huge_segments<TH>(scratch, scratch_tokens, T, status);
  }
}

// ---- live tokens of the owned region, in order: out(off, ids, n) is called by every warp for each of its runs of 256
//      positions, `off` = live tokens in front of it, ids in shared memory.  The last warp notes the total in S.total.
//      kWoff: S.woff[w] = live tokens in front of word w. ----
template <int TH, bool kWoff, class Out>
__device__ __forceinline__ void tile_emit(TileSmem<TH>& S, int first, int end, uint16_t* woff, Out out)
{
  constexpr int NW = TileSmem<TH>::kWarps;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint8_t* cut8 = reinterpret_cast<const uint8_t*>(S.cut);
  uint16_t* ids       = S.region(warp);
  int off = 0;  // live tokens in front of this warp's positions
  for (int w = lane; w < warp * 16; w += 32) off += __popc(S.cut[w] & range_mask(w * 32, first, end));
  off = __reduce_add_sync(0xFFFFFFFFu, off);
  // two runs of 256 positions per warp; the halo is one more, of the last warp
  const int runs = warp < NW - 1 ? 2 : 3;
  for (int run = 0; run < runs; ++run) {
    const int p0 = warp * 512 + run * 256 + lane * 8;
    if (!kWoff && p0 - lane * 8 >= end) break;
    const uint32_t m = uint32_t(cut8[p0 >> 3]) & range_mask(p0, first, end) & 0xFFu;
    const int cnt    = __popc(m);
    int inc          = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += y;
    }
    int at = inc - cnt;
    if (kWoff && (lane & 3) == 0) woff[p0 >> 5] = uint16_t(off + at);
    const uint4 t8 = *reinterpret_cast<const uint4*>(&S.tok[p0]);
    const uint32_t t[4] = {t8.x, t8.y, t8.z, t8.w};
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if ((m >> b) & 1u) ids[at++] = uint16_t((b & 1) ? t[b >> 1] >> 16 : t[b >> 1]);
    const int n = __shfl_sync(0xFFFFFFFFu, inc, 31);
    __syncwarp();
    out(off, ids, n);
    off += n;
    __syncwarp();
  }
  if (warp == NW - 1 && lane == 0) S.total = off;
}

// ---- a segment that runs past the window (rare): the whole CTA merges it in an HBM workspace of scratch_tokens slots
//      per array; it ends at the first never-merge boundary behind the window, at the latest at cend.  Returns its
//      number of ids, at *ids. ----
template <int TH>
__device__ __noinline__ int merge_oversize(const uint8_t* bytes, int64_t start, int64_t window_end, int64_t cend,
                                           uint16_t* scratch, int64_t scratch_tokens, const DeviceTable& T, int* status)
{
  TileSmem<TH>& S = tile_smem<TH>();
  const int tid = threadIdx.x;
  if (tid == 0) S.over_end = cend;
  __syncthreads();
  int64_t ge = cend;
  for (int64_t pos = window_end; pos < cend; pos += TH) {
    const int64_t p = pos + tid;
    const bool cutp = (p < cend) && !adj_bit(T.adj, bytes[p - 1], bytes[p]);
    if (__syncthreads_or(cutp)) {
      if (cutp) atomicMin(reinterpret_cast<unsigned long long*>(&S.over_end), (unsigned long long)p);
      __syncthreads();
      ge = S.over_end;
      break;
    }
  }
  const int64_t L64 = ge - start;
  int len           = 0;
  if (L64 > scratch_tokens || scratch == nullptr) {
    if (tid == 0) atomicMax(status, int(kStatusScratchTooSmall));
  } else {
    const int L   = int(L64);
    uint16_t* wt  = scratch;
    uint16_t* wrk = scratch + scratch_tokens;
    for (int i = tid; i < L; i += TH) {
      const uint32_t cur = bytes[start + i];
      wt[i]  = __ldg(T.byte_to_id + cur);
      wrk[i] = (i + 1 < L) ? __ldg(T.byte_pair_rank + ((cur << 8) | bytes[start + i + 1])) : uint16_t(NONE);
    }
    __syncthreads();
    len = group_merge<TH / 32>(wt, wrk, L, T, S.gs(), status);
  }
  __syncthreads();
  return len;
}
