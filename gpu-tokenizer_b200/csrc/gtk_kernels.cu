// gtk_kernels.cu -- sm_100a kernels of the greedy byte-level BPE path.
//
//   merge (opt)  persistent CTAs walk the byte stream in tiles (gtk_tile.cuh); what starts where is kept in one
//                record per tile (replaces bpe_merge_kernel_optimized's role as the fast entry point,
//                gputok_binding.cu:704-846, with the greedy rule of gputok_blockbpe.cu:248-300, and the host
//                chunk/flatten loops, gputok_binding.cu:718-752)
//   pack         a tile's tokens to int32 ids at the tile's place, and the offsets of the chunks and texts that
//                start in it (replaces the padded D2H + host unflatten, gputok_binding.cu:807-836)
//   merge (base) one CTA per chunk on the same engine (replaces bpe_merge_kernel_blockbpe,
//                gputok_blockbpe.cu:328-538)
//   merge (wide) one CTA per chunk, pass by pass, for merge tables whose ids or ranks need more than
//                16 bits: 32-bit tokens and ranks, 16-byte-slot pair table
//   local-min    the reference's other rule (bpe_merge_kernel_optimized,
//                gputok_binding.cu:290-414), one CTA per chunk
//   small        chunker, tiles, scans and pack of a small batch in one
//                single-CTA launch (latency mode)
//   chunker, scans  of the kernels that work chunk by chunk: text lengths -> chunk offsets, chunk counts -> id offsets
//
// Nothing here is a dense contraction: the kernels are integer/byte work bound
// by latency and issue throughput, so there is no tensor-core code.
// Kernels report trouble through a status word and never trap; every loop is
// bounded.  -DGTK_CHECKED adds range checks on every data-dependent index.
#include "gtk_device.cuh"
#include "gtk_table.hpp"

#include <algorithm>
#include <cstddef>
#include <type_traits>

namespace gtk {
namespace {


// Checked build (-DGTK_CHECKED): every index into shared memory, the lane scratch, the staging buffer and the
// per-chunk / per-unit arrays that is computed from data is compared with its limit before it is used.  A
// violation is recorded (first failing check, offending value, limit, number of violations) and the access is
// skipped, so a wrong index shows up as a report, never as a fault; read the record with
// gtk_debug_check_words.  Without the flag the checks compile to nothing.
#ifdef GTK_CHECKED
__device__ int g_check_words[4];
__device__ __noinline__ bool check_failed(int id, long long value, long long limit)
{
  if (atomicAdd(&g_check_words[3], 1) == 0) {
    g_check_words[0] = id;
    g_check_words[1] = int(value);
    g_check_words[2] = int(limit);
  }
  return false;
}
#define GTK_IN(value, limit, id) \
  ((static_cast<unsigned long long>(value) < static_cast<unsigned long long>(limit)) || check_failed((id), (long long)(value), (long long)(limit)))
#else
#define GTK_IN(value, limit, id) true
#endif

constexpr uint32_t NONE = 0xFFFFu;  // pair not mergeable
constexpr uint32_t SEL  = 0xFFFEu;  // pair selected for the current pass
constexpr uint32_t DEAD = 0xFFFFu;  // token slot holds nothing

// ------------------------------------------------------------------------------------------------
// merge table probes
// ------------------------------------------------------------------------------------------------

// What a probe of the pair table needs, small enough to travel in registers.
struct PairTable {
  const uint4* buckets;
  const uint2* overflow;           // nullptr when no bucket overflowed
  const uint32_t* merged_of_rank;  // nullptr when merged id = 256 + rank
  uint32_t overflow_mask;
};

__device__ __forceinline__ PairTable pair_table(const DeviceTable& T)
{
  return PairTable{T.pair_buckets, T.pair_overflow, T.merged_is_256_plus_rank ? nullptr : T.merged_of_rank,
                   T.pair_overflow_mask};
}

// keys of a full bucket that has no match may live in the overflow table
__device__ __noinline__ uint32_t probe_overflow(const uint2* overflow, uint32_t mask, uint32_t key)
{
  uint32_t h = ((key * 0x85EBCA77u) >> 7) & mask;
  for (uint32_t d = 0; d <= mask; ++d) {
    const uint2 s = __ldg(overflow + h);
    if (s.x == key) return s.y;
    if (s.x == 0xFFFFFFFFu) return NONE;
    h = (h + 1u) & mask;
  }
  return NONE;
}

// Rank of the key whose hash is h in its home bucket v.  An entry is low16(h) << 16 | rank, so XOR with
// low16(h) << 16 leaves the bare rank (< 65536) for the key's own entry and something larger for every other
// entry: the minimum over the four words is the rank, or a value >= 65536 when the key is not there (an empty
// word can only "match" with rank 0xFFFF, which is the right answer for a bucket that is not full).
__device__ __forceinline__ uint32_t bucket_rank(const uint4& v, uint32_t h)
{
  const uint32_t f = h << 16;
  return min(min(v.x ^ f, v.y ^ f), min(v.z ^ f, v.w ^ f));
}

// any value >= SEL means "no such merge"
__device__ __forceinline__ uint32_t resolve_rank_raw(const uint4& v, uint32_t key, const uint2* overflow,
                                                     uint32_t mask)
{
  uint32_t r = bucket_rank(v, key * 0x9E3779B1u);
  if (r >= SEL && overflow != nullptr && v.w != 0xFFFFFFFFu) r = probe_overflow(overflow, mask, key);
  return r;
}

__device__ __forceinline__ uint32_t resolve_rank(const uint4& v, uint32_t key, const uint2* overflow, uint32_t mask)
{
  return min(resolve_rank_raw(v, key, overflow, mask), NONE);
}

__device__ __forceinline__ uint32_t probe_rank(const DeviceTable& T, uint32_t left, uint32_t right)
{
  const uint32_t key = (left << 16) | right;
  const uint4 v      = __ldg(T.pair_buckets + ((key * 0x9E3779B1u) >> 16));
  return resolve_rank(v, key, T.pair_overflow, T.pair_overflow_mask);
}

// Tables whose ids or ranks do not fit 16 bits are served from the 16-byte-slot open-addressing table
// ({right, left, rank, merged id}, linear probing, empty = all ones): rank of the pair, 0xFFFFFFFF if none.
__device__ __forceinline__ uint32_t probe_rank_wide(const DeviceTable& T, uint32_t left, uint32_t right)
{
  const uint32_t mask = (1u << T.wide_log2) - 1u;
  uint32_t h = (((left << 16) ^ right) * 0x9E3779B1u) >> (32u - T.wide_log2);
  for (uint32_t d = 0; d <= T.wide_max_probe; ++d) {
    const uint4 v = __ldg(T.wide_slots + h);
    if (v.x == right && v.y == left) return v.z;
    if ((v.x & v.y) == 0xFFFFFFFFu) return 0xFFFFFFFFu;
    h = (h + 1u) & mask;
  }
  return 0xFFFFFFFFu;
}

// rank of a pair in the marker convention of the element type (16-bit: 0xFFFF = none, 32-bit: all ones = none)
template <typename TT>
__device__ __forceinline__ uint32_t probe_rank_t(const DeviceTable& T, uint32_t left, uint32_t right)
{
  if (sizeof(TT) == 2) return probe_rank(T, left, right);
  return probe_rank_wide(T, left, right);
}

__device__ __forceinline__ uint32_t merged_id(const DeviceTable& T, uint32_t rank)
{
  return T.merged_is_256_plus_rank ? 256u + rank : __ldg(T.merged_of_rank + rank);
}

// may bytes u, v end up in one token (the matrix is laid out as [v / 32][u], bit v % 32)
__device__ __forceinline__ bool adj_bit(const uint32_t* adj, uint32_t u, uint32_t v)
{
  return (__ldg(adj + (((v >> 5) << 8) | u)) >> (v & 31u)) & 1u;
}

__device__ __forceinline__ unsigned long long global_timer()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t lanemask_lt()
{
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ------------------------------------------------------------------------------------------------
// The NW warps of a CTA merge one sequence pass by pass.  tok/rk may point to
// shared memory or to an HBM workspace.
//
// Slots: tok[i] is a token id or the DEAD tombstone; for a live slot rk[i] is the
// cached rank of the pair (tok[i], next live token), NONE when there is none; a
// dead slot has rk NONE.  Tombstones stay where they are and the slots are
// compacted only when an eighth of them is dead, so a pass costs two sweeps over
// the cached ranks plus work proportional to the number of merges:
//   (1) minimum of the cached ranks (four ranks per 64-bit load, rk is 8-byte
//       aligned; warp redux + cross-warp exchange);
//   (2) selection of the occurrences of that pair;
//   (3) every selected occurrence writes the merged id and a tombstone and
//       remembers its slot;
//   (4) the two pairs next to every new token are probed again (only those);
//   (5) in-place compaction when due -- each thread keeps its elements in
//       registers between the read and the write, offsets come from warp ballots
//       and popc plus a cross-warp sum.
//
// With a monotone table all non-overlapping occurrences of the winning pair,
// taken left to right, are merged in one pass; this is what Algorithm 1 does
// over consecutive passes because no merge at the minimum rank can expose a
// lower rank.  Otherwise only the left-most occurrence is merged.
// ------------------------------------------------------------------------------------------------
constexpr int kMergeList = 64;  // merges of one pass that are re-probed from a list; more fall back to a sweep
struct GroupScratch {
  uint32_t red[2][32];
  uint32_t wsum[32];
  int dead;  // tombstones since the last compaction
  int list[kMergeList];  // slots merged in the current pass
};

template <int NW>
__device__ __forceinline__ void gsync()
{
  if (NW == 1) __syncwarp();
  else __syncthreads();
}

template <int NW>
__device__ __forceinline__ uint32_t group_min(uint32_t v, GroupScratch* gs, int& parity, int lane, int warp)
{
  v = __reduce_min_sync(0xFFFFFFFFu, v);
  if (NW > 1) {
    if (lane == 0) gs->red[parity][warp] = v;
    __syncthreads();
    uint32_t x = (lane < NW) ? gs->red[parity][lane] : 0xFFFFFFFFu;
    v          = __reduce_min_sync(0xFFFFFFFFu, x);
    parity ^= 1;
  }
  return v;
}

// first live slot after i (n when there is none) / before i (-1 when there is none)
__device__ __forceinline__ int next_live(const uint16_t* tok, int i, int n)
{
  int j = i + 1;
  while (j < n && tok[j] == DEAD) ++j;
  return j;
}
__device__ __forceinline__ int prev_live(const uint16_t* tok, int i)
{
  int p = i - 1;
  while (p >= 0 && tok[p] == DEAD) --p;
  return p;
}

// Sweeps read the cached ranks four at a time (one 64-bit load) and reduce them with the packed 16-bit
// three-input minimum; the up to three slots between n and the next multiple of four hold NONE (pad_ranks).
__device__ __forceinline__ void pad_ranks(uint16_t* rk, int n, int tid)
{
  if (tid < ((4 - (n & 3)) & 3)) rk[n + tid] = uint16_t(NONE);
}

// calls f(i) for every slot i < n whose cached rank equals `pick`
template <int NW, class F>
__device__ __forceinline__ void for_each_rank(const uint16_t* rk, int n, int tid, uint32_t pick, F f)
{
  const int nw      = (n + 3) >> 2;
  const uint32_t p2 = pick | (pick << 16);
  for (int w = tid; w < nw; w += NW * 32) {
    const uint2 x = reinterpret_cast<const uint2*>(rk)[w];
    // a half-word of z is zero exactly when one of the four ranks equals pick
    const uint32_t z = __vimin3_u16x2(x.x ^ p2, x.y ^ p2, 0xFFFFFFFFu);
    if ((z & 0xFFFFu) == 0u || (z >> 16) == 0u) {
      const uint32_t q[4] = {x.x & 0xFFFFu, x.x >> 16, x.y & 0xFFFFu, x.y >> 16};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (q[k] == pick) f(4 * w + k);
    }
  }
}

// In-place compaction of tok/rk[0..n): returns the number of live slots, which end up at the front in order.
template <int NW>
__device__ __forceinline__ int group_compact(uint16_t* tok, uint16_t* rk, int n, GroupScratch* gs, int lane, int warp,
                                             uint32_t lt)
{
  constexpr int G = NW * 32;
  constexpr int E = 4;
  int out = 0;
  for (int base = 0; base < n; base += G * E) {
    uint16_t t[E], q[E];
    uint32_t bal[E];
    int wt = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int i  = base + warp * 32 * E + k * 32 + lane;
      const bool v = i < n;
      t[k]   = v ? tok[i] : uint16_t(DEAD);
      q[k]   = v ? rk[i] : uint16_t(NONE);
      bal[k] = __ballot_sync(0xFFFFFFFFu, t[k] != DEAD);
      wt += __popc(bal[k]);
    }
    if (lane == 0) gs->wsum[warp] = uint32_t(wt);
    __syncthreads();  // all loads of the batch are done, warp totals visible
    int pre = 0, tot = 0;
    for (int w = 0; w < NW; ++w) {
      const int x = int(gs->wsum[w]);
      if (w < warp) pre += x;
      tot += x;
    }
    int o = out + pre;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      if (t[k] != DEAD) {
        const int d = o + __popc(bal[k] & lt);
        tok[d] = t[k];
        rk[d]  = q[k];
      }
      o += __popc(bal[k]);
    }
    out += tot;
    __syncthreads();
  }
  return out;
}

template <int NW>
__device__ int group_merge(uint16_t* tok, uint16_t* rk, int L, const DeviceTable& T, GroupScratch* gs,
                           int* status)
{
  constexpr int G = NW * 32;
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = lanemask_lt();
  const bool batch  = T.monotone != 0;
  int parity = 0;
  int n      = L;  // slots in use
  int dead   = 0;  // tombstones among them
  pad_ranks(rk, n, tid);
  if (tid == 0) gs->dead = 0;
  __syncthreads();
  for (int pass = 0; pass < L && n - dead >= 2; ++pass) {
    // (1) lowest cached rank
    uint32_t m2 = 0xFFFFFFFFu;
    for (int w = tid; w < (n + 3) >> 2; w += G) {
      const uint2 x = reinterpret_cast<const uint2*>(rk)[w];
      m2 = __vimin3_u16x2(m2, x.x, x.y);
    }
    const uint32_t r = group_min<NW>(min(m2 & 0xFFFFu, m2 >> 16), gs, parity, lane, warp);
    if (r >= SEL) break;
    const uint32_t c = merged_id(T, r);
    const bool same  = batch && (__ldg(T.same_of_rank + r) != 0);
    // (2) selection
    if (!batch) {
      uint32_t p = 0xFFFFFFFFu;
      for_each_rank<NW>(rk, n, tid, r, [&](int i) { p = min(p, uint32_t(i)); });
      p = group_min<NW>(p, gs, parity, lane, warp);
      __syncthreads();
      if (tid == 0) rk[p] = uint16_t(SEL);
      __syncthreads();
    } else if (same) {
      // occurrences of (a,a) overlap inside a run a a a ...; left to right
      // selection keeps the even offsets of every maximal run of matches
      for_each_rank<NW>(rk, n, tid, r, [&](int i) {
        const int pl = prev_live(tok, i);
        if (pl >= 0) {
          const uint32_t pv = rk[pl];
          if (pv == r || pv == SEL) return;  // not the first match of its run
        }
        int j = i;
        for (;;) {
          rk[j] = uint16_t(SEL);
          const int j1 = next_live(tok, j, n);
          if (j1 >= n || rk[j1] != r) break;
          const int j2 = next_live(tok, j1, n);
          if (j2 >= n || rk[j2] != r) break;
          j = j2;
        }
      });
      __syncthreads();
    }
    const uint32_t pick = (!batch || same) ? SEL : r;
    // (3) apply: the selected occurrences never share a slot, so the writes are disjoint.  The merged slots are
    // collected in a list; the tombstone counter hands out the places
    for_each_rank<NW>(rk, n, tid, pick, [&](int i) {
      const int j = next_live(tok, i, n);  // exists: the pair has a cached rank
      if (!GTK_IN(i, n, 30)) return;
      tok[i] = uint16_t(c);
      rk[i]  = uint16_t(NONE);
      if (j < n) {
        tok[j] = uint16_t(DEAD);
        rk[j]  = uint16_t(NONE);
      }
      const int place = atomicAdd(&gs->dead, 1) - dead;
      if (place < kMergeList) gs->list[place] = i;
    });
    // (4) ranks of the two pairs next to every new token
    auto refresh = [&](int i) {
      const int jn = next_live(tok, i, n);
      rk[i] = uint16_t((jn < n) ? probe_rank(T, c, tok[jn]) : NONE);
      const int pl = prev_live(tok, i);
      if (pl >= 0) rk[pl] = uint16_t(probe_rank(T, tok[pl], c));
    };
    __syncthreads();
    const int now = gs->dead;
    if (now == dead) {  // a pass must remove at least one token
      if (tid == 0 && status) atomicMax(status, int(kStatusBadSegment));
      break;
    }
    const int merged = now - dead;
    dead = now;
    if (merged <= kMergeList) {  // the first threads take one merged slot each: one or two warps do the probes
      if (tid < merged) refresh(gs->list[tid]);
    } else {
      for (int i = tid; i < n; i += G)
        if (tok[i] == c) refresh(i);
    }
    __syncthreads();
    // (5) compaction when an eighth of the slots is dead
    if (dead * 8 >= n) {
      n    = group_compact<NW>(tok, rk, n, gs, lane, warp, lt);
      dead = 0;
      pad_ranks(rk, n, tid);
      if (tid == 0) gs->dead = 0;
      __syncthreads();
    }
  }
  if (dead) n = group_compact<NW>(tok, rk, n, gs, lane, warp, lt);
  return n;
}

// The same merge with a compaction in every pass: cheaper for the short sequences a single warp handles
// inside a tile (a few dozen to a few hundred tokens), where a sweep costs little and the tombstone searches of
// the lazy variant do not pay.
template <int NW, typename TT>
__device__ int group_merge_dense(TT* tok, TT* rk, int L, const DeviceTable& T, GroupScratch* gs,
                           int* status)
{
  constexpr int G = NW * 32;
  constexpr int E = 4;
  // markers in the element type: all ones = no rank / tombstone, all ones minus one = selected
  constexpr uint32_t kNone = uint32_t(TT(~TT(0))), kSel = kNone - 1u, kDead = kNone;
  const int lane  = threadIdx.x & 31;
  const int warp  = (NW == 1) ? 0 : (threadIdx.x >> 5);
  const int tid   = (NW == 1) ? lane : int(threadIdx.x);
  const uint32_t lt = lanemask_lt();
  int parity = 0;
  int len    = L;
  for (int pass = 0; pass < L && len >= 2; ++pass) {
    // (1) lowest cached rank
    uint32_t m = kNone;
    for (int i = tid; i < len - 1; i += G) m = min(m, uint32_t(rk[i]));
    m = group_min<NW>(m, gs, parity, lane, warp);
    if (m >= kSel) break;
    const uint32_t r = m;
    const uint32_t c = merged_id(T, r);
    const bool batch = T.monotone != 0;
    const bool same  = batch && (__ldg(T.same_of_rank + r) != 0);
    // (2) selection
    if (!batch) {
      uint32_t p = 0xFFFFFFFFu;
      for (int i = tid; i < len - 1; i += G)
        if (rk[i] == r) { p = uint32_t(i); break; }
      p = group_min<NW>(p, gs, parity, lane, warp);
      gsync<NW>();
      if (tid == 0) rk[p] = TT(kSel);
      gsync<NW>();
    } else if (same && NW == 1) {
      // occurrences of (a,a) overlap inside a run a a a ...; left to right selection keeps the even offsets of
      // every maximal run of matches.  One warp, 32 slots per round: a ballot gives the matches, the distance of a
      // match to the start of its run is the distance to the nearest non-match below it (the run may reach back
      // into earlier rounds: `before` carries the parity of the matches that directly precede this round)
      uint32_t before = 0;
      for (int base = 0; base < len - 1; base += 32) {
        const int i       = base + lane;
        const bool match  = (i < len - 1) && (rk[i] == r);
        const uint32_t mm = __ballot_sync(0xFFFFFFFFu, match);
        if (match) {
          const uint32_t gaps = ~mm & lt;  // non-matches below this lane
          const uint32_t off  = gaps ? uint32_t(lane) - (32u - uint32_t(__clz(int(gaps)))) : uint32_t(lane) + before;
          if ((off & 1u) == 0u) rk[i] = TT(kSel);
        }
        const uint32_t tail = uint32_t(__clz(int(~mm)));  // matches at the top of this round
        before = (tail == 32u) ? ((before + 32u) & 1u) : (tail & 1u);
      }
      __syncwarp();
    } else if (same) {
      // the same selection for a CTA-wide group: the first match of every run walks its run
      for (int i = tid; i < len - 1; i += G) {
        if (rk[i] != r) continue;
        if (i > 0) {
          const uint32_t pv = rk[i - 1];
          if (pv == r || pv == kSel) continue;  // not the first match of its run
        }
        int j = i;
        for (;;) {
          rk[j] = TT(kSel);
          if (j + 2 < len - 1 && rk[j + 1] == r && rk[j + 2] == r) j += 2;
          else break;
        }
      }
      gsync<NW>();
    }
    const uint32_t pick = (!batch || same) ? kSel : r;
    // (3) apply
    for (int i = tid; i < len - 1; i += G) {
      if (rk[i] == pick) {
        tok[i]     = TT(c);
        tok[i + 1] = TT(kDead);
      }
    }
    gsync<NW>();
    // (4) in-place compaction, batch by batch, registers as the second buffer
    int out = 0;
    for (int base = 0; base < len; base += G * E) {
      TT t[E], q[E];
      uint32_t bal[E];
      int wt = 0;
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const int i = base + warp * 32 * E + k * 32 + lane;
        const bool v = i < len;
        t[k]   = v ? tok[i] : TT(kDead);
        q[k]   = v ? rk[i] : TT(kNone);
        bal[k] = __ballot_sync(0xFFFFFFFFu, t[k] != kDead);
        wt += __popc(bal[k]);
      }
      int pre = 0, tot = wt;
      if (NW > 1) {
        if (lane == 0) gs->wsum[warp] = uint32_t(wt);
        __syncthreads();  // all loads of the batch are done, warp totals visible
        tot = 0;
        for (int w = 0; w < NW; ++w) {
          const int x = int(gs->wsum[w]);
          if (w < warp) pre += x;
          tot += x;
        }
      } else {
        __syncwarp();
      }
      int o = out + pre;
#pragma unroll
      for (int k = 0; k < E; ++k) {
        if (t[k] != kDead) {
          const int d = o + __popc(bal[k] & lt);
          tok[d] = t[k];
          rk[d]  = q[k];
        }
        o += __popc(bal[k]);
      }
      out += tot;
      gsync<NW>();
    }
    if (!GTK_IN(out, L + 1, 29)) break;
    if (out >= len) {  // a pass must remove at least one token
      if (tid == 0 && status) atomicMax(status, int(kStatusBadSegment));
      break;
    }
    len = out;
    // (5) refresh ranks next to new tokens
    for (int d = tid; d < len; d += G) {
      if (tok[d] == c) {
        rk[d] = TT((d + 1 < len) ? probe_rank_t<TT>(T, c, tok[d + 1]) : kNone);
        if (d > 0) rk[d - 1] = TT(probe_rank_t<TT>(T, tok[d - 1], c));
      }
    }
    gsync<NW>();
  }
  return len;
}

// ------------------------------------------------------------------------------------------------
// block-wide helpers
// ------------------------------------------------------------------------------------------------

// exclusive scan of one int per thread over the CTA; *total receives the sum.
// `buf` must hold 33 ints of shared memory; contains two barriers.
__device__ __forceinline__ int block_exclusive_scan(int v, int* buf, int* total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
    if (lane >= d) inc += y;
  }
  if (lane == 31) buf[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < nw) ? buf[lane] : 0;
    int winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, winc, d);
      if (lane >= d) winc += y;
    }
    buf[lane] = winc - w;
    if (lane == 31) buf[32] = winc;
  }
  __syncthreads();
  *total = buf[32];
  return buf[warp] + inc - v;
}

// ------------------------------------------------------------------------------------------------
// multi-block exclusive scan: counts (int32 array, or chunks-per-text computed
// on the fly) -> int64 offsets[n+1].  Three kernels: per-block sums, scan of
// the block sums by one CTA, final pass.  n may live on the device.
// ------------------------------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems   = 16;
constexpr int kScanBlock   = kScanThreads * kScanItems;

struct CountsI32 {
  const int32_t* p;
  __device__ int64_t operator()(int64_t i) const { return p[i]; }
};
struct ChunksPerText {
  const int64_t* off;
  int chunk;
  __device__ int64_t operator()(int64_t i) const
  {
    const int64_t len = off[i + 1] - off[i];
    if (len <= 0) return 0;
    if (len < (int64_t(1) << 31)) return int64_t((uint32_t(len) + uint32_t(chunk) - 1u) / uint32_t(chunk));  // the usual case, a 32-bit division
    return (len + chunk - 1) / chunk;
  }
};

__device__ __forceinline__ int64_t block_sum_i64(int64_t v, int64_t* buf)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  int64_t s = 0;
  for (int w = 0; w < kScanThreads / 32; ++w) s += buf[w];
  __syncthreads();
  return s;
}

template <class In>
__global__ void __launch_bounds__(kScanThreads) k_scan_partial(In in, int64_t n_imm, const int64_t* n_ptr,
                                                               int64_t* block_sums)
{
  __shared__ int64_t buf[kScanThreads / 32];
  const int64_t n    = n_ptr ? *n_ptr : n_imm;
  const int64_t base = int64_t(blockIdx.x) * kScanBlock;
  int64_t s          = 0;
  for (int e = 0; e < kScanItems; ++e) {
    const int64_t i = base + int64_t(e) * kScanThreads + threadIdx.x;
    if (i < n) s += in(i);
  }
  s = block_sum_i64(s, buf);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = s;
}

// one CTA: exclusive scan of block_sums[0..nb) in place
__global__ void __launch_bounds__(kScanThreads) k_scan_block_sums(int64_t* block_sums, int64_t nb)
{
  __shared__ int64_t wtot[kScanThreads / 32];
  __shared__ int64_t carry_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += kScanThreads) {
    const int64_t i = base + threadIdx.x;
    const int64_t v = (i < nb) ? block_sums[i] : 0;
    int64_t inc     = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int64_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += y;
    }
    if (lane == 31) wtot[warp] = inc;
    __syncthreads();
    int64_t pre = carry_s;
    for (int w = 0; w < warp; ++w) pre += wtot[w];
    if (i < nb) block_sums[i] = pre + inc - v;
    __syncthreads();
    if (threadIdx.x == kScanThreads - 1) carry_s = pre + inc;
    __syncthreads();
  }
}

template <class In>
__global__ void __launch_bounds__(kScanThreads) k_scan_final(In in, int64_t n_imm, const int64_t* n_ptr,
                                                             const int64_t* block_sums, int64_t* out,
                                                             int64_t* total_out)
{
  __shared__ int64_t wtot[kScanThreads / 32];
  const int64_t n = n_ptr ? *n_ptr : n_imm;
  if (n == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      out[0] = 0;
      if (total_out) *total_out = 0;
    }
    return;
  }
  const int64_t base = int64_t(blockIdx.x) * kScanBlock;
  if (base >= n) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // blocked layout: thread t owns items base + t*kScanItems .. +kScanItems
  int64_t v[kScanItems];
  int64_t s = 0;
  const int64_t first = base + int64_t(threadIdx.x) * kScanItems;
#pragma unroll
  for (int e = 0; e < kScanItems; ++e) {
    const int64_t i = first + e;
    v[e] = (i < n) ? in(i) : 0;
    s += v[e];
  }
  int64_t inc = s;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int64_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
    if (lane >= d) inc += y;
  }
  if (lane == 31) wtot[warp] = inc;
  __syncthreads();
  int64_t pre = block_sums[blockIdx.x];
  for (int w = 0; w < warp; ++w) pre += wtot[w];
  int64_t run = pre + inc - s;
#pragma unroll
  for (int e = 0; e < kScanItems; ++e) {
    const int64_t i = first + e;
    if (i < n) {
      out[i] = run;
      run += v[e];
      if (i == n - 1) {
        out[n] = run;
        if (total_out) *total_out = run;
      }
    }
  }
}

template <class In>
int run_scan(In in, int64_t n_upper, int64_t n_imm, const int64_t* n_ptr, int64_t* block_sums, int64_t* out,
             int64_t* total_out, cudaStream_t stream)
{
  int64_t nb = (n_upper + kScanBlock - 1) / kScanBlock;
  if (nb < 1) nb = 1;
  k_scan_partial<In><<<unsigned(nb), kScanThreads, 0, stream>>>(in, n_imm, n_ptr, block_sums);
  k_scan_block_sums<<<1, kScanThreads, 0, stream>>>(block_sums, nb);
  k_scan_final<In><<<unsigned(nb), kScanThreads, 0, stream>>>(in, n_imm, n_ptr, block_sums, out, total_out);
  return 3;
}

// ------------------------------------------------------------------------------------------------
// chunker
// ------------------------------------------------------------------------------------------------

// chunk c -> owning text by binary search over the scanned chunk counts, then
// its start byte.  Empty texts own no chunk and are skipped by the search.
__global__ void k_chunk_fill(const int64_t* __restrict__ text_off, const int64_t* __restrict__ text_chunk_base,
                             int64_t n_texts, int chunk_bytes, int64_t* __restrict__ chunk_off)
{
  const int64_t C = text_chunk_base[n_texts];
  for (int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; c <= C; c += int64_t(gridDim.x) * blockDim.x) {
    if (c == C) {
      chunk_off[c] = text_off[n_texts];
      continue;
    }
    int64_t lo = 0, hi = n_texts;  // last t with text_chunk_base[t] <= c
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (text_chunk_base[mid] <= c) lo = mid; else hi = mid;
    }
    chunk_off[c] = text_off[lo] + (c - text_chunk_base[lo]) * int64_t(chunk_bytes);
  }
}

// ------------------------------------------------------------------------------------------------
// merge kernel, segment-parallel ("opt")
// ------------------------------------------------------------------------------------------------

#include "gtk_tile.cuh"

// Window k of a batch walked in tiles of kTile bytes: n_tiles that hold text, `tail` bytes of it in the last of them.
__device__ __forceinline__ Span batch_span(const EncodeBuffers& b, int k, int n_tiles, int tail)
{
  const int rest = min(n_tiles - 1 - k, 2) * kTile + tail;  // as far as it matters
  return Span{b.bytes, int64_t(k) * kTile, 0, min(kTile, rest), min(kWindow, rest), k > 0, k == 0};
}

// Where the texts of a batch end.  A caller's device buffer may be longer than they are.
__device__ __forceinline__ int64_t text_end(const EncodeBuffers& b)
{
  return b.text_end ? max(min(__ldg(reinterpret_cast<const long long*>(b.text_end)), (long long)b.n_bytes), 0ll) : b.n_bytes;
}

// first index in [0, n) whose value is not below x, n if there is none; one warp, 32 places per step
__device__ __forceinline__ int64_t warp_lower_bound(const int64_t* v, int64_t n, int64_t x)
{
  const int lane = threadIdx.x & 31;
  int64_t lo = 0, hi = n;  // the answer is in [lo, hi]
  while (hi > lo) {
    const int64_t step = (hi - lo + 31) >> 5, i = lo + (lane + 1) * step - 1;
    const int below    = __popc(__ballot_sync(0xFFFFFFFFu, i < hi && v[i] < x));
    lo += below * step;
    hi = min(hi, lo + step - 1);
  }
  return min(lo, n);
}

// The tile records: one thread per tile.  The tile kernel would pay for the search and the divisions in every warp of every
// tile (128 MiB: 710 us instead of 590).
__global__ void __launch_bounds__(128) k_tile_info(EncodeBuffers b)
{
  const int64_t chunk = b.chunk_bytes, n_end = text_end(b);
  for (int64_t k = int64_t(blockIdx.x) * 128 + threadIdx.x; k < b.n_tiles; k += int64_t(gridDim.x) * 128) {
    const int64_t lo = k * kTile;
    TileInfo i{0, 0, kTileNoCut, 0};
    if (lo >= n_end) {  // the tile kernel leaves it out
      b.unit_first[k] = lo;
      b.unit_cnt[k]   = 0;
    }
    if (b.n_texts == 1) {
      i.t0    = lo > 0;
      i.c0    = (min(lo, n_end) + chunk - 1) / chunk;
      i.flags = kTilePlain | (lo > 0 ? kTileRunsIn : 0);
      const int64_t p0 = i.c0 * chunk - lo;
      if (p0 < kWindow && lo + p0 < n_end) i.p0 = int(p0);
    } else {
      int64_t a = 0, e = b.n_texts;  // first text that starts at or behind the tile's first byte
      while (a < e) {
        const int64_t mid = (a + e) >> 1;
        if (b.text_off[mid] < lo) a = mid + 1; else e = mid;
      }
      const int64_t end = b.text_off[a];
      i.t0 = a;
      i.c0 = b.text_chunk_base[a];
      if (a > 0 && end > lo) {
        const int64_t s = b.text_off[a - 1], d = lo - s;
        const int64_t n = d < (int64_t(1) << 31) ? int64_t((uint32_t(d) + uint32_t(chunk) - 1u) / uint32_t(chunk)) : (d + chunk - 1) / chunk;
        const int64_t at = s + n * chunk;
        i.flags = kTileRunsIn | (end >= min(lo + kWindow, n_end) ? kTilePlain : 0);
        if (at < end) {
          i.c0 = b.text_chunk_base[a - 1] + n;
          if (at - lo < kWindow) i.p0 = int(at - lo);
        }
      }
    }
    b.tile_info[k] = i;
  }
}

// Calls f(position, chunk number or -1, text number or -1) for everything that starts in window positions [0, limit): chunks
// and texts (an empty text and the chunk behind it start at the same position, in calls of their own; the start of a batch's
// only text is not reported).  The lanes of the calling warps share the texts between them, and the boundaries inside a text
// that has more than a few in the window; `first`, `stride`: the calling warp's number and how many there are.
template <class F>
__device__ __forceinline__ void for_each_start(const EncodeBuffers& b, const TileInfo& ti, int64_t lo, int limit, int first,
                                               int stride, F f)
{
  const int lane = threadIdx.x & 31;
  const int step = min(b.chunk_bytes, 2 * kWindow);  // a longer one leaves the window just the same
  if (ti.flags & kTilePlain) {
    for (int i = first * 32 + lane; ti.p0 + i * step < limit; i += stride * 32) f(ti.p0 + i * step, ti.c0 + i, int64_t(-1));
    return;
  }
  const int64_t t_lo = ti.t0 - ((ti.flags & kTileRunsIn) ? 1 : 0);
  for (int64_t q0 = int64_t(first) * 32;; q0 += int64_t(stride) * 32) {
    const int64_t t = t_lo + q0 + lane;
    int at = kTileNoCut, end = 0;  // first boundary inside the text, where the text ends
    int64_t c = 0;
    bool more = false;
    if (t < b.n_texts) {
      const int64_t s = b.text_off[t];
      more            = s < lo + limit;
      if (more) {
        const int64_t e = b.text_off[t + 1];
        end = int(min(e - lo, int64_t(limit)));
        if (s >= lo) {
          c = b.text_chunk_base[t];
          f(int(s - lo), e > s ? c : int64_t(-1), t);
          at = int(s - lo) + step;
          ++c;
        } else {  // the text that runs in
          at = ti.p0;
          c  = ti.c0;
        }
      }
    }
    const bool many = at + 4 * step < end;
    if (!many)
      for (int p = at; p < end; p += step) f(p, c++, int64_t(-1));
    for (uint32_t m = __ballot_sync(0xFFFFFFFFu, many); m; m &= m - 1) {
      const int src    = __ffs(int(m)) - 1;
      const int a0     = __shfl_sync(0xFFFFFFFFu, at, src), e0 = __shfl_sync(0xFFFFFFFFu, end, src);
      const int64_t c0 = __shfl_sync(0xFFFFFFFFu, c, src);
      for (int k = lane; a0 + k * step < e0; k += 32) f(a0 + k * step, c0 + k, int64_t(-1));
    }
    if (!__all_sync(0xFFFFFFFFu, more)) break;
  }
}

// One tile of a batch: tokenises every segment that starts in bytes [k*kTile, (k+1)*kTile), writes the tokens compacted to
// staging and what the pack kernel needs to know of the tile: number of ids, first chunk and text, and how many of its ids
// stand in front of every chunk and text that starts in it.
__device__ __forceinline__ void opt_tile(TileSmem<kOptThreads>& S, const EncodeBuffers& b, const DeviceTable& T, int k)
{
  __shared__ uint16_t woff[TileSmem<kOptThreads>::kWords];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* status   = b.counters + 1;
  const Span sp = batch_span(b, k, S.n_tiles, S.tail);
  const TileInfo ti = b.tile_info[k];
  tile_cut(S, sp, T, [&](auto mark) { for_each_start(b, ti, sp.lo, sp.wlen, 0, 1, [&](int p, int64_t, int64_t) { mark(p); }); });
  tile_lookup(S, sp, T, status);
  const int first = S.first;
  const int end   = (S.over_start >= 0) ? S.over_start : S.end;
  uint16_t* ws    = b.seg_scratch ? b.seg_scratch + int64_t(blockIdx.x) * 2 * b.seg_scratch_tokens : nullptr;
  tile_merge(S, T, ws, b.seg_scratch_tokens, status);
  const int64_t region_start = sp.lo + min(first, sp.wlen);
  tile_emit<kOptThreads, true>(S, first, end, woff, [&](int off, const uint16_t* ids, int n) {
    uint16_t* dst = b.staging + region_start + off;
    for (int j = lane; j < n; j += 32)
      if (GTK_IN(region_start + off + j, b.n_bytes, 22)) dst[j] = ids[j];
  });
  __syncthreads();
  const int total = S.total;
  if (S.no_space && tid == 0) atomicMax(status, int(kStatusScratchTooSmall));
  // ids of the tile in front of every chunk and text that starts in it (a chunk start is a segment start, so it lies inside
  // the owned region, or is the start of the oversize segment right behind it)
  for_each_start(b, ti, sp.lo, sp.own_hi, warp, kOptThreads / 32, [&](int p, int64_t c, int64_t t) {
    const int rel = woff[p >> 5] + __popc(S.cut[p >> 5] & range_mask(p & ~31, first, end) & ((1u << (p & 31)) - 1u));
    if (c >= 0 && GTK_IN(c, b.chunk_cap, 24)) b.chunk_rel[c] = rel;
    if (t >= 0 && GTK_IN(t, b.n_texts, 25)) b.text_rel[t] = rel;
  });
  int over = 0;
  if (S.over_start >= 0) {  // CTA-uniform, rare
    const int64_t start = sp.lo + S.over_start;
    const int64_t t     = b.n_texts == 1 ? 0 : warp_lower_bound(b.text_off, b.n_texts, start + 1) - 1;  // text that holds it
    const int64_t s     = b.n_texts == 1 ? 0 : b.text_off[t], e = b.n_texts == 1 ? int64_t(S.n_tiles - 1) * kTile + S.tail : b.text_off[t + 1];
    const int64_t cend  = min(e, s + ((start - s) / b.chunk_bytes + 1) * b.chunk_bytes);
    over = merge_oversize<kOptThreads>(b.bytes, start, sp.lo + kWindow, cend, ws, b.seg_scratch_tokens, T, status);
    for (int j = tid; j < over; j += kOptThreads)
      if (GTK_IN(region_start + total + j, b.n_bytes, 26)) b.staging[region_start + total + j] = ws[j];
  }
  if (tid == 0) {
    b.unit_first[k] = region_start;
    b.unit_cnt[k]   = total + over;
    atomicAdd(b.group_cnt + k / kTileGroup, total + over);
  }
}

// Bound by latency and issue together (see gtk_tile.cuh): about 60 % of the issue slots, DRAM 3 %.  This kernel alone, 128 MiB
// in 4 KiB chunks: English-like text 1027 us with five table loads and full token and rank arrays per position and no
// reuse of merged segments within the batch, 565 us now; the sample novel 941 -> 490 us; 64 MiB with multi-byte words and runs
// 750 -> 500 us.  Six CTAs per SM with 40 registers: 16 MiB of English-like text 147 us per call, 128 MiB 657; seven with 36
// registers 163 and 657, five with 48 registers 153 and 708 (128 MiB with runs 1050 / 1073 / 1088).  CTAs of 128 threads: the same.
#ifndef GTK_OPT_CTAS
#define GTK_OPT_CTAS 6
#endif
__global__ void __launch_bounds__(kOptThreads, GTK_OPT_CTAS) k_merge_opt(EncodeBuffers b, const __grid_constant__ DeviceTable T)
{
  TileSmem<kOptThreads>& S = tile_smem<kOptThreads>();
  tile_setup(S);
  const int lo = int(b.tile_lo);  // tiles are counted in 32 bits: 8 TB of text
  int k        = lo + int(blockIdx.x);  // the first tile of every CTA, the others by ticket
  {
    const int64_t n   = text_end(b);
    const int n_tiles = int((n + kTile - 1) / kTile);
    if (threadIdx.x == 0) {
      S.n_tiles = n_tiles;
      S.tail    = int(n - int64_t(n_tiles - 1) * kTile);
    }
    if (k >= min(int(b.tile_hi), n_tiles)) return;
  }
  if (b.starts_clock && blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned long long*>(b.counters + 12) = global_timer();
  do {
    int next = 0;
    if (threadIdx.x == 0) next = atomicAdd(b.ticket, 1);  // on its way while the tile is worked on
    tile_reset(S);
    __syncthreads();
    opt_tile(S, b, T, k);
    if (threadIdx.x == 0) S.ticket = next;
    __syncthreads();
    k = lo + int(gridDim.x) + S.ticket;
  } while (k < min(int(b.tile_hi), S.n_tiles));
}

// ------------------------------------------------------------------------------------------------
// small batches (latency mode): ONE kernel, one CTA, does the chunker, every tile, the output
// scans and the pack.  Input and output pointers may be mapped host memory, so a call is one
// launch and one stream synchronisation.
// ------------------------------------------------------------------------------------------------

// single-CTA exclusive scan of f(0..n) into out[0..n] (int64); returns the total to every thread
template <class F>
__device__ int64_t cta_exclusive_scan(F f, int64_t n, int64_t* out, int* scanbuf, int64_t* carry_s)
{
  if (threadIdx.x == 0) *carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < n; base += kOptThreads) {
    const int64_t i = base + threadIdx.x;
    const int v     = (i < n) ? int(f(i)) : 0;
    int total;
    const int off       = block_exclusive_scan(v, scanbuf, &total);
    const int64_t carry = *carry_s;
    if (i < n) out[i] = carry + off;
    __syncthreads();
    if (threadIdx.x == 0) *carry_s = carry + total;
    __syncthreads();
  }
  const int64_t total = *carry_s;
  if (threadIdx.x == 0) out[n] = total;
  __syncthreads();
  return total;
}

// The scans of a medium batch, one CTA of kMediumThreads: rounds of four items per thread.  The items are
// evaluated in lane order (coalesced loads) into shared memory and scanned in blocks of four per thread (each
// thread then writes 32 contiguous bytes of offsets).
constexpr int kMediumThreads = 1024;  // more warps hide the latency of the dependent loads of a single CTA
template <class F>
__device__ int64_t cta_exclusive_scan_medium(F f, int64_t n, int64_t* out, int* scanbuf, int64_t* carry_s, int* stage)
{
  constexpr int E = 4;
  const int tid = threadIdx.x;
  if (tid == 0) *carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < n; base += int64_t(kMediumThreads) * E) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int64_t i = base + e * kMediumThreads + tid;
      stage[e * kMediumThreads + tid] = (i < n) ? int(f(i)) : 0;
    }
    __syncthreads();
    const int4 v = reinterpret_cast<const int4*>(stage)[tid];
    int total;
    const int off       = block_exclusive_scan(v.x + v.y + v.z + v.w, scanbuf, &total);
    const int64_t first = base + int64_t(tid) * E;
    const int64_t r0    = *carry_s + off;
    const int64_t r[4]  = {r0, r0 + v.x, r0 + v.x + v.y, r0 + v.x + v.y + v.z};
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (first + e < n) out[first + e] = r[e];
    __syncthreads();
    if (tid == 0) *carry_s += total;
    __syncthreads();
  }
  const int64_t total = *carry_s;
  if (tid == 0) out[n] = total;
  __syncthreads();
  return total;
}

// Medium batches (a few thousand texts, chunks and tiles at most): the whole chunker in one single-CTA launch
// instead of five, and both output scans plus the text offsets in one instead of seven -- at these sizes the
// launches, not the work, are what the multi-block kernels cost.
constexpr int64_t kMediumMaxItems = 16384;

__global__ void __launch_bounds__(kMediumThreads) k_chunker_medium(EncodeBuffers b, int per_text)
{
  __shared__ int scanbuf[33];
  __shared__ int64_t carry_s;
  __shared__ __align__(16) int stage[4 * kMediumThreads];
  const int tid = threadIdx.x;
  // this launch also resets the call's counters and per-chunk counts (two memsets less on the host)
  if (tid < 16) b.counters[tid] = 0;
  for (int64_t c = tid; c <= b.chunk_cap; c += kMediumThreads) b.chunk_cnt[c] = 0;
  const int64_t C = cta_exclusive_scan_medium(ChunksPerText{b.text_off, b.chunk_bytes}, b.n_texts, b.text_chunk_base,
                                              scanbuf, &carry_s, stage);
  if (tid == 0) b.totals[0] = C;
  if (per_text) {
    // many short texts: every text writes the offsets of its own chunks (no search); a thread takes the texts of up to
    // 32 chunks, a warp the longer ones.
    // A medium batch has at most 2048 tiles, so byte offsets and chunk numbers fit 32 bits.
    constexpr int kLongTexts = 128;
    __shared__ int n_long;
    __shared__ int long_text[kLongTexts];
    const uint32_t cb = uint32_t(b.chunk_bytes);
    if (tid == 0) {
      b.chunk_off[C] = b.text_off[b.n_texts];
      n_long         = 0;
    }
    __syncthreads();
    for (int64_t t = tid; t < b.n_texts; t += kMediumThreads) {
      const uint32_t c0 = uint32_t(b.text_chunk_base[t]), nc = uint32_t(b.text_chunk_base[t + 1]) - c0;
      const uint32_t at = uint32_t(b.text_off[t]);
      if (nc == 1) {
        b.chunk_off[c0] = at;
      } else if (nc <= 32) {
        for (uint32_t c = 0; c < nc; ++c) b.chunk_off[c0 + c] = at + c * cb;
      } else {
        const int q = atomicAdd(&n_long, 1);
        if (q < kLongTexts) long_text[q] = int(t);
      }
    }
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5;
    if (n_long <= kLongTexts) {  // the usual case: the few long texts come from the list
      for (int q = warp; q < n_long; q += kMediumThreads / 32) {
        const int64_t t   = long_text[q];
        const uint32_t cc = uint32_t(b.text_chunk_base[t]), nn = uint32_t(b.text_chunk_base[t + 1]) - cc;
        const uint32_t at = uint32_t(b.text_off[t]);
        for (uint32_t c = lane; c < nn; c += 32) b.chunk_off[cc + c] = at + c * cb;
      }
      return;
    }
    for (int64_t t0 = int64_t(warp) * 32; t0 < b.n_texts; t0 += kMediumThreads) {
      const int64_t t   = t0 + lane;
      const uint32_t c0 = (t < b.n_texts) ? uint32_t(b.text_chunk_base[t]) : 0u;
      const uint32_t nc = (t < b.n_texts) ? uint32_t(b.text_chunk_base[t + 1]) - c0 : 0u;
      for (uint32_t m = __ballot_sync(0xFFFFFFFFu, nc > 32); m; m &= m - 1) {
        const int src     = __ffs(int(m)) - 1;
        const uint32_t cc = __shfl_sync(0xFFFFFFFFu, c0, src), nn = __shfl_sync(0xFFFFFFFFu, nc, src);
        const uint32_t at = uint32_t(b.text_off[t0 + src]);
        for (uint32_t c = lane; c < nn; c += 32) b.chunk_off[cc + c] = at + c * cb;
      }
    }
    return;
  } else {
    for (int64_t c = tid; c <= C; c += kMediumThreads) {
      if (c == C) {
        b.chunk_off[c] = b.text_off[b.n_texts];
        continue;
      }
      int64_t lo = 0, hi = b.n_texts;  // last t with text_chunk_base[t] <= c
      while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (b.text_chunk_base[mid] <= c) lo = mid; else hi = mid;
      }
      b.chunk_off[c] = b.text_off[lo] + (c - b.text_chunk_base[lo]) * int64_t(b.chunk_bytes);
    }
  }
}

// ids per group of tiles, scanned (group_base), for large batches
__global__ void __launch_bounds__(kMediumThreads) k_scan_groups(EncodeBuffers b)
{
  __shared__ int scanbuf[33];
  __shared__ int64_t carry_s;
  __shared__ __align__(16) int stage[4 * kMediumThreads];
  cta_exclusive_scan_medium(CountsI32{b.group_cnt}, b.n_tiles / kTileGroup + 1, b.group_base, scanbuf, &carry_s, stage);
}

// Counter i of a call is zero at its start, [12..13] the time of the reset, which is the first launch of the call.
__device__ __forceinline__ void reset_counter(int32_t* counters, int i)
{
  if (i == 12) *reinterpret_cast<unsigned long long*>(counters + 12) = global_timer();
  else if (i != 13) counters[i] = 0;
}

// chunks per text, scanned (totals[0], text_chunk_base), for the tile kernel; reset: the call's counters and group counts too
__global__ void __launch_bounds__(kMediumThreads) k_scan_texts_medium(EncodeBuffers b, int reset)
{
  if (reset) {
    if (threadIdx.x < 16) reset_counter(b.counters, threadIdx.x);
    for (int64_t i = threadIdx.x; i <= b.n_tiles / kTileGroup; i += kMediumThreads) b.group_cnt[i] = 0;
    if (b.n_texts == 1) return;
  }
  __shared__ int scanbuf[33];
  __shared__ int64_t carry_s;
  __shared__ __align__(16) int stage[4 * kMediumThreads];
  const int64_t C = cta_exclusive_scan_medium(ChunksPerText{b.text_off, b.chunk_bytes}, b.n_texts, b.text_chunk_base,
                                              scanbuf, &carry_s, stage);
  if (threadIdx.x == 0) b.totals[0] = C;
}

__global__ void __launch_bounds__(kMediumThreads) k_scans_medium(EncodeBuffers b)
{
  __shared__ int scanbuf[33];
  __shared__ int64_t carry_s;
  __shared__ __align__(16) int stage[4 * kMediumThreads];
  const int tid   = threadIdx.x;
  const int64_t C = b.totals[0];
  const int64_t N = cta_exclusive_scan_medium(CountsI32{b.chunk_cnt}, C, b.chunk_id_off, scanbuf, &carry_s, stage);
  if (tid == 0) b.totals[1] = N;
  if (b.text_id_off)
    for (int64_t t = tid; t <= b.n_texts; t += kMediumThreads) b.text_id_off[t] = b.chunk_id_off[b.text_chunk_base[t]];
}

// One tile of a small batch: the tiles are walked in order by one CTA, so its ids and the id offsets of the chunks that
// start in it go straight to the output, at the running id count S.run.
__device__ __forceinline__ void small_tile(TileSmem<kOptThreads>& S, const EncodeBuffers& b, const DeviceTable& T, int64_t k,
                                           int64_t C)
{
  __shared__ uint16_t woff[TileSmem<kOptThreads>::kWords];
  const int tid = threadIdx.x, lane = tid & 31;
  int* status   = b.counters + 1;
  const Span sp = batch_span(b, int(k), int(b.n_tiles), int(b.n_bytes - (b.n_tiles - 1) * kTile));
  const int64_t c0 = b.tile_chunk0[k];
  tile_cut(S, sp, T, [&](auto mark) {
    for (int64_t c = c0 + lane; c <= C; c += 32) {
      const int64_t p = b.chunk_off[c] - sp.lo;
      if (p >= sp.wlen) break;
      if (p >= 0) mark(int(p));
    }
  });
  tile_lookup(S, sp, T, status);
  const int first = S.first;
  const int end   = (S.over_start >= 0) ? S.over_start : S.end;
  tile_merge(S, T, b.seg_scratch, b.seg_scratch_tokens, status);
  const int64_t out_base = S.run;  // written by thread 0 behind the barrier at the end of the last tile
  const uint16_t* map    = b.low_id_map;
  auto put = [&](int64_t at, uint32_t t) {
    if (at < b.out_capacity) b.out_ids[at] = int32_t((map && t < 256u) ? uint32_t(__ldg(map + t)) : t);
  };
  tile_emit<kOptThreads, true>(S, first, end, woff, [&](int off, const uint16_t* ids, int n) {
    for (int j = lane; j < n; j += 32) put(out_base + off + j, ids[j]);
  });
  __syncthreads();
  const int total = S.total;
  if (S.no_space && tid == 0) atomicMax(status, int(kStatusScratchTooSmall));
  int over        = 0;
  const uint16_t* over_ids = nullptr;
  if (S.over_start >= 0) {  // CTA-uniform
    const int64_t start = sp.lo + S.over_start;
    int64_t c = c0;
    while (c + 1 < C && b.chunk_off[c + 1] <= start) ++c;
    const int64_t cend = b.chunk_off[c + 1];
    over_ids = b.seg_scratch;
    over = merge_oversize<kOptThreads>(b.bytes, start, sp.lo + kWindow, cend, b.seg_scratch, b.seg_scratch_tokens, T, status);
  }
  for (int j = tid; j < over; j += kOptThreads) put(out_base + total + j, over_ids[j]);
  // id offset of every chunk that starts in this tile: the ids in front of the tile plus the live tokens of the
  // tile in front of the chunk's first byte (a chunk start is a segment start, so it lies inside the owned
  // region, or is the start of the oversize segment right behind it)
  for (int64_t c = c0 + tid; c < C; c += kOptThreads) {
    const int64_t p64 = b.chunk_off[c] - sp.lo;
    if (p64 >= sp.own_hi) break;
    if (p64 >= 0) {
      const int p = int(p64);
      const uint32_t in_front = S.cut[p >> 5] & range_mask(p & ~31, first, end) & ((1u << (p & 31)) - 1u);
      const int64_t at = out_base + woff[p >> 5] + __popc(in_front);
      b.chunk_id_off[c]    = at;
      b.chunk_id_mirror[c] = at;
    }
  }
  __syncthreads();
  if (tid == 0) {
    S.run = out_base + total + over;
    if (k == b.n_tiles - 1) {  // the tile with the last byte closes the offsets
      b.chunk_id_off[C]    = S.run;
      b.chunk_id_mirror[C] = S.run;
    }
  }
}

__global__ void __launch_bounds__(kOptThreads) k_encode_small(EncodeBuffers b, const __grid_constant__ DeviceTable T)
{
  TileSmem<kOptThreads>& S = tile_smem<kOptThreads>();
  __shared__ int scanbuf[33];
  __shared__ int64_t carry_s;
  const int tid = threadIdx.x;
  unsigned long long t_start = 0;
  if (tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
  tile_setup(S);
  if (tid < 4) b.counters[tid] = 0;
  // One text of a few chunks (the one-string-per-call case): its chunk table is arithmetic and lives in shared
  // memory, so nothing is read over PCIe but the text itself and no search or scan runs.
  constexpr int kFastChunks = 64;
  __shared__ int64_t s_chunk_off[kFastChunks + 1];
  __shared__ int32_t s_tile_chunk0[kSmallMaxBytes / kTile + 1];
  const int64_t one_c = (b.n_bytes + b.chunk_bytes - 1) / b.chunk_bytes;
  const bool one_text = b.n_texts == 1 && one_c <= kFastChunks;  // CTA-uniform
  int64_t C;
  if (one_text) {
    C = one_c;
    for (int64_t c = tid; c <= C; c += kOptThreads) s_chunk_off[c] = min(c * int64_t(b.chunk_bytes), b.n_bytes);
    for (int64_t k = tid; k < b.n_tiles; k += kOptThreads) s_tile_chunk0[k] = int32_t((k * kTile) / b.chunk_bytes);
    b.chunk_off   = s_chunk_off;
    b.tile_chunk0 = s_tile_chunk0;
  } else {
  if (b.text_off_copy) {  // one parallel read over PCIe instead of dependent reads in the searches below
    for (int64_t t = tid; t <= b.n_texts; t += kOptThreads) b.text_off_copy[t] = b.text_off[t];
    b.text_off = b.text_off_copy;
    __syncthreads();
  }
  // chunker: chunks per text -> offsets of every chunk -> first chunk of every tile
  C = cta_exclusive_scan(ChunksPerText{b.text_off, b.chunk_bytes}, b.n_texts, b.text_chunk_base,
                         scanbuf, &carry_s);
  for (int64_t c = tid; c <= C; c += kOptThreads) {
    if (c == C) {
      b.chunk_off[c] = b.text_off[b.n_texts];
      continue;
    }
    int64_t lo = 0, hi = b.n_texts;
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (b.text_chunk_base[mid] <= c) lo = mid; else hi = mid;
    }
    b.chunk_off[c] = b.text_off[lo] + (c - b.text_chunk_base[lo]) * int64_t(b.chunk_bytes);
  }
  __syncthreads();
  for (int64_t k = tid; k < b.n_tiles; k += kOptThreads) {
    const int64_t pos = k * kTile;
    int64_t lo = 0, hi = C;
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (b.chunk_off[mid] <= pos) lo = mid; else hi = mid;
    }
    b.tile_chunk0[k] = int32_t(lo);
  }
  }
  // tiles, one after the other; each writes its ids and the id offsets of the chunks that start in it
  if (tid == 0) S.run = 0;
  for (int64_t k = 0; k < b.n_tiles; ++k) {
    __syncthreads();
    tile_reset(S);
    __syncthreads();
    small_tile(S, b, T, k, C);
  }
  __syncthreads();
  // the offsets of the texts follow from those of their chunks; the caller-visible chunk offsets may live in
  // mapped host memory, so they are read back from the copy in device memory
  if (one_text) {
    if (tid < 2) b.text_id_off[tid] = tid ? S.run : 0;
  } else {
    for (int64_t t = tid; t <= b.n_texts; t += kOptThreads) b.text_id_off[t] = b.chunk_id_mirror[b.text_chunk_base[t]];
  }
  // The results may live in mapped host memory and the host may be polling totals[3] instead of waiting for the
  // stream: every store of this CTA is made visible system-wide before the call number goes out as the last one.
  __syncthreads();
  if (tid == 0) {
    unsigned long long t_end;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
    b.totals[0] = C;
    b.totals[1] = S.run;
    b.totals[2] = int64_t(b.counters[1]);
    b.totals[4] = int64_t(t_end - t_start);
    __threadfence_system();
    *reinterpret_cast<volatile int64_t*>(b.totals + 3) = b.small_seq;
  }
}

// ------------------------------------------------------------------------------------------------
// merge kernels, one CTA per chunk
// ------------------------------------------------------------------------------------------------

// A CTA tokenises chunk [cs, ce) window by window; put(i, id) takes the chunk's i-th id, S.run counts them.  Returns false,
// with the chunk half done, when a segment needs a workspace and there is none.
template <int TH, class Put>
__device__ __forceinline__ bool tokenise_chunk(TileSmem<TH>& S, const uint8_t* bytes, int64_t cs, int64_t ce,
                                               const DeviceTable& T, uint16_t* scratch, int64_t scratch_tokens,
                                               int* status, Put put)
{
  // the first window starts at the 16-byte boundary in front of the chunk, so that every window loads whole vectors
  const int skip = int(reinterpret_cast<uintptr_t>(bytes + cs) & 15u);
  for (int64_t lo = cs - skip; lo < ce; lo += S.kOwn) {
    const bool head = lo <= cs;
    const Span sp{bytes, lo, head ? skip : 0, int(min(int64_t(S.kOwn), ce - lo)), int(min(int64_t(S.kWin), ce - lo)), !head,
                  head};
    __syncthreads();
    tile_reset(S);
    if (head && threadIdx.x == 0) S.run = 0;
    __syncthreads();
    tile_cut(S, sp, T, [](auto) {});
    tile_lookup(S, sp, T, status);
    const int first = S.first;
    const int end   = (S.over_start >= 0) ? S.over_start : S.end;
    tile_merge(S, T, scratch, scratch_tokens, status);
    if (S.no_space || (S.over_start >= 0 && scratch == nullptr)) {  // CTA-uniform
      __syncthreads();
      return false;
    }
    const int64_t run = S.run;
    tile_emit<TH, false>(S, first, end, nullptr, [&](int off, const uint16_t* ids, int n) {
      for (int j = threadIdx.x & 31; j < n; j += 32) put(run + off + j, ids[j]);
    });
    __syncthreads();
    const int total = S.total;
    int over        = 0;
    if (S.over_start >= 0) {  // CTA-uniform
      over = merge_oversize<TH>(bytes, lo + S.over_start, lo + S.kWin, ce, scratch, scratch_tokens, T, status);
      for (int j = threadIdx.x; j < over; j += TH) put(run + total + j, scratch[j]);
    }
    if (threadIdx.x == 0) S.run = run + total + over;
  }
  __syncthreads();
  return true;
}

template <int TH>
constexpr int chunk_kernel_ctas()  // 1536 resident threads per SM: 40 registers each, as in the tile kernel
{
  return 1536 / TH > 0 ? 1536 / TH : 1;
}

// GTK_MODE_BASE: one CTA per chunk from a ticket.  The threads per CTA are the caller's choice (the reference's
// BLOCK_SIZE) or follow the chunk size: a CTA of TH threads works on windows of 16 * TH bytes.
template <int TH>
__global__ void __launch_bounds__(TH, chunk_kernel_ctas<TH>()) k_merge_base(EncodeBuffers b, const __grid_constant__ DeviceTable T)
{
  TileSmem<TH>& S = tile_smem<TH>();
  const int tid   = threadIdx.x;
  const int64_t C = b.totals[0];
  int* status     = b.counters + 1;
  tile_setup(S);
  uint16_t* ws = b.seg_scratch ? b.seg_scratch + int64_t(blockIdx.x) * 2 * b.seg_scratch_tokens : nullptr;
  for (;;) {
    __syncthreads();
    if (tid == 0) S.ticket = atomicAdd(b.counters + 2, 1);
    __syncthreads();
    const int64_t c = S.ticket;
    if (c >= C) break;
    const int64_t cs = b.chunk_off[c];
    const bool done = tokenise_chunk(S, b.bytes, cs, b.chunk_off[c + 1], T, ws, b.seg_scratch_tokens, status,
                                     [&](int64_t at, uint32_t id) {
      if (GTK_IN(cs + at, b.n_bytes, 31)) b.staging[cs + at] = uint16_t(id);
    });
    if (tid == 0) {
      if (!done) atomicMax(status, int(kStatusScratchTooSmall));
      b.chunk_cnt[c] = done ? int(S.run) : 0;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Merge tables whose ids or ranks do not fit 16 bits (beyond roughly 65 000 merges): one CTA per chunk, 32-bit
// tokens and ranks (shared memory up to kWideSmemTokens tokens, else the HBM workspace), the pass-by-pass
// merge with a compaction in every pass, probes into the 16-byte-slot table.  The reference carries int32
// ids and a 64-bit pair key and so accepts any merges file (gputok_blockbpe.cu:139-157); this kernel keeps
// that property for the GPU entry points at the speed of the literal design.
// ------------------------------------------------------------------------------------------------
constexpr int kWideThreads    = 256;
constexpr int kWideSmemTokens = 4096;

__global__ void __launch_bounds__(kWideThreads) k_merge_wide(EncodeBuffers b, DeviceTable T)
{
  __shared__ __align__(16) uint32_t s_tok[kWideSmemTokens];
  __shared__ __align__(16) uint32_t s_rk[kWideSmemTokens];
  __shared__ GroupScratch gs;
  __shared__ int ticket;
  const int tid   = threadIdx.x;
  const int64_t C = b.totals[0];
  int* status     = b.counters + 1;
  for (;;) {
    __syncthreads();
    if (tid == 0) ticket = atomicAdd(b.counters + 2, 1);
    __syncthreads();
    const int64_t c = ticket;
    if (c >= C) break;
    const int64_t cs  = b.chunk_off[c];
    const int64_t L64 = b.chunk_off[c + 1] - cs;
    uint32_t *tok = s_tok, *rk = s_rk;
    if (L64 > kWideSmemTokens) {
      if (L64 > b.seg_scratch_tokens || b.seg_scratch32 == nullptr) {
        if (tid == 0) {
          atomicMax(status, int(kStatusScratchTooSmall));
          b.chunk_cnt[c] = 0;
        }
        continue;
      }
      tok = b.seg_scratch32 + int64_t(blockIdx.x) * 2 * b.seg_scratch_tokens;
      rk  = tok + b.seg_scratch_tokens;
    }
    const int L = int(L64);
    for (int i = tid; i < L; i += kWideThreads) {
      const uint32_t cur = __ldg(T.byte_to_id + b.bytes[cs + i]);
      tok[i] = cur;
      rk[i]  = (i + 1 < L) ? probe_rank_wide(T, cur, __ldg(T.byte_to_id + b.bytes[cs + i + 1])) : 0xFFFFFFFFu;
    }
    __syncthreads();
    const int len = group_merge_dense<kWideThreads / 32>(tok, rk, L, T, &gs, status);
    for (int j = tid; j < len; j += kWideThreads) b.staging32[cs + j] = int32_t(tok[j]);
    if (tid == 0) b.chunk_cnt[c] = len;
  }
}

// packs the staged 32-bit tokens of every chunk (one warp per chunk)
__global__ void __launch_bounds__(256) k_pack_wide(const int32_t* __restrict__ staging, const int64_t* __restrict__ first,
                                                   const int32_t* __restrict__ cnt, const int64_t* __restrict__ base,
                                                   const int64_t* n_units_ptr, int32_t* __restrict__ out,
                                                   int64_t capacity, const uint16_t* __restrict__ low_id_map)
{
  const int64_t U    = *n_units_ptr;
  const int lane     = threadIdx.x & 31;
  const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw   = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t u = warp; u < U; u += nw) {
    const int64_t src = first[u], dst = base[u];
    int64_t m = cnt[u];
    if (dst + m > capacity) m = capacity > dst ? capacity - dst : 0;
    for (int64_t j = lane; j < m; j += 32) {
      const uint32_t t = uint32_t(staging[src + j]);
      out[dst + j] = int32_t((low_id_map && t < 256u) ? uint32_t(__ldg(low_id_map + t)) : t);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// local-minimum rule, one CTA per chunk (GTK_MODE_LOCALMIN).  The reference's tokenize_batch runs
// this rule, not Algorithm 1 (bpe_merge_kernel_optimized, gputok_binding.cu:290-414): per pass
// every adjacent pair gets its rank; a mergeable pair is merged unless its left neighbour ranks
// strictly lower or its right neighbour ranks lower or equal; all such pairs merge in the same
// pass; at most max_iters passes.  The reference compacts with one thread; here the compaction is
// the in-place ballot/popc routine.
// ------------------------------------------------------------------------------------------------
template <int NW>
__device__ int compact_tokens(uint16_t* tok, int len, GroupScratch* gs)
{
  constexpr int G = NW * 32, E = 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = lanemask_lt();
  int out = 0;
  for (int base = 0; base < len; base += G * E) {
    uint16_t t[E];
    uint32_t bal[E];
    int wt = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int i = base + warp * 32 * E + k * 32 + lane;
      t[k]   = (i < len) ? tok[i] : uint16_t(DEAD);
      bal[k] = __ballot_sync(0xFFFFFFFFu, t[k] != DEAD);
      wt += __popc(bal[k]);
    }
    if (lane == 0) gs->wsum[warp] = uint32_t(wt);
    __syncthreads();
    int pre = 0, tot = 0;
    for (int w = 0; w < NW; ++w) {
      const int x = int(gs->wsum[w]);
      if (w < warp) pre += x;
      tot += x;
    }
    int o = out + pre;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      if (t[k] != DEAD) tok[o + __popc(bal[k] & lt)] = t[k];
      o += __popc(bal[k]);
    }
    out += tot;
    __syncthreads();
  }
  return out;
}

__global__ void __launch_bounds__(kBaseThreads) k_merge_localmin(EncodeBuffers b, DeviceTable T, int max_iters)
{
  __shared__ __align__(16) uint16_t s_tok[kBaseSmemTokens];
  __shared__ __align__(16) uint16_t s_rk[kBaseSmemTokens];
  __shared__ GroupScratch gs;
  __shared__ int ticket;
  const int tid   = threadIdx.x;
  const int64_t C = b.totals[0];
  int* status     = b.counters + 1;
  for (;;) {
    __syncthreads();
    if (tid == 0) ticket = atomicAdd(b.counters + 2, 1);
    __syncthreads();
    const int64_t c = ticket;
    if (c >= C) break;
    const int64_t cs  = b.chunk_off[c];
    const int64_t L64 = b.chunk_off[c + 1] - cs;
    uint16_t *tok = s_tok, *rk = s_rk;
    if (L64 > kBaseSmemTokens) {
      if (L64 > b.seg_scratch_tokens || b.seg_scratch == nullptr) {
        if (tid == 0) {
          atomicMax(status, int(kStatusScratchTooSmall));
          b.chunk_cnt[c] = 0;
        }
        continue;
      }
      tok = b.seg_scratch + int64_t(blockIdx.x) * 2 * b.seg_scratch_tokens;
      rk  = tok + b.seg_scratch_tokens;
    }
    int len = int(L64);
    for (int i = tid; i < len; i += kBaseThreads) tok[i] = __ldg(T.byte_to_id + b.bytes[cs + i]);
    __syncthreads();
    for (int iter = 0; iter < max_iters && len >= 2; ++iter) {
      for (int i = tid; i < len - 1; i += kBaseThreads) rk[i] = uint16_t(probe_rank(T, tok[i], tok[i + 1]));
      __syncthreads();
      bool mine = false;
      for (int i = tid; i < len - 1; i += kBaseThreads) {
        const uint32_t r = rk[i];
        if (r == NONE) continue;
        if (i > 0 && uint32_t(rk[i - 1]) < r) continue;
        if (i + 1 < len - 1 && uint32_t(rk[i + 1]) <= r) continue;
        tok[i]     = uint16_t(merged_id(T, r));  // two kept positions are never adjacent
        tok[i + 1] = uint16_t(DEAD);
        mine       = true;
      }
      if (!__syncthreads_or(mine)) break;
      len = compact_tokens<kBaseThreads / 32>(tok, len, &gs);
    }
    for (int j = tid; j < len; j += kBaseThreads) b.staging[cs + j] = tok[j];
    if (tid == 0) b.chunk_cnt[c] = len;
  }
}

// ------------------------------------------------------------------------------------------------
// output: pack staged 16-bit tokens of every unit into the int32 id buffer
// ------------------------------------------------------------------------------------------------
// A run of m tokens at sp -> ids at dp, by `stride` lanes of which this is number `lane`: groups of four as one 16-byte store
// once the destination is aligned, sixteen 16-bit loads in flight per lane and trip.
template <class Conv>
__device__ __forceinline__ void pack_run(const uint16_t* sp, int32_t* dp, int m, int lane, int stride, Conv conv)
{
  const int head = min(m, int(((16u - uint32_t(reinterpret_cast<uintptr_t>(dp) & 15u)) >> 2) & 3u));
  if (lane < head) dp[lane] = conv(sp[lane]);
  const int quads = (m - head) >> 2;
  for (int q0 = lane; q0 < quads; q0 += 4 * stride) {
    uint32_t t[4][4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int q = q0 + stride * g;
      if (q < quads) {
        const uint16_t* s4 = sp + head + 4 * q;
#pragma unroll
        for (int e = 0; e < 4; ++e) t[g][e] = s4[e];
      }
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int q = q0 + stride * g;
      if (q < quads)
        *reinterpret_cast<int4*>(dp + head + 4 * q) = make_int4(conv(t[g][0]), conv(t[g][1]), conv(t[g][2]), conv(t[g][3]));
    }
  }
  const int done = head + 4 * quads;
  if (done + lane < m) dp[done + lane] = conv(sp[done + lane]);
}

// One warp per chunk of the kernels that work chunk by chunk.
__global__ void __launch_bounds__(256) k_pack_chunks(const uint16_t* __restrict__ staging, const int64_t* __restrict__ first,
                                                     const int32_t* __restrict__ cnt, const int64_t* __restrict__ base,
                                                     const int64_t* n_units_ptr, int32_t* __restrict__ out, int64_t capacity,
                                                     const uint16_t* __restrict__ low_id_map)
{
  const int64_t U    = *n_units_ptr;
  const int lane     = threadIdx.x & 31;
  const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw   = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t u = warp; u < U; u += nw) {
    const int64_t dst = base[u];
    pack_run(staging + first[u], out + dst, int(min(int64_t(cnt[u]), max(capacity - dst, int64_t(0)))), lane, 32,
             [&](uint32_t t) { return int32_t((low_id_map && t < 256u) ? uint32_t(__ldg(low_id_map + t)) : t); });
  }
}

// Everything behind the tile kernel.  A CTA packs a run of tiles, its warps one tile each, or (kWhole, for batches that leave
// the chip idle otherwise) all of them one tile together.  Where its first tile's ids go is a sum over the counts of the
// tile groups in front and of the tiles in front within the group, which every CTA forms for itself; for large batches
// (a thousand groups at 256 MiB) k_scan_groups has formed the former.  The offsets of the chunks and texts that start in a tile are the tile's place plus
// what the tile kernel has counted.  Bound by the latency of the staged tokens and by the stores.
template <bool kWhole>
__global__ void __launch_bounds__(256) k_pack_tiles(EncodeBuffers b, int64_t per_cta, int groups_scanned, int64_t* publish,
                                                    int64_t seq)
{
  constexpr int kWarps = 8;
  __shared__ int64_t warp_sum[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t K = b.n_tiles, a = min(b.tile_lo + int64_t(blockIdx.x) * per_cta, b.tile_hi), e = min(a + per_cta, b.tile_hi);
  const uint16_t* map = b.low_id_map;
  auto conv = [&](uint32_t t) { return int32_t((map && t < 256u) ? uint32_t(__ldg(map + t)) : t); };
  const int64_t C = b.n_texts == 1 ? (text_end(b) + b.chunk_bytes - 1) / b.chunk_bytes : b.totals[0];
  if (a < e) {
    const int64_t g = a / kTileGroup;
    int64_t sum     = 0;
    if (groups_scanned) {
      if (tid == 0) sum = b.group_base[g];
    } else {
      for (int64_t i = b.tile_lo / kTileGroup + tid; i < g; i += 256) sum += b.group_cnt[i];
      if (tid == 0 && b.tile_lo > 0) sum += b.piece_ids[0];
    }
    for (int64_t i = g * kTileGroup + tid; i < a; i += 256) sum += b.unit_cnt[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
    if (lane == 0) warp_sum[warp] = sum;
    __syncthreads();
    int64_t base = 0;
    for (int w = 0; w < kWarps; ++w) base += warp_sum[w];
    constexpr int kStep = kWhole ? 1 : kWarps;
    for (int64_t k0 = a; k0 < e; k0 += kStep) {
      const int mine = kWhole ? 0 : warp;
      const int cnt  = (lane < kStep && k0 + lane < e) ? b.unit_cnt[k0 + lane] : 0;
      const int m    = __shfl_sync(0xFFFFFFFFu, cnt, mine);
      const int64_t k = k0 + mine, dst = base + __reduce_add_sync(0xFFFFFFFFu, lane < mine ? cnt : 0);
      base += __reduce_add_sync(0xFFFFFFFFu, cnt);
      if (k >= e) continue;
      const int l = kWhole ? tid : lane;
      constexpr int kStride = kWhole ? 256 : 32;
      pack_run(b.staging + b.unit_first[k], b.out_ids + dst, int(min(int64_t(m), max(b.out_capacity - dst, int64_t(0)))), l,
               kStride, conv);
      const bool end    = k == K - 1;
      const int64_t c_e = end ? C : b.tile_info[k + 1].c0;
      for (int64_t c = b.tile_info[k].c0 + l; c < c_e; c += kStride) b.chunk_id_off[c] = dst + b.chunk_rel[c];
      if (b.text_id_off) {
        const int64_t t_e = end ? b.n_texts : b.tile_info[k + 1].t0;
        for (int64_t t = b.tile_info[k].t0 + l; t < t_e; t += kStride) {
          if (b.n_texts == 1) {
            b.text_id_off[0] = 0;
          } else {
            const bool behind = end && b.text_off[t] >= b.n_bytes;  // an empty text behind all bytes
            b.text_id_off[t]  = behind ? dst + m : dst + b.text_rel[t];
          }
        }
      }
      if (k == b.tile_hi - 1 && l == 0 && b.piece_ids) b.piece_ids[1] = dst + m;
      if (end && l == 0) {
        b.chunk_id_off[C] = dst + m;
        if (b.text_id_off) b.text_id_off[b.n_texts] = dst + m;
        b.totals[0] = C;
        b.totals[1] = dst + m;
      }
    }
  }
  if (a >= e && b.tile_lo == b.tile_hi && b.piece_ids && tid == 0) b.piece_ids[1] = b.tile_lo > 0 ? b.piece_ids[0] : 0;
  if (K == 0) {  // texts without a byte
    if (b.text_id_off)
      for (int64_t t = tid; t <= b.n_texts; t += 256) b.text_id_off[t] = 0;
    if (tid == 0) b.chunk_id_off[0] = b.totals[0] = b.totals[1] = 0;
  }
  if (!publish) return;
  // The CTA that finishes last (a counter, no waiting) tells the host, which may be polling the call number: the last store,
  // behind a system-wide fence, which covers what the other CTAs have published to this one.
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(b.counters + 8, 1) != int(gridDim.x) - 1) return;
    __threadfence_system();
    publish[0] = C;
    publish[1] = *reinterpret_cast<volatile int64_t*>(b.totals + 1);
    publish[2] = int64_t(*reinterpret_cast<volatile int32_t*>(b.counters + 1));
    publish[4] = int64_t(global_timer() - *reinterpret_cast<volatile unsigned long long*>(b.counters + 12));
    __threadfence_system();
    *reinterpret_cast<volatile int64_t*>(publish + 3) = seq;
  }
}

__global__ void k_text_id_off(const int64_t* __restrict__ text_chunk_base, const int64_t* __restrict__ chunk_id_off,
                              int64_t n_texts, int64_t* __restrict__ text_id_off)
{
  for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t <= n_texts; t += int64_t(gridDim.x) * blockDim.x)
    text_id_off[t] = chunk_id_off[text_chunk_base[t]];
}

inline unsigned grid_for(int64_t items, int threads, int64_t cap = 65535)
{
  int64_t g = (items + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return unsigned(g);
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------------

// The scans have no dependent searches, so one CTA serves them up to a few thousand items; the chunker's binary
// searches (one per chunk and one per tile) are latency-bound in a single CTA and only pay while there are few.
static bool medium_scans(const EncodeBuffers& b)
{
  return b.n_texts <= kMediumMaxItems && b.chunk_cap <= kMediumMaxItems;
}
// The single-CTA chunker finds the text of every chunk by binary search, which is cheap for a few texts and a few
// thousand chunks; a batch of many short texts (no more chunk-sized pieces than texts) is laid out per text instead.
static bool medium_chunker_by_search(const EncodeBuffers& b)
{
  return b.n_texts <= 256 && b.chunk_cap <= 2048 && b.n_tiles <= 1024;
}
static bool medium_chunker_per_text(const EncodeBuffers& b)
{
  return b.n_texts <= kMediumMaxItems && b.chunk_cap <= kMediumMaxItems && b.n_tiles <= 2048 &&
         b.chunk_cap <= 2 * b.n_texts + 1;
}

// true when the chunker is the single-CTA kernel, which also resets counters[0..16) and chunk_cnt[0..chunk_cap]
bool chunker_resets_counters(const EncodeBuffers& b)
{
  return medium_chunker_by_search(b) || medium_chunker_per_text(b);
}

// One launch instead of memsets and a device-to-device copy, which take the stream 13 us: 8 MiB in L2 or HBM each way.
__global__ void __launch_bounds__(512) k_begin_batch(int32_t* counters, int32_t* group_cnt, int64_t n_groups,
                                                     const uint4* __restrict__ from, uint4* __restrict__ to, int n_words)
{
  const int i0 = blockIdx.x * 512 + threadIdx.x, step = gridDim.x * 512;
  if (i0 < 16) reset_counter(counters, i0);
  for (int64_t i = i0; i < n_groups; i += step) group_cnt[i] = 0;
  if (to)
    for (int i = i0; i < n_words; i += 4 * step) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k * step < n_words) v[k] = __ldg(from + i + k * step);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k * step < n_words) to[i + k * step] = v[k];
    }
}

static bool medium_batch(const EncodeBuffers& b) { return medium_chunker_by_search(b) || medium_chunker_per_text(b); }

int launch_begin_batch(const EncodeBuffers& b, const uint4* long_words, uint4* learned, cudaStream_t stream)
{
  if (medium_batch(b) && !learned) {
    k_scan_texts_medium<<<1, kMediumThreads, 0, stream>>>(b, 1);
    return 1;
  }
  const int64_t n_groups = b.n_tiles / kTileGroup + 1;
  const int grid = learned ? 256 : grid_for(n_groups, 512, 256);  // 256 CTAs: four words of the table per thread
  k_begin_batch<<<grid, 512, 0, stream>>>(b.counters, b.group_cnt, n_groups, long_words, learned, learned ? 2 << kLongBits : 0);
  return 1;
}

// {n_chunks, ids up to the end of the piece, status, seq} to the host, seq last.  A kernel of its own on a stream of its own: the
// fence behind stores to the host takes tens of microseconds while the link is busy, and the next piece need not wait for it.
__global__ void k_publish_piece(EncodeBuffers b, int64_t* publish, int64_t seq)
{
  publish[0] = b.totals[0];
  publish[1] = b.piece_ids[1];
  publish[2] = int64_t(b.counters[1]);
  __threadfence_system();
  *reinterpret_cast<volatile int64_t*>(publish + 3) = seq;
}

int launch_publish_piece(const EncodeBuffers& b, int64_t* publish, int64_t seq, cudaStream_t stream)
{
  k_publish_piece<<<1, 1, 0, stream>>>(b, publish, seq);
  return 1;
}

int launch_scan_texts(const EncodeBuffers& b, bool learned, cudaStream_t stream)
{
  if (b.n_texts == 1 || (medium_batch(b) && !learned)) return 0;
  if (b.n_texts <= kMediumMaxItems && b.chunk_cap < (int64_t(1) << 30)) {  // its sums are 32 bits wide
    k_scan_texts_medium<<<1, kMediumThreads, 0, stream>>>(b, 0);
    return 1;
  }
  return run_scan(ChunksPerText{b.text_off, b.chunk_bytes}, b.n_texts, b.n_texts, nullptr, b.scan_block_sums,
                  b.text_chunk_base, b.totals + 0, stream);
}

int launch_tile_info(const EncodeBuffers& b, cudaStream_t stream)
{
  if (b.n_tiles <= 0) return 0;
  k_tile_info<<<grid_for(b.n_tiles, 128, 4096), 128, 0, stream>>>(b);
  return 1;
}

// Medium batches: the pack kernel sums the group counts itself; beyond that one more launch does it once.
int launch_scan_groups(const EncodeBuffers& b, cudaStream_t stream)
{
  if (medium_batch(b)) return 0;
  k_scan_groups<<<1, kMediumThreads, 0, stream>>>(b);
  return 1;
}

int launch_pack_tiles(const EncodeBuffers& b, int sm_count, bool groups_scanned, int64_t* publish, int64_t seq, cudaStream_t stream)
{
  // Up to eight tiles per SM: a CTA for each, so that its 256 threads share the tile's 1400 ids; beyond, a warp for each.  A call over
  // 2 / 4 / 4.6 (the line: 1184 tiles) / 5 / 8 / 16 MiB of English-like text: 57 / 83 / 94 / 95 / 108 / 158 us with a CTA for each, 58 / 84 / 90 /
  // 92 / 102 / 144 with a warp.
  const int64_t n = b.tile_hi - b.tile_lo;
  if (n <= int64_t(sm_count) * 8) {
    k_pack_tiles<true><<<unsigned(std::max<int64_t>(n, 1)), 256, 0, stream>>>(b, 1, groups_scanned, publish, seq);
    return 1;
  }
  const int64_t per = 8;  // 128 MiB: this kernel 72 us, with four times as many tiles per CTA 82 us
  k_pack_tiles<false><<<unsigned((n + per - 1) / per), 256, 0, stream>>>(b, per, groups_scanned, publish, seq);
  return 1;
}

int launch_chunker(const EncodeBuffers& b, cudaStream_t stream)
{
  if (medium_chunker_by_search(b) || medium_chunker_per_text(b)) {
    k_chunker_medium<<<1, kMediumThreads, 0, stream>>>(b, medium_chunker_by_search(b) ? 0 : 1);
    return 1;
  }
  int launches = run_scan(ChunksPerText{b.text_off, b.chunk_bytes}, b.n_texts, b.n_texts, nullptr,
                          b.scan_block_sums, b.text_chunk_base, b.totals + 0, stream);
  k_chunk_fill<<<grid_for(b.chunk_cap + 1, 256, 2048), 256, 0, stream>>>(b.text_off, b.text_chunk_base, b.n_texts,
                                                                         b.chunk_bytes, b.chunk_off);
  return launches + 1;
}

int launch_merge_opt(const EncodeBuffers& b, const DeviceTable& t, int grid, cudaStream_t stream)
{
  if (b.tile_hi <= b.tile_lo) return 0;
  if (grid > b.tile_hi - b.tile_lo) grid = int(b.tile_hi - b.tile_lo);
  k_merge_opt<<<grid, kOptThreads, 0, stream>>>(b, t);
  return 1;
}

// Threads per CTA of the one-CTA-per-chunk kernels.  block_threads = 0 picks them from the chunk size: a CTA covers 16
// bytes per thread, so 64 threads take a chunk of up to 1 KiB in one window, 128 one of 2 KiB; beyond that 256 threads
// work window by window (larger CTAs leave more of their threads waiting at barriers).  64 .. 1024 (a power of two)
// forces it, which is what the reference's BLOCK_SIZE compile-time constant does (gputok_blockbpe.cu:313-315).
int chunk_kernel_threads(int chunk_bytes, int block_threads)
{
  if (block_threads > 0) return block_threads;
  return chunk_bytes <= 1024 ? 64 : chunk_bytes <= 2048 ? 128 : 256;
}

namespace {
template <int TH>
constexpr int tile_dynamic_smem()
{
  return TH <= 256 ? 0 : int(sizeof(TileSmem<TH>));
}
template <int TH>
int base_blocks_per_sm()
{
  if (tile_dynamic_smem<TH>())
    cudaFuncSetAttribute(k_merge_base<TH>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_dynamic_smem<TH>());
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_merge_base<TH>, TH, tile_dynamic_smem<TH>());
  return nb;
}
}  // namespace

int launch_merge_base(const EncodeBuffers& b, const DeviceTable& t, int grid, int block_threads, cudaStream_t stream)
{
  if (b.n_bytes <= 0) return 0;
  if (grid > b.chunk_cap) grid = int(b.chunk_cap);
  if (grid < 1) grid = 1;
  switch (chunk_kernel_threads(b.chunk_bytes, block_threads)) {
    case 64: k_merge_base<64><<<grid, 64, 0, stream>>>(b, t); break;
    case 128: k_merge_base<128><<<grid, 128, 0, stream>>>(b, t); break;
    case 256: k_merge_base<256><<<grid, 256, 0, stream>>>(b, t); break;
    case 512: k_merge_base<512><<<grid, 512, tile_dynamic_smem<512>(), stream>>>(b, t); break;
    default: k_merge_base<1024><<<grid, 1024, tile_dynamic_smem<1024>(), stream>>>(b, t); break;
  }
  return 1;
}

int launch_merge_wide(const EncodeBuffers& b, const DeviceTable& t, int grid, cudaStream_t stream)
{
  if (b.n_bytes <= 0) return 0;
  if (grid > b.chunk_cap) grid = int(b.chunk_cap);
  if (grid < 1) grid = 1;
  k_merge_wide<<<grid, kWideThreads, 0, stream>>>(b, t);
  return 1;
}

int launch_pack_wide(const EncodeBuffers& b, int grid, cudaStream_t stream)
{
  if (b.n_bytes <= 0) return 0;
  k_pack_wide<<<grid, 256, 0, stream>>>(b.staging32, b.chunk_off, b.chunk_cnt, b.chunk_id_off, b.totals + 0, b.out_ids,
                                        b.out_capacity, b.low_id_map);
  return 1;
}

int wide_kernel_max_blocks_per_sm()
{
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_merge_wide, kWideThreads, 0);
  return nb;
}

int launch_merge_localmin(const EncodeBuffers& b, const DeviceTable& t, int grid, int max_iters, cudaStream_t stream)
{
  if (b.n_bytes <= 0) return 0;
  if (grid > b.chunk_cap) grid = int(b.chunk_cap);
  if (grid < 1) grid = 1;
  k_merge_localmin<<<grid, kBaseThreads, 0, stream>>>(b, t, max_iters);
  return 1;
}

int launch_output_scans(const EncodeBuffers& b, cudaStream_t stream)
{
  if (medium_scans(b)) {
    k_scans_medium<<<1, kMediumThreads, 0, stream>>>(b);
    return 1;
  }
  // per-chunk counts -> packed id offset of every chunk (+ total id count)
  int launches = run_scan(CountsI32{b.chunk_cnt}, b.chunk_cap, 0, b.totals + 0, b.scan_block_sums, b.chunk_id_off,
                          b.totals + 1, stream);
  if (b.text_id_off) {
    k_text_id_off<<<grid_for(b.n_texts + 1, 256, 2048), 256, 0, stream>>>(b.text_chunk_base, b.chunk_id_off,
                                                                          b.n_texts, b.text_id_off);
    ++launches;
  }
  return launches;
}

int launch_pack_chunks(const EncodeBuffers& b, int grid, cudaStream_t stream)
{
  if (b.n_bytes <= 0) return 0;
  k_pack_chunks<<<grid, 256, 0, stream>>>(b.staging, b.chunk_off, b.chunk_cnt, b.chunk_id_off, b.totals + 0, b.out_ids,
                                          b.out_capacity, b.low_id_map);
  return 1;
}

int launch_encode_small(const EncodeBuffers& b, const DeviceTable& t, cudaStream_t stream)
{
  k_encode_small<<<1, kOptThreads, 0, stream>>>(b, t);
  return 1;
}

#ifdef GTK_CHECKED
// Checked build only: the record of index checks that failed since the last reset ([0] id of the first failing
// check, [1] its value, [2] its limit, [3] number of failures), plus a self-test of the mechanism: a kernel
// evaluates one check that must fail and skips the guarded store.
__global__ void k_check_selftest(int* sink)
{
  const int bad = 5 + int(threadIdx.x);
  if (GTK_IN(bad, 4, 99)) sink[bad] = 1;
}

extern "C" __attribute__((visibility("default"))) int gtk_debug_check_words(int out[4], int reset, int selftest)
{
  if (selftest) {
    int* sink = nullptr;
    if (cudaMalloc(&sink, 64) != cudaSuccess) return -1;
    k_check_selftest<<<1, 1>>>(sink);
    cudaDeviceSynchronize();
    cudaFree(sink);
  }
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  if (cudaMemcpyFromSymbol(out, g_check_words, sizeof(int) * 4) != cudaSuccess) return -1;
  if (reset) {
    const int z[4] = {0, 0, 0, 0};
    cudaMemcpyToSymbol(g_check_words, z, sizeof(z));
  }
  return 0;
}
#endif


__global__ void k_publish_totals(const int64_t* totals, const int32_t* counters, int64_t* mapped)
{
  if (threadIdx.x == 0) {
    mapped[0] = totals[0];
    mapped[1] = totals[1];
    int32_t* c = reinterpret_cast<int32_t*>(mapped + 2);
    c[0] = counters[0];
    c[1] = counters[1];
    c[2] = counters[2];
    c[3] = counters[3];
    __threadfence_system();
  }
}

// Results of a batch that ran in one piece, from their device arena [text id offsets | chunk id offsets | ids] into
// mapped host memory: the first prefix_bytes (a multiple of 16) and the n_ids ids behind them, n_ids read from the
// totals on the device.  The CTA that finishes last (a counter, no waiting) publishes the totals and, as the very
// last store behind a system-wide fence, the call number that the host polls for.
__global__ void __launch_bounds__(256) k_results_to_host(const uint4* __restrict__ src, uint4* dst, int64_t prefix_bytes,
                                                         const int64_t* totals, int32_t* counters, int64_t* mapped,
                                                         int64_t seq)
{
  const int64_t n16 = (prefix_bytes + totals[1] * 4 + 15) / 16;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n16; i += int64_t(gridDim.x) * blockDim.x)
    dst[i] = src[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(counters + 8, 1) != int(gridDim.x) - 1) return;
    __threadfence_system();
    mapped[0] = totals[0];
    mapped[1] = totals[1];
    mapped[2] = int64_t(counters[1]);  // status word
    __threadfence_system();
    *reinterpret_cast<volatile int64_t*>(mapped + 3) = seq;
  }
}

int launch_results_to_host(const EncodeBuffers& b, const void* src, void* dst, int64_t prefix_bytes, int64_t* mapped,
                           int64_t seq, cudaStream_t stream)
{
  k_results_to_host<<<148, 256, 0, stream>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst), prefix_bytes,
                                           b.totals, b.counters, mapped, seq);
  return 1;
}

int launch_publish_totals(const EncodeBuffers& b, int64_t* mapped, cudaStream_t stream)
{
  k_publish_totals<<<1, 32, 0, stream>>>(b.totals, b.counters, mapped);
  return 1;
}

int opt_kernel_max_blocks_per_sm()
{
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_merge_opt, kOptThreads, 0);
  return nb;
}

// Call once per device and chunk size (that device current): opts the kernel in to its dynamic shared memory
// and returns the resident CTAs per SM.
int base_kernel_max_blocks_per_sm(int chunk_bytes, int block_threads)
{
  switch (chunk_kernel_threads(chunk_bytes, block_threads)) {
    case 64: return base_blocks_per_sm<64>();
    case 128: return base_blocks_per_sm<128>();
    case 256: return base_blocks_per_sm<256>();
    case 512: return base_blocks_per_sm<512>();
    default: return base_blocks_per_sm<1024>();
  }
}

int localmin_kernel_max_blocks_per_sm()
{
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_merge_localmin, kBaseThreads, 0);
  return nb;
}

}  // namespace gtk

// ------------------------------------------------------------------------------------------------
// Allocation-free entry point (declared in include/gputok_b200.h): the one-CTA-per-chunk kernel with its ticket counter
// and status words in a fixed device array instead of buffers from cudaMalloc.  The kernel needs no workspace but for
// segments of several hundred bytes; chunks that have one are left to a second kernel, which merges the whole chunk pass
// by pass with the workspace of the fixed array.
// ------------------------------------------------------------------------------------------------
#include "../../include/gputok_b200.h"

namespace {

constexpr int kNoAllocCtas        = 128;                          // CTAs of the second kernel
constexpr int kNoAllocMaxTokens   = GTK_NOALLOC_MAX_CHUNK_BYTES;  // longest chunk (one token per byte at most)
constexpr size_t kNoAllocHeader   = 256;  // [0] chunk ticket, [1] status word, [2] chunks put off, [3] ticket of the second kernel, [4] CTAs done
constexpr size_t kNoAllocPerCta   = size_t(2) * kNoAllocMaxTokens * sizeof(uint16_t);  // tokens + ranks
constexpr size_t kNoAllocBytes    = kNoAllocHeader + size_t(kNoAllocCtas) * kNoAllocPerCta;  // 8 MiB + 256 B
constexpr int kMaxDevices         = 64;
constexpr int32_t kPutOff         = -1;  // count of a chunk that waits for the second kernel

// Lives in the library image on every GPU that loads it.  In host code this name is only a
// stand-in for the symbol; the device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// 2 MiB of the sample novel in 4 KiB chunks, whole call: 5.9 ms when every chunk went through the kernel below (one pass
// over the chunk per merge rank), 44 us now; see gtk_tile.cuh for what bounds it.
template <int TH>
__global__ void __launch_bounds__(TH, gtk::chunk_kernel_ctas<TH>())
k_chunks_noalloc(const uint8_t* __restrict__ bytes, int64_t n_bytes, const int64_t* __restrict__ chunk_off,
                 int64_t n_chunks, int max_chunk, int32_t* __restrict__ out_ids, int32_t* __restrict__ out_counts,
                 const __grid_constant__ gtk::DeviceTable T, const uint16_t* __restrict__ low_id_map, int* header,
                 int32_t* done, int32_t seq)
{
  using namespace gtk;
  TileSmem<TH>& S = tile_smem<TH>();
  const int tid   = threadIdx.x;
  int* status     = header + 1;
  tile_setup(S);
  for (int64_t c = blockIdx.x; c < n_chunks;) {  // the first chunk of every CTA, the others by ticket
    int next = 0;
    if (tid == 0) next = atomicAdd(header, 1);
    const int64_t cs  = chunk_off[c];
    const int64_t L64 = chunk_off[c + 1] - cs;
    // The offsets come from the caller's device memory and are used as indices below: a chunk that is not
    // inside bytes[0, n_bytes) is skipped (count 0) and reported through the status word, never touched.
    const bool outside = cs < 0 || L64 < 0 || cs > n_bytes || L64 > n_bytes - cs;
    int count = 0;
    if (outside || L64 > max_chunk) {
      if (tid == 0) atomicMax(status, outside ? int(kStatusBadOffsets) : int(kStatusScratchTooSmall));
    } else if (L64 > 0) {
      const bool done = tokenise_chunk(S, bytes, cs, cs + L64, T, nullptr, 0, status, [&](int64_t at, uint32_t t) {
        if (GTK_IN(at, L64, 32)) out_ids[cs + at] = int32_t((low_id_map && t < 256u) ? uint32_t(__ldg(low_id_map + t)) : t);
      });
      count = done ? int(S.run) : kPutOff;
      if (!done && tid == 0) atomicAdd(header + 2, 1);
    }
    if (tid == 0) {
      out_counts[c] = count;
      S.ticket      = next;
    }
    __syncthreads();
    c = int64_t(gridDim.x) + S.ticket;
  }
  // the CTA that finishes last (a counter, no waiting) tells the host, which polls for the call number
  if (tid != 0) return;
  __threadfence();
  if (atomicAdd(header + 4, 1) != int(gridDim.x) - 1) return;
  __threadfence_system();
  done[1] = *reinterpret_cast<volatile int*>(header + 1);
  done[2] = *reinterpret_cast<volatile int*>(header + 2);
  __threadfence_system();
  *reinterpret_cast<volatile int32_t*>(done + 3) = seq;
}

// the chunks that the first kernel has put off
__global__ void __launch_bounds__(gtk::kBaseThreads)
k_merge_chunks_noalloc(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ chunk_off,
                       int64_t n_chunks, int32_t* __restrict__ out_ids,
                       int32_t* __restrict__ out_counts, const __grid_constant__ gtk::DeviceTable T,
                       const uint16_t* __restrict__ low_id_map, unsigned char* scratch)
{
  using namespace gtk;
  __shared__ __align__(16) uint16_t s_tok[kBaseSmemTokens];
  __shared__ __align__(16) uint16_t s_rk[kBaseSmemTokens];
  __shared__ GroupScratch gs;
  __shared__ int ticket;
  const int tid   = threadIdx.x;
  int* header     = reinterpret_cast<int*>(scratch);
  uint16_t* w_tok = reinterpret_cast<uint16_t*>(scratch + kNoAllocHeader + size_t(blockIdx.x) * kNoAllocPerCta);
  uint16_t* w_rk  = w_tok + kNoAllocMaxTokens;
  for (;;) {
    __syncthreads();
    if (tid == 0) ticket = atomicAdd(header + 3, 1);
    __syncthreads();
    const int64_t c = ticket;
    if (c >= n_chunks) break;
    if (out_counts[c] != kPutOff) continue;
    const int64_t cs = chunk_off[c];  // checked by the first kernel, as the length is
    const int L      = int(chunk_off[c + 1] - cs);
    uint16_t* tok = (L <= kBaseSmemTokens) ? s_tok : w_tok;
    uint16_t* rk  = (L <= kBaseSmemTokens) ? s_rk : w_rk;
    for (int i = tid; i < L; i += kBaseThreads) {
      const uint32_t cur = bytes[cs + i];
      tok[i] = __ldg(T.byte_to_id + cur);
      rk[i]  = (i + 1 < L) ? __ldg(T.byte_pair_rank + ((cur << 8) | bytes[cs + i + 1])) : uint16_t(NONE);
    }
    __syncthreads();
    const int len = group_merge<kBaseThreads / 32>(tok, rk, L, T, &gs, header + 1);
    for (int j = tid; j < len; j += kBaseThreads) {
      const uint32_t t = tok[j];
      out_ids[cs + j]  = int32_t((low_id_map && t < 256u) ? uint32_t(__ldg(low_id_map + t)) : t);
    }
    __syncthreads();  // the count is read at the top of the loop
    if (tid == 0) out_counts[c] = len;
  }
}

// Device address of the fixed array, looked up once per device with that device current.
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices] = {};

cudaError_t noalloc_scratch_for(int device, unsigned char** out)
{
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[device] = static_cast<unsigned char*>(p);
  }
  *out = g_noalloc_ptr[device];
  return cudaSuccess;
}

}  // namespace

extern "C" GTK_API int gtk_encode_chunks_noalloc(gtk_tokenizer* h, const uint8_t* d_bytes, int64_t n_bytes,
                                                 const int64_t* d_chunk_offsets, int64_t n_chunks,
                                                 int32_t max_chunk_bytes, int32_t* d_out_ids, int32_t* d_out_counts)
{
  gtk::HandleView v;
  if (!gtk::handle_view(h, &v)) return GTK_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(*v.mu);
  auto fail = [&](int code, const std::string& msg) {
    *v.last_error = msg;
    return code;
  };
  if (v.device < 0) return fail(GTK_ERR_NO_DEVICE, "host-only handle: no GPU entry points");
  if (v.wide) return fail(GTK_ERR_TABLE, "the allocation-free entry point serves merge tables with ids < 65535 and ranks < 65534 only");
  if (v.device >= kMaxDevices) return fail(GTK_ERR_INVALID_ARG, "device ordinal beyond the supported range");
  if (n_chunks < 0 || n_bytes < 0 || max_chunk_bytes <= 0) return fail(GTK_ERR_INVALID_ARG, "negative or zero size");
  if (n_chunks > int64_t(0x7FFFFFF0)) return fail(GTK_ERR_INVALID_ARG, "more than 2^31 chunks in one call");
  if (max_chunk_bytes > GTK_NOALLOC_MAX_CHUNK_BYTES)
    return fail(GTK_ERR_CAPACITY, "max_chunk_bytes " + std::to_string(max_chunk_bytes) +
                                      " exceeds the allocation-free limit of " +
                                      std::to_string(GTK_NOALLOC_MAX_CHUNK_BYTES) + " bytes per chunk");
  if (n_chunks == 0) return GTK_OK;
  if (!d_bytes || !d_chunk_offsets || !d_out_ids || !d_out_counts) return fail(GTK_ERR_INVALID_ARG, "null device pointer");
  cudaError_t e = cudaSetDevice(v.device);
  unsigned char* scratch = nullptr;
  if (e == cudaSuccess) e = noalloc_scratch_for(v.device, &scratch);
  if (e != cudaSuccess) return fail(GTK_ERR_CUDA, std::string("fixed workspace lookup: ") + cudaGetErrorString(e));
  // the previous call's tickets and status words must start at zero
  e = cudaMemsetAsync(scratch, 0, kNoAllocHeader, v.stream);
  if (e != cudaSuccess) return fail(GTK_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
  const int threads = gtk::chunk_kernel_threads(max_chunk_bytes, 0);
  const int grid    = int(std::min<int64_t>(n_chunks, int64_t(v.sm_count) * (1536 / threads)));
  int* header       = reinterpret_cast<int*>(scratch);
  v.pinned_words[3] = 0;
  const int32_t seq = 1;
  switch (threads) {
    case 64:
      k_chunks_noalloc<64><<<grid, 64, 0, v.stream>>>(d_bytes, n_bytes, d_chunk_offsets, n_chunks, max_chunk_bytes, d_out_ids,
                                                      d_out_counts, v.table, v.low_id_map, header, v.pinned_words, seq);
      break;
    case 128:
      k_chunks_noalloc<128><<<grid, 128, 0, v.stream>>>(d_bytes, n_bytes, d_chunk_offsets, n_chunks, max_chunk_bytes, d_out_ids,
                                                        d_out_counts, v.table, v.low_id_map, header, v.pinned_words, seq);
      break;
    default:
      k_chunks_noalloc<256><<<grid, 256, 0, v.stream>>>(d_bytes, n_bytes, d_chunk_offsets, n_chunks, max_chunk_bytes, d_out_ids,
                                                        d_out_counts, v.table, v.low_id_map, header, v.pinned_words, seq);
      break;
  }
  e = cudaGetLastError();
  // the results and the status are complete when the call number is there: no copy, no synchronisation (52 -> 44 us a call)
  if (e == cudaSuccess) e = gtk::wait_for_word(v.pinned_words + 3, seq, v.stream);
  if (e == cudaSuccess && v.pinned_words[2] > 0) {
    k_merge_chunks_noalloc<<<int(std::min<int64_t>(n_chunks, kNoAllocCtas)), gtk::kBaseThreads, 0, v.stream>>>(
      d_bytes, d_chunk_offsets, n_chunks, d_out_ids, d_out_counts, v.table, v.low_id_map, scratch);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(v.pinned_words, scratch, 16, cudaMemcpyDeviceToHost, v.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(v.stream);
  }
  if (e != cudaSuccess) return fail(GTK_ERR_CUDA, std::string("allocation-free merge kernel: ") + cudaGetErrorString(e));
  const int status = v.pinned_words[1];
  if (status == gtk::kStatusBadOffsets)
    return fail(GTK_ERR_INVALID_ARG, "d_chunk_offsets must be non-decreasing and stay inside [0, n_bytes]: the "
                                     "offending chunks were skipped (count 0)");
  if (status == gtk::kStatusScratchTooSmall)
    return fail(GTK_ERR_CAPACITY, "a chunk is longer than max_chunk_bytes (" + std::to_string(max_chunk_bytes) + ")");
  if (status != gtk::kStatusOk) return fail(GTK_ERR_KERNEL, "merge pass made no progress");
  return GTK_OK;
}

