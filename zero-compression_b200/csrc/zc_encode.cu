// zc_encode.cu -- the ZB2 block encoder on sm_100a.  It writes, at each level, exactly the payload the
// reference CPU codec writes (src/codec2.h:43-153 with the depth of src/main.cpp:45, 54).
//
// The CPU parse walks hash chains: for position i, the `depth` most recent earlier positions whose
// 4-byte hash (16 bits) equals i's, the longest match kept (the nearest on a tie), one lazy step.  A
// chain is exactly the run of i's predecessors in a stable sort of the positions by hash, so:
//
//   k_sort_*       stable two-pass LSD radix sort of each block's positions by hash (8 + 8 bits), a
//                  CTA per 4096-position tile: digit counts, per-block scan, ranked scatter (ranks by shared
//                  masks or match_any, the tile reordered in shared memory, digit runs written together).
//                  An entry is one word: the position and 12 more bits of its 4 bytes' product
//   k_enc_chain    per sorted entry: does its chain hold an entry with the same 12 bits (a candidate of 4
//                  equal bytes)?  No: no match.  Yes: the position is marked with its place in the order
//   k_enc_walk     the greedy + lazy parse as a chain 0 -> next(0) -> ..., walked in parallel from the start
//                  of every segment of every block; a warp's walks step together, and the exact matches that
//                  a step needs are computed by the warp for all its walks at once (warp_finish), only at
//                  positions that a walk visits
//   k_enc_parse    one CTA per block: the segments that the chain enters, found over the walks' exits, re-walked from
//                  there until they meet the first walk (rounds until no exit moves), then the tokens written
//   k_enc_streams  one CTA per block, a lane a token: group starts from a running maximum of per-token thresholds
//                  and next-start chains, recent offsets from each group's start, tok / ext / sym / group streams
//                  placed by scans, offset bits gathered in shared memory, literals
//   k_enc_rans     one CTA per (block, stream): histogram, 12-bit normalisation with the reference's
//                  tie-breaks, 64 lanes coding backwards (src/codec.h:41-147)
//   k_enc_pack     one CTA per (block, part): the payload (src/codec2.h:139-152), or "stored"
//   k_enc_scan / k_enc_emit: record sizes -> offsets, payloads packed back to back
#include "zc_internal.cuh"
#include "zc_kernels.h"

namespace zc {

// per-position match record: NONE; SAT | r (the position's chain holds a candidate; r is the position's
// index in the hash-sorted order, where its chain starts: the exact best is computed when a walk of the
// parse needs it); BELOW | r (the parse found that the position's match cannot win the lazy test of the
// position before it, and left it unfinished: finished like SAT if a walk needs it exactly); or the exact
// (length - 4) << 20 | (distance - 1).  Lengths are <= 4096, so an exact record has at most 0xFFC in its
// top 12 bits, and r < 2^20 - 3, so SAT | r is never NONE.
constexpr uint32_t M_NONE = 0xFFFFFFFFu;
constexpr uint32_t M_SAT = 0xFFF00000u;
constexpr uint32_t M_BELOW = 0xFFE00000u;  // unfinished, and known to lose the lazy test of the position before
__device__ __forceinline__ bool m_is_sat(uint32_t v) { return (v >> 20) >= 0xFFEu && v != M_NONE; }
__device__ __forceinline__ bool m_is_below(uint32_t v) { return (v >> 20) == 0xFFEu; }
__device__ __forceinline__ uint32_t m_pack(uint32_t m, uint32_t d) { return ((m - 4u) << 20) | (d - 1u); }
__device__ __forceinline__ uint32_t m_len(uint32_t v) { return (v >> 20) + 4u; }
__device__ __forceinline__ uint32_t m_dist(uint32_t v) { return (v & 0xFFFFFu) + 1u; }

// 4 bytes at byte offset x of a 4-aligned buffer, from the two aligned words around it
__device__ __forceinline__ uint32_t load4(const uint8_t* base, uint64_t x) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(base) + (x >> 2);
  return __funnelshift_r(__ldg(w), __ldg(w + 1), (uint32_t)(x & 3u) * 8u);
}
// The CPU parse's hash is the top 16 bits of the 4 bytes' product with 2654435761 (src/codec2.h:47).  The
// product is a bijection of the 4 bytes, so its next 12 bits (the tag) tell 4 equal bytes from a mere hash
// collision, up to its last 4 bits.
__device__ __forceinline__ uint32_t product(uint32_t x) { return x * 2654435761u; }
// a sorted entry: its position (20 bits) and its tag
__device__ __forceinline__ uint32_t entry(uint32_t p, uint32_t prod) { return p | (prod << 16 & 0xFFF00000u); }
__device__ __forceinline__ uint32_t e_pos(uint32_t e) { return e & 0xFFFFFu; }
__device__ __forceinline__ uint32_t e_tag(uint32_t e) { return e >> 20; }

// a token in one 8-byte word: where its match starts, its length (4 .. 4096) and offset
__device__ __forceinline__ uint2 tk_pack(uint32_t i, uint32_t m, uint32_t d) { return make_uint2(i | (m - 4u) << 20, d); }
__device__ __forceinline__ uint32_t tk_i(const uint2& t) { return t.x & 0xFFFFFu; }
__device__ __forceinline__ uint32_t tk_m(const uint2& t) { return (t.x >> 20) + 4u; }

// 16 bytes at byte offset x of a 16-aligned buffer, from the two aligned vectors around them (two L1
// requests a lane where five word loads would make five; the scattered candidates' loads are what the
// parse waits for)
__device__ __forceinline__ uint4 load16(const uint8_t* base, uint64_t x) {
  const uint4* c = reinterpret_cast<const uint4*>(base + (x & ~(uint64_t)15));
  const uint4 a = __ldg(c), b = __ldg(c + 1);
  const bool w2 = x & 8u, w1 = x & 4u;
  const uint32_t sh = (uint32_t)(x & 3u) * 8u;
  const uint32_t t0 = w2 ? a.z : a.x, t1 = w2 ? a.w : a.y, t2 = w2 ? b.x : a.z, t3 = w2 ? b.y : a.w, t4 = w2 ? b.z : b.x,
                 t5 = w2 ? b.w : b.y;
  const uint32_t u0 = w1 ? t1 : t0, u1 = w1 ? t2 : t1, u2 = w1 ? t3 : t2, u3 = w1 ? t4 : t3, u4 = w1 ? t5 : t4;
  return make_uint4(__funnelshift_r(u0, u1, sh), __funnelshift_r(u1, u2, sh), __funnelshift_r(u2, u3, sh),
                    __funnelshift_r(u3, u4, sh));
}
// the first differing byte of two 16-byte windows (16 when equal)
__device__ __forceinline__ uint32_t lcp16(const uint4& a, const uint4& b) {
  const uint32_t x0 = a.x ^ b.x, x1 = a.y ^ b.y, x2 = a.z ^ b.z, x3 = a.w ^ b.w;
  const uint32_t x = x0 ? x0 : x1 ? x1 : x2 ? x2 : x3;
  const uint32_t o = x0 ? 0u : x1 ? 4u : x2 ? 8u : 12u;
  return x ? o + (((uint32_t)__ffs(x) - 1u) >> 3) : 16u;
}

// ---------------------------------------------------------------- 1. stable sort by hash
// Two stable LSD passes over the 16-bit hash (low byte, then high byte), each as three kernels over
// tiles of 4096 positions, every tile its own CTA: k_sort_count (the tile's digit counts), k_sort_scan
// (per block: each tile's start for each digit, digit-major), k_sort_scatter (ranks the tile's entries
// per digit in order, reorders the tile by digit in shared memory, and writes each digit's run to its place).
// Pass 0 reads positions in order and hashes them; it writes each entry's word and, in a byte array, its digit of
// pass 1, which reads both and writes words alone: 16 bytes moved a position in all (22 with the hash beside the
// position in both passes).  The counts array holds tiles_per_block(B) * 256 words per block.
constexpr uint32_t kSortTile = 4096, kSortThreads = 512, kSortPer = kSortTile / kSortThreads;
constexpr int kCrowd = 3;

__device__ __forceinline__ uint32_t sort_tiles(uint32_t B) { return (B + kSortTile - 1) / kSortTile; }

template <int PASS>
__device__ __forceinline__ uint32_t sort_digit(uint32_t h) { return PASS == 0 ? (h & 0xFFu) : (h >> 8); }

// each thread counts 16 consecutive entries of the tile: pass 0 hashes them from three aligned 16-byte
// loads of the input (the 19 bytes it needs, inside the input's readable slack), pass 1 reads their
// 16 digits as one 16-byte load; per-warp histograms in shared memory, summed at the end
template <int PASS>
__global__ void __launch_bounds__(256) k_sort_count(EncArgs A) {
  const uint32_t b = blockIdx.y, t = blockIdx.x, tid = threadIdx.x, w = tid >> 5;
  __shared__ uint32_t hist[8][256];
  const uint32_t n = A.in_len[b], count = n >= 4 ? n - 3 : 0;
  const uint32_t i0 = t * kSortTile, i1 = min(i0 + kSortTile, count);
#pragma unroll
  for (int k = 0; k < 8; ++k) hist[k][tid] = 0;
  __syncthreads();
  const uint32_t i = i0 + 16 * tid;
  if (i < i1) {
    uint32_t h[16];
    if (PASS == 0) {
      const uint64_t a = A.in_off[b] + i;
      const uint4* q16 = reinterpret_cast<const uint4*>(A.in + (a & ~(uint64_t)15));
      const uint4 c0 = __ldg(q16), c1 = __ldg(q16 + 1), c2 = __ldg(q16 + 2);
      const uint32_t w12[12] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w, c2.x, c2.y, c2.z, c2.w};
      const uint32_t o = (uint32_t)(a >> 2) & 3u, sh = (uint32_t)(a & 3u) * 8u;
      uint32_t u[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) u[k] = o == 0 ? w12[k] : o == 1 ? w12[k + 1] : o == 2 ? w12[k + 2] : w12[k + 3];
      uint32_t x[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) x[k] = __funnelshift_r(u[k], u[k + 1], sh);
#pragma unroll
      for (int j = 0; j < 16; ++j) h[j] = product(__funnelshift_r(x[j >> 2], x[(j >> 2) + 1], 8 * (j & 3))) >> 16;
    } else {
      const uint4 v = *reinterpret_cast<const uint4*>(A.tmp_d + (size_t)b * A.B + i);
      const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 16; ++j) h[j] = (vw[j >> 2] >> (8 * (j & 3)) & 0xFFu) << 8;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (i + j < i1) atomicAdd(&hist[w][sort_digit<PASS>(h[j])], 1u);
  }
  __syncthreads();
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) sum += hist[k][tid];
  A.scnt[((size_t)b * sort_tiles(A.B) + t) * 256 + tid] = sum;
}

// per block: counts -> each tile's start per digit (digit-major order over the block's tiles).  A thread a digit, or
// kScanParts of them over more than 16 tiles, each with a run of tiles: sums of the runs, then the starts, four tiles'
// counts in flight a thread.  (One thread a digit, a tile after the other: 0.42 ms per GiB for both passes at block
// 18 against 0.23, 0.19 for 256 blocks of 1 MiB against 0.07; at 16 tiles 0.030 against 0.034 with four.)
constexpr uint32_t kScanParts = 4;

__global__ void __launch_bounds__(256 * kScanParts) k_sort_scan(EncArgs A) {
  const uint32_t b = blockIdx.x, d = threadIdx.x & 255u, part = threadIdx.x >> 8, lane = lane_id();
  __shared__ uint32_t sums[kScanParts][256], ws[8];
  const uint32_t T = sort_tiles(A.B), parts = blockDim.x >> 8, per = (T + parts - 1) / parts;
  const uint32_t t0 = min(part * per, T), t1 = min(t0 + per, T);
  uint32_t* c = A.scnt + (size_t)b * T * 256 + d;
  uint32_t run = 0;
#pragma unroll 4
  for (uint32_t t = t0; t < t1; ++t) run += c[t * 256];
  sums[part][d] = run;
  __syncthreads();
  uint32_t before = 0, total = 0;  // of the digit: the tiles before this run, all tiles
  for (uint32_t k = 0; k < parts; ++k) {
    const uint32_t v = sums[k][d];
    if (k < part) before += v;
    total += v;
  }
  const uint32_t inc = warp_incl_scan(total);
  if (part == 0 && lane == 31) ws[d >> 5] = inc;
  __syncthreads();
  uint32_t at = before + inc - total;
  for (uint32_t k = 0; k < (d >> 5); ++k) at += ws[k];
  for (uint32_t t = t0; t < t1; t += 4) {
    uint32_t v[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) v[k] = t + k < t1 ? c[(t + k) * 256] : 0u;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      if (t + k < t1) c[(t + k) * 256] = at;
      at += v[k];
    }
  }
}

// The tile's entries ranked per digit, reordered and written: latency, shared memory and instruction issue about evenly,
// so 64 warps an SM matter most (tiles of 8192, with 48, took 12.0 ms for both passes over 1 GiB of lz_mix at block 18
// where these took 9.9).  The warps' digit counts are 16 bits, cleared by one store a thread and summed two digits a
// word (32-bit words: 10.8 ms).  Now 9.3 ms, 64 MiB of text 0.62 (0.83 before), 1000 files 1.44 (2.10).
template <int PASS>
__global__ void __launch_bounds__(kSortThreads, 4) k_sort_scatter(EncArgs A) {
  constexpr uint32_t NW = kSortThreads / 32;
  __shared__ __align__(16) uint16_t cw[NW][256];  // per-warp digit counts, then the warp's start within the digit
  __shared__ __align__(16) uint32_t st_e[kSortTile];  // (while entries are ranked: the warps' masks)
  __shared__ uint16_t st_h[kSortTile];
  __shared__ uint32_t dst[256], ws[4];  // (dst: where a digit's run goes, less its start in the tile)
  static_assert(sizeof(cw) == 16 * kSortThreads && kSortTile <= 0xFFFF, "16 bytes a thread; counts of 16 bits");
  static_assert(kSortTile >= 256 * NW, "the masks lie in the tile's array");
  const uint32_t b = blockIdx.y, t = blockIdx.x, tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
  const uint32_t n = A.in_len[b], count = n >= 4 ? n - 3 : 0;
  const uint32_t i0 = t * kSortTile;
  if (i0 >= count) return;
  const uint32_t tn = min(kSortTile, count - i0);
  const size_t so = (size_t)b * A.B;
  reinterpret_cast<uint4*>(&cw[0][0])[tid] = make_uint4(0, 0, 0, 0);
  // ranks: warp w holds the tile's entries [kSortPer * 32 w, kSortPer * 32 (w + 1)), 32 per round, in order
  // (all of a thread's entries are loaded first: the ranking's warp syncs would otherwise keep each load
  // behind the previous entry's ranking)
  uint32_t ke[kSortPer], kh[kSortPer];  // kh: the hash, and above it the entry's rank among its warp's of the digit
  const uint32_t l0 = w * (32 * kSortPer) + lane;
  if (PASS == 0) {  // (32 positions are 8 words: a thread's loads lie at one address and constants from it)
    const uint64_t x0 = A.in_off[b] + i0 + l0;
    const uint32_t* in = reinterpret_cast<const uint32_t*>(A.in) + (x0 >> 2);
    const uint32_t sh = (uint32_t)(x0 & 3u) * 8u;
#pragma unroll
    for (uint32_t j = 0; j < kSortPer; ++j) {
      ke[j] = 0; kh[j] = 0;
      if (l0 + j * 32 < tn) {
        const uint32_t x = product(__funnelshift_r(__ldg(in + 8 * j), __ldg(in + 8 * j + 1), sh));
        ke[j] = entry(i0 + l0 + j * 32, x);
        kh[j] = x >> 16;
      }
    }
  } else {  // (of the hash, the high byte alone, in the high byte's place)
#pragma unroll
    for (uint32_t j = 0; j < kSortPer; ++j) {
      ke[j] = 0; kh[j] = 0;
      if (l0 + j * 32 < tn) {
        ke[j] = A.tmp_e[so + i0 + l0 + j * 32];
        kh[j] = (uint32_t)A.tmp_d[so + i0 + l0 + j * 32] << 8;
      }
    }
  }
  __syncthreads();
  // The lanes with a lane's digit: a mask a digit and warp, or-ed together in shared memory, or match_any, which takes
  // two of an SM's cycles for each different value in the warp; in masks equal digits wait for one word.  A round takes
  // match_any if the one before had a digit of more than kCrowd lanes, as in short periods and runs; pass 0 begins with
  // masks (in position order the hashes' low bytes are nearly all different), pass 1 with match_any.  Both passes, ms,
  // match_any alone / masks by this rule in pass 0 / in both: 1 GiB of lz_mix 9.9 / 9.24 / 9.33, 64 MiB of text 0.77 /
  // 0.62 / 0.62, 1000 files 1.94 / 1.65 / 1.44.  (Masks alone in pass 0: 9.6, 0.63, 1.68.)
  uint32_t* mask = st_e + 256 * w;
  bool crowded = PASS == 1;
#pragma unroll
  for (uint32_t j = 0; j < kSortPer; ++j) {
    const bool on = l0 + j * 32 < tn;
    const uint32_t d = on ? sort_digit<PASS>(kh[j]) : 256u;
    uint32_t peers;
    if (crowded) {
      peers = __match_any_sync(kFull, d);
    } else {
      if (on) mask[d] = 0;
      __syncwarp();
      if (on) atomicOr(&mask[d], 1u << lane);
      __syncwarp();
      peers = on ? mask[d] : 0u;
    }
    const uint32_t lower = peers & ((1u << lane) - 1u), c = on ? cw[w][d] : 0u;
    __syncwarp();
    if (on && !lower) cw[w][d] = (uint16_t)(c + __popc(peers));
    crowded = __any_sync(kFull, __popc(peers) > kCrowd);
    __syncwarp();
    kh[j] |= (c + __popc(lower)) << 16;
  }
  __syncthreads();
  // two digits a thread (a word of counts): the tile's counts, and those of the digits before them in the warp
  uint32_t run = 0, inc = 0, both = 0;
  uint32_t* cw2 = reinterpret_cast<uint32_t*>(&cw[0][0]) + tid;
  if (tid < 128) {
#pragma unroll 8
    for (uint32_t k = 0; k < NW; ++k) run += cw2[k * 128];
    both = (run & 0xFFFFu) + (run >> 16);
    inc = warp_incl_scan(both);
    if (lane == 31) ws[w] = inc;
  }
  __syncthreads();
  if (tid < 128) {  // each warp's starts of the digits in the reordered tile
    uint32_t at = inc - both;
    for (uint32_t k = 0; k < w; ++k) at += ws[k];
    at |= (at + (run & 0xFFFFu)) << 16;
    const uint2 g = *reinterpret_cast<const uint2*>(A.scnt + ((size_t)b * sort_tiles(A.B) + t) * 256 + 2 * tid);
    dst[2 * tid] = g.x - (at & 0xFFFFu);
    dst[2 * tid + 1] = g.y - (at >> 16);
#pragma unroll 8
    for (uint32_t k = 0; k < NW; ++k) { const uint32_t c = cw2[k * 128]; cw2[k * 128] = at; at += c; }
  }
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < kSortPer; ++j) {
    if (l0 + j * 32 >= tn) continue;
    const uint32_t h = kh[j] & 0xFFFFu, at = cw[w][sort_digit<PASS>(h)] + (kh[j] >> 16);
    st_e[at] = ke[j];
    st_h[at] = (uint16_t)h;
  }
  __syncthreads();
  uint32_t* oe = (PASS == 0 ? A.tmp_e : A.srt) + so;
  uint8_t* od = A.tmp_d + so;
#pragma unroll 4
  for (uint32_t i = tid; i < tn; i += kSortThreads) {
    const uint32_t h = st_h[i], dest = dst[sort_digit<PASS>(h)] + i;
    oe[dest] = st_e[i];
    if (PASS == 0) od[dest] = (uint8_t)(h >> 8);
  }
}

// ---------------------------------------------------------------- 2. which positions have a candidate
// A CTA of 256 threads per kChainTile consecutive sorted entries of a block.  A position whose chain (its
// `depth` predecessors in the order, as far as they have its hash) holds no entry of its own tag has no
// match: its record is NONE, and exact.  Every other position is marked SAT with its place in the order, and
// the parse computes its match if a walk comes there.  No input byte is read: a pass that compared every
// position's candidates took 21.4 ms per GiB on lz_mix at block 18, level 5 (the input's bytes at scattered
// positions, two 16-byte loads each, then up to 32 compares), for records of which the parse reads 7 %.
// What bounds this one is the records' scattered stores (one L1 request each).
//
// Chains are not told apart by the hash, which an entry does not hold, but by the positions: they rise within
// a chain, so an entry whose predecessor's position is higher starts a chain (bnd: a bit an entry).  A
// start that this misses only leaves entries of another hash among the candidates, which have another tag or,
// once in thousands, fewer than 4 bytes in common: the parse finds no match there.
// A warp's match_any over 32 entries' tags decides those with a candidate among the 32 and those whose chain
// starts there; the others go to a list that the CTA's lanes scan further back, two tags a word.  (A list of all
// entries whose predecessor has another tag took 1.0 ms per GiB more.)
constexpr uint32_t kChainTile = 2048, kChainLook = 256;  // (depth is at most kChainLook)

__global__ void __launch_bounds__(256) k_enc_chain(EncArgs A) {
  __shared__ __align__(16) uint16_t tag[kChainTile + kChainLook];
  __shared__ uint32_t bnd[(kChainTile + kChainLook) / 32];
  __shared__ uint16_t list[kChainTile];
  __shared__ uint32_t nlist;
  const uint32_t b = blockIdx.y, t = threadIdx.x, lane = lane_id(), below = (1u << lane) - 1u;
  const uint32_t r0 = blockIdx.x * kChainTile;
  const uint32_t n = A.in_len[b];
  if (r0 >= n) return;
  const uint32_t count = n >= 4 ? n - 3 : 0;
  const size_t so = (size_t)b * A.B;
  const uint32_t* E = A.srt + so;
  const uint32_t D = (uint32_t)A.depth;
  const uint32_t look = (D + 31u) & ~31u;  // (whole words of bnd)
  const uint32_t e0 = r0 > look ? r0 - look : 0, e1 = min(r0 + kChainTile, count), own = r0 - e0;
  if (t == 0) nlist = 0;
  __syncthreads();
  // (the next entries are loaded before these are looked at: 5.4 ms per GiB of lz_mix without, 4.4 with)
  uint32_t next = e0 + t < e1 ? E[e0 + t] : 0u, next0 = lane == 0 && e0 + t > 0 && e0 + t < e1 ? E[e0 + t - 1] : 0xFFFFFFFFu;
  for (uint32_t i = t; e0 + (i & ~31u) < e1; i += 256) {
    const uint32_t r = e0 + i;
    const bool on = r < e1;
    const uint32_t e = next, e_0 = next0;
    if (r + 256 < e1) {
      next = E[r + 256];
      if (lane == 0) next0 = E[r + 255];
    } else {
      next = 0u;
    }
    uint32_t before = __shfl_up_sync(kFull, e, 1);
    if (lane == 0) before = e_0;
    const unsigned m = __ballot_sync(kFull, e_pos(before) >= e_pos(e));
    if (lane == 0) bnd[i >> 5] = m;
    tag[i] = (uint16_t)e_tag(e);
    if (i < own) continue;  // (whole warps: own is a multiple of 32)
    const uint32_t starts = m & (below | 1u << lane);
    const uint32_t chain = starts ? 0xFFFFFFFFu << (31u - __clz(starts)) : 0xFFFFFFFFu;  // lanes from the chain's start on
    const uint32_t same = __match_any_sync(kFull, e_tag(e)) & below & chain;
    const bool found = same && lane - (31u - __clz(same)) <= D;
    const bool ask = on && !found && !starts && lane < D;  // (lane entries back were looked at)
    const unsigned am = __ballot_sync(kFull, ask);
    if (am) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&nlist, (uint32_t)__popc(am));
      at = __shfl_sync(kFull, at, 0);
      if (ask) list[at + __popc(am & below)] = (uint16_t)i;
    }
    if (on && !ask) A.minfo[so + e_pos(e)] = found ? M_SAT | r : M_NONE;
  }
  // positions past the last hashed one (the block's final 3 bytes) have no match
  for (uint32_t r = max(r0, count) + t; r < min(r0 + kChainTile, n); r += 256) A.minfo[so + r] = M_NONE;
  __syncthreads();
  const uint32_t* tw = reinterpret_cast<const uint32_t*>(tag);
  for (uint32_t k = t; k < nlist; k += 256) {
    const uint32_t i = list[k], tt = tag[i] * 0x00010001u;
    uint32_t lo = i > D ? i - D : 0;  // the chain's first entry within the depth: the last start before these 32
    for (int w = (int)(i >> 5) - 1; w >= (int)(lo >> 5); --w)
      if (bnd[w]) { lo = max(lo, 32u * w + 31u - __clz(bnd[w])); break; }
    bool found = false;
    const int w0 = (int)(lo >> 1);
    for (int w = (int)((i & ~31u) >> 1) - 1; w >= w0; --w) {  // two tags a word, the nearest first
      const uint32_t x = tw[w] ^ tt;
      uint32_t z = (x - 0x00010001u) & ~x & 0x80008000u;  // a half of x that is zero (a borrow can only add one)
      if (w == w0 && (lo & 1u)) z &= 0x80000000u;
      if (z) { found = true; break; }
    }
    A.minfo[so + e_pos(E[e0 + i])] = found ? M_SAT | (e0 + i) : M_NONE;
  }
}

// ---------------------------------------------------------------- 3. the parse
struct ParseBlock {
  const uint8_t* in;
  uint64_t base;
  uint32_t n, depth;
  uint32_t* minfo;
  const uint32_t* srt;
};

// A warp's requests for exact matches, one a lane (slot = lane), and the candidates still to be compared, in shared
// memory.  A candidate is slot << 20 | its position.
constexpr uint32_t kTasks = 4;                        // chain loads in flight together
constexpr uint32_t kItems = 32 + 32 * kTasks;         // the most candidates that wait at a time
constexpr uint32_t kBatch = 32, kPause = 256;
struct Finish {
  uint4 xw[32];                                       // the first 16 bytes at the request's position
  uint32_t x[32], key[32];                            // its position; best so far
  uint4 req[32];  // the requests one after the other: the entry's place | tag << 20; position | an offset << 20; the 4
                  // bytes there, which a candidate that matters has too; slot << 20
  uint32_t it[kItems], deep[kItems];  // not compared, then those equal for 32 bytes; equal for 16
  uint32_t batch[kBatch];
};

// key: (length - 1) << 20 | the candidate's position: the longest match, the nearest on a tie, is the largest
__device__ __forceinline__ uint32_t k_len(uint32_t key) { return (key >> 20) + 1u; }

// What a walk knows of the bytes that it comes to: up to position `end` they equal those `dist` before them (0: nothing).
struct Known {
  uint32_t end = 0, dist = 0;
};

// Works the lists off: cnt candidates not compared (W.it), n2 equal for 16 bytes (W.deep), into the slots' keys.
// (One of the two counts is 0, so no list grows over kItems.)  With KNOW, each lane brings its request's `kn`.
template <bool KNOW>
__device__ __forceinline__ void finish_lists(const ParseBlock& P, Finish& W, uint32_t cnt, uint32_t n2, const Known& kn) {
  const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
  const uint64_t base = P.base;
  uint32_t* const far = W.it;  // (equal for 32 bytes: written when W.it has been worked off)
  __syncwarp();
  // the first 16 bytes, a lane a candidate
  for (uint32_t k = 0; k < cnt; k += 32) {
    const bool on = k + lane < cnt;
    const uint32_t c = on ? W.it[k + lane] : 0u, i = c >> 20, j = c & 0xFFFFFu;
    bool more = false;
    if (on) {
      const uint32_t lim = min(kMaxMatch, P.n - W.x[i]);
      const uint32_t l = lcp16(load16(P.in, base + j), W.xw[i]);
      if (l >= 4u) atomicMax(&W.key[i], (min(l, lim) - 1u) << 20 | j);  // (lim >= 4)
      more = l == 16u && lim > 16u;
    }
    const unsigned mm = __ballot_sync(kFull, more);
    if (more) W.deep[n2 + __popc(mm & below)] = c;
    n2 += (uint32_t)__popc(mm);
  }
  if (!n2) { __syncwarp(); return; }
  __syncwarp();
  // the next 16, a lane a candidate
  uint32_t n3 = 0;
  bool one = false;  // of each request, one candidate is extended at a time
  for (uint32_t k = 0; k < n2; k += 32) {
    const bool on = k + lane < n2;
    const uint32_t c = on ? W.deep[k + lane] : 0u, i = c >> 20, j = c & 0xFFFFFu;
    const uint32_t x = W.x[i], key = W.key[i], lim = min(kMaxMatch, P.n - x);
    uint32_t known = 0;
    if (KNOW) {
      const uint32_t ke = __shfl_sync(kFull, kn.end, i), kd = __shfl_sync(kFull, kn.dist, i);
      if (kd == x - j && ke > x + 32) known = ke - x;
      one |= __any_sync(kFull, on && known);
    }
    bool more = false;
    if (on && !(k_len(key) == lim && j < (key & 0xFFFFFu))) {  // (a nearer match of the whole length cannot be beaten)
      const uint32_t l = known ? 16u : lcp16(load16(P.in, base + j + 16), load16(P.in, base + x + 16));
      const uint32_t len = min(known ? known : 16u + l, lim);
      if (len > 16u) atomicMax(&W.key[i], (len - 1u) << 20 | j);
      more = l == 16u && lim > max(known, 32u);
    }
    const unsigned mm = __ballot_sync(kFull, more);
    if (more) far[n3 + __popc(mm & below)] = c;
    n3 += (uint32_t)__popc(mm);
  }
  __syncwarp();
  // The rest are extended, up to 32 at a time, 32 lanes / their number each and 16 bytes a lane a step, until none is
  // left.  Of more than 32, those that can still win, of each request the first one, then the next two, four and so on:
  // one that is nearer than its request's best wins with the best's length, a farther one only with more, so it is dropped
  // when its byte there differs.  (Always the first one alone: where lengths rise with the distance, as in runs of one value
  // among few others, a request took a turn for each of its candidates.  Walks, ms, 64 MiB with a byte in 100 not zero,
  // block 16, depth 256, 13.3 / 4.5; 256 MiB of lz_mix at block 20, depth 256, 6.6 / 5.5.)
  // (Eight at a time, four lanes each: the walks took 10.3 ms for 1 GiB of lz_mix against 9.2.  Four lanes each at most: the
  // whole call 27.1 ms against 26.2, and 25 us for one match of 4096 bytes.)
  // In runs and periods the matches of all the warp's requests go on to the longest length or the run's end, at one
  // distance.  So a candidate at the distance of the one after it is compared only up to that one's position: it
  // ends where that one ends.  The parse's walks also bring what they know of the bytes before them (Known), and where
  // two candidates of a request go on after kPause bytes, the turns begin with one of each request again.
  // Walks and parse, ms, before all this / now: 256 MiB of one value at block 18 22.2 / 3.8, at block 20 and depth 256
  // 19.1 / 3.2; of a period of 5000 bytes 61.1 / 8.6 and 69.7 / 6.8; one such block of 1 MiB 30.1 / 2.2.
  for (uint32_t quota = 1; n3; quota = min(2 * quota, kBatch)) {
    uint32_t m = 0, nb = 0, carry = 32, run = 0;  // kept ones, those of this turn, the last kept one's slot and its count
    const uint32_t* batch = W.batch;
    const bool few = n3 <= kBatch && !one;
    if (few) {  // (so few that all are extended)
      batch = far;
      nb = n3;
      n3 = 0;
    }
    for (uint32_t k = 0; k < n3; k += 32) {
      const bool on = k + lane < n3;
      const uint32_t c = on ? far[k + lane] : 0u, i = c >> 20, j = c & 0xFFFFFu;
      const uint32_t x = W.x[i], key = W.key[i], lim = min(kMaxMatch, P.n - x);
      const bool best = j == (key & 0xFFFFFu);  // (the best is here only until it has been extended)
      const uint32_t at = k_len(key) - (j > (key & 0xFFFFFu) ? 1u : 0u);
      bool keep = on && at < lim;
      if (keep && !best) keep = __ldg(P.in + base + j + at) == __ldg(P.in + base + x + at);
      const unsigned km = __ballot_sync(kFull, keep);
      const unsigned pm = km & below;
      const uint32_t pi = __shfl_sync(kFull, i, pm ? 31u - __clz(pm) : 0u);
      const unsigned hm = __ballot_sync(kFull, keep && (pm ? pi : carry) != i) & (below | 1u << lane);  // first ones so far
      const uint32_t rank = hm ? __popc(pm >> (31u - __clz(hm))) : run + __popc(pm);  // among its request's
      const unsigned fm = __ballot_sync(kFull, keep && rank < quota);
      const uint32_t fk = nb + __popc(fm & below);
      const bool sel = keep && rank < quota && fk < kBatch;
      if (sel) W.batch[fk] = c;
      const unsigned rm = km & ~__ballot_sync(kFull, sel);
      if (rm >> lane & 1u) far[m + __popc(rm & below)] = c;
      m += (uint32_t)__popc(rm);
      nb = min(kBatch, nb + (uint32_t)__popc(fm));
      if (km) {
        carry = __shfl_sync(kFull, i, 31u - __clz(km));
        run = __shfl_sync(kFull, rank, 31u - __clz(km)) + 1u;
      }
      __syncwarp();
    }
    n3 = m;
    if (!nb) break;  // (none was kept)
    const uint32_t sh = (uint32_t)__clz(nb - 1u) - 27u;  // 2^sh lanes each
    const uint32_t g = lane >> sh, gl = lane & ((1u << sh) - 1u);
    bool act = g < nb, back = false;
    const uint32_t c = act ? batch[g] : 0u, i = c >> 20, j = c & 0xFFFFFu;
    const uint32_t x = W.x[i], lim = min(kMaxMatch, P.n - x);
    const bool mine = act && gl == 0;
    // the next candidate, if it is at this distance too, and the bytes before it (requests rise in position)
    uint32_t next = min((g + 1u) << sh, 31u);
    const uint32_t gap = __shfl_sync(kFull, x, next) - x, step = __shfl_sync(kFull, x - j, next);
    if (g + 1u >= nb || step != x - j) next = lane;
    const uint32_t upto = next != lane ? min(lim, gap) : lim;
    uint32_t len = 32, o = 32;
    if (KNOW) {
      const uint32_t ke = __shfl_sync(kFull, kn.end, i), kd = __shfl_sync(kFull, kn.dist, i);
      if (kd == x - j && ke > x + 32) o = ke - x;
    }
    for (uint32_t done = 32; __any_sync(kFull, act); o += 16u << sh, done += 16u << sh) {
      if (KNOW && few && done - kPause < 16u << sh) {  // (once)
        const uint32_t peers = __match_any_sync(kFull, mine && act ? i : 32u + lane);
        if (__any_sync(kFull, peers & below)) { back = act; act = false; }
      }
      const uint32_t q = o + 16u * gl;
      uint32_t e = upto;  // the match's end, if it lies in this lane's 16 bytes
      bool stop = act;
      if (act && q < upto) {
        const uint32_t l = lcp16(load16(P.in, base + j + q), load16(P.in, base + x + q));
        e = min(q + l, upto);
        stop = l < 16u || q + 16u >= upto;
      }
      const unsigned sm = __ballot_sync(kFull, stop) >> (g << sh) & 0xFFFFFFFFu >> (32u - (1u << sh));
      const uint32_t v = __shfl_sync(kFull, e, (g << sh) + (sm ? (uint32_t)__ffs(sm) - 1u : 0u));
      if (act && sm) { len = v; act = false; }
    }
    if (back || len != gap) next = lane;
    if (__any_sync(kFull, next != lane)) {  // a match that reaches the next candidate's position ends where that one does
      uint32_t end = x + len;
#pragma unroll
      for (uint32_t k = 0; k < 5; ++k) next = __shfl_sync(kFull, next, next);
      end = __shfl_sync(kFull, end, next);
      back = __shfl_sync(kFull, back, next);
      len = min(end - x, lim);
    }
    if (mine && !back) atomicMax(&W.key[i], (len - 1u) << 20 | j);
    const unsigned bm = __ballot_sync(kFull, mine && back);
    if (bm) {  // (far is empty)
      if (mine && back) far[__popc(bm & below)] = c;
      n3 = (uint32_t)__popc(bm);
      one = true;
    }
    __syncwarp();
  }
  __syncwarp();
}

// The exact matches at p, where v is unfinished, and at p + 1, where v2 is, for every lane with `act`, by the
// whole warp; v and v2 get the records, which replace the unfinished ones in minfo.  A position's chain is the
// entries before its place in the order, nearest first (the order src/codec2.h:58-67 walks them); the longest
// of the first `depth` wins, the nearest on a tie.  Three rounds:
//   0  p's nearest candidate (one of the first three entries with its tag), a lane a request, to its full length
//   1  p's other candidates: one can only win if it is longer, so it must have the 4 bytes of p that end with the
//      byte after that length; the few that do are compared
//   2  p + 1's candidates: its match is only needed if it is long enough to replace p's, which happens only if
//      8 m2 - bitlen(d2) - 8 > 8 m - bitlen(d), so (bitlen(d2) >= 0) only if 8 m2 > 8 m + 8 - bitlen(d): a
//      candidate must have the 4 bytes that end that shortest match.  When none reaches the length, v2 is NONE and
//      minfo keeps p + 1 unfinished, marked BELOW.
// In rounds 1 and 2 a request's chain is one load of its 32 predecessors (four requests a load at depth 8) and one
// word load a candidate of its tag, four such loads in flight together; the candidates that pass, of all the
// warp's requests, form one list and are compared a lane each whatever request they belong to.
// (One request after the other by the whole warp, its 32 candidates a lane each, waited for three to six
// dependent loads a request: 5.4 us each with 64 warps an SM.  Comparing every candidate of the tag, 16 bytes and
// on, took 530 warp instructions a token of lz_mix at block 18, level 5.)
template <bool KNOW>
__device__ __forceinline__ void warp_finish(const ParseBlock& P, Finish& W, bool act, uint32_t p, uint32_t& v,
                                            uint32_t& v2, const Known& kn) {
  const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
  const uint32_t G = min(32u, P.depth);  // lanes a request: 32, or 8 at depth 8
  const uint32_t gl = lane & (G - 1u), NR = 32u / G;
  const bool on0 = act && m_is_sat(v), on1 = act && m_is_sat(v2);
  const uint32_t r2 = v2 & 0xFFFFFu;
  uint32_t n2 = 0, rt = 0;
  __syncwarp();
  if (__any_sync(kFull, on0)) {
    bool more = false;
    uint32_t c = 0;
    if (on0) {
      const uint32_t r = v & 0xFFFFFu;
      const uint32_t e1 = P.srt[r - min(r, 1u)], e2 = P.srt[r - min(r, 2u)], e3 = P.srt[r - min(r, 3u)];
      const uint4 w = load16(P.in, P.base + p);
      rt = r | (product(w.x) << 16 & 0xFFF00000u);
      const uint32_t tag = rt >> 20;
      const uint32_t e = e_tag(e1) == tag ? e1 : e_tag(e2) == tag ? e2 : e3;
      const uint32_t j = e_pos(e), lim = min(kMaxMatch, P.n - p);
      uint32_t key = 0;
      if (e_tag(e) == tag && j < p) {  // (with fewer than three predecessors, e may be p's own entry)
        const uint32_t l = lcp16(load16(P.in, P.base + j), w);
        if (l >= 4u) key = (min(l, lim) - 1u) << 20 | j;
        more = l == 16u && lim > 16u;
      }
      c = lane << 20 | j;
      W.xw[lane] = w;
      W.x[lane] = p;
      W.key[lane] = key;
    }
    const unsigned mm = __ballot_sync(kFull, more);
    if (more) W.deep[__popc(mm & below)] = c;
    n2 = (uint32_t)__popc(mm);
  }
  finish_lists<KNOW>(P, W, 0, n2, kn);
  const uint32_t subs = P.depth > 32 ? 3u : 1u;  // chains are scanned 32 entries first, then the next 128, then the rest
  uint32_t need = 0;
#pragma unroll 1
  for (uint32_t ph = 1; ph < 3; ++ph) {
    const uint32_t x = p + ph - 1u, lim = min(kMaxMatch, P.n - x);
    bool ask = on0;
    uint32_t least = 0;
    if (ph == 2) {
      if (on0) {
        const uint32_t key = W.key[lane];
        v = key ? m_pack(k_len(key), p - (key & 0xFFFFFu)) : M_NONE;
        P.minfo[p] = v;
      }
      ask = on1 && v != M_NONE;
      if (ask) {
        need = ((8u * m_len(v) + 8u - bitlen(m_dist(v))) >> 3) + 1u;
        least = need - 1u;
        const uint4 w = load16(P.in, P.base + x);
        W.xw[lane] = w;
        W.x[lane] = x;
        W.key[lane] = 0;
        rt = r2 | (product(w.x) << 16 & 0xFFF00000u);
      }
    }
#pragma unroll 1
    for (uint32_t sub = 0; sub < subs; ++sub) {
      // the requests whose chains go on, each with the 4 bytes that a candidate must have to be longer than the best
      // so far (and than least)
      uint32_t at = 0;
      if (ask) {
        const uint32_t key = W.key[lane];
        at = max(least, key ? k_len(key) : 0u);
        ask = at < lim;
      }
      const unsigned am = __ballot_sync(kFull, ask);
      if (!am) break;
      const uint32_t mine = __popc(am & below);
      if (ask) {
        const uint32_t po = max(at, 3u) - 3u;
        W.req[mine] = make_uint4(rt, x | po << 20, load4(P.in, P.base + x + po), lane << 20);
      }
      __syncwarp();
      const uint32_t nreq = (uint32_t)__popc(am);
      // a load is NR requests' first entries (sub 0), or 32 entries of a request's next 128
      const uint32_t from = sub == 0 ? 0u : 128u * sub - 96u, nt = sub ? nreq * kTasks : (nreq + NR - 1) / NR;
      uint32_t t = 0, ended = 0;  // ended: a bit for each request whose chain does not go on
      do {
        uint32_t cnt = 0;
        while (t < nt && cnt <= 32) {
          uint32_t e[kTasks], xp[kTasks], pw[kTasks], w[kTasks], slot[kTasks];
          bool hit[kTasks];
#pragma unroll
          for (uint32_t u = 0; u < kTasks; ++u) {
            const uint32_t k = sub ? t / kTasks : (t + u) * NR + lane / G;
            const uint32_t q = sub ? from + 32 * u + lane : gl;
            const uint4 rq = W.req[min(k, nreq - 1u)];
            const uint32_t r = rq.x & 0xFFFFFu;
            xp[u] = rq.y; pw[u] = rq.z; slot[u] = rq.w;
            e[u] = k < nreq && q < min(P.depth, r) ? P.srt[r - 1u - q] : ~rq.x;  // (else: another tag)
            hit[u] = e[u] - (rq.x & 0xFFF00000u) < (rq.y & 0xFFFFFu);             // the same tag and an earlier position
          }
#pragma unroll
          for (uint32_t u = 0; u < kTasks; ++u)
            w[u] = hit[u] ? load4(P.in, P.base + e_pos(e[u]) + (xp[u] >> 20)) : 0u;
#pragma unroll
          for (uint32_t u = 0; u < kTasks; ++u) {
            const bool pass = hit[u] && w[u] == pw[u];
            const unsigned hm = __ballot_sync(kFull, pass);
            if (pass) W.it[cnt + __popc(hm & below)] = slot[u] | e_pos(e[u]);
            cnt += (uint32_t)__popc(hm);
          }
          if (sub + 1 < subs) {  // where the positions do not fall, or the order's start is reached, a chain has ended
                                 // (entries of other hashes that this misses are harmless: their bytes differ)
#pragma unroll
            for (uint32_t u = 0; u < kTasks; ++u) {
              const uint32_t up = __shfl_up_sync(kFull, e_pos(e[u]), 1);
              const uint32_t k = sub ? t / kTasks : t + u;
              if (__any_sync(kFull, lane > 0 && e_pos(e[u]) >= up)) ended |= 1u << (k & 31u);
            }
          }
          t += kTasks;
        }
        finish_lists<KNOW>(P, W, cnt, 0, kn);
      } while (t < nt);
      ask = ask && !(ended >> mine & 1u);
    }
  }
  if (on1) {
    v2 = M_NONE;
    if (need) {
      const uint32_t key = need <= min(kMaxMatch, P.n - p - 1u) ? W.key[lane] : 0u;
      uint32_t rec = M_BELOW | r2;  // marked, so a later walk's lazy test skips it
      if (key && k_len(key) >= need) rec = v2 = m_pack(k_len(key), p + 1 - (key & 0xFFFFFu));
      P.minfo[p + 1] = rec;
    }
  }
}

// One step of the CPU parse (src/codec2.h:69-80) for every lane with `act` (all 32 lanes call it):
// returns the next position (p itself when !act); the token, when the step emits one, in (ti, tm, td).
// Positions without a match are literal steps to the next one: a run of them is taken together with the token
// after it, up to `lim` (the walk's end), where the walk lands if the run reaches it.  A position whose
// finished record turns out to be NONE is a literal step by itself.
template <bool KNOW>
__device__ __forceinline__ uint32_t warp_step(const ParseBlock& P, Finish& W, uint32_t p, uint32_t lim, bool act,
                                              bool& tok, uint32_t& ti, uint32_t& tm, uint32_t& td,
                                              const Known& kn = Known()) {
  uint32_t v = M_NONE, v2 = M_NONE;
  if (act) {
    // eight records at a time, from two aligned loads: the first that is not NONE ends the run (a load a record, or
    // four, made a step wait for two to four times as many); its own and the next one's come from the L1 then
    const uint32_t* m = P.minfo;
    while (p < lim) {
      const uint32_t at = p & ~3u;
      const uint4 a = *reinterpret_cast<const uint4*>(m + at);
      uint4 c = make_uint4(0, 0, 0, 0);
      if (at + 4 < P.n) c = *reinterpret_cast<const uint4*>(m + at + 4);
      uint32_t some = (a.x != M_NONE ? 1u : 0u) | (a.y != M_NONE ? 2u : 0u) | (a.z != M_NONE ? 4u : 0u) |
                      (a.w != M_NONE ? 8u : 0u) | (c.x != M_NONE ? 16u : 0u) | (c.y != M_NONE ? 32u : 0u) |
                      (c.z != M_NONE ? 64u : 0u) | (c.w != M_NONE ? 128u : 0u);
      some >>= p & 3u;
      if (some) {
        p = min(p + (uint32_t)__ffs(some) - 1u, lim);
        break;
      }
      p = min(at + 8, lim);
    }
    if (p < lim) v = m[p];
    if (v != M_NONE && p + 1 < P.n) v2 = m[p + 1];
    if (m_is_below(v2)) v2 = M_NONE;  // (of no use to p's lazy test)
  }
  if (__any_sync(kFull, m_is_sat(v) || m_is_sat(v2))) warp_finish<KNOW>(P, W, act, p, v, v2, kn);
  tok = false;
  if (!act) return p;
  if (v == M_NONE) return p < lim ? p + 1 : p;
  uint32_t m = m_len(v), d = m_dist(v), at = p;
  if (v2 != M_NONE) {
    const uint32_t m2 = m_len(v2), d2 = m_dist(v2);
    if ((int)(8 * m2) - (int)bitlen(d2) - 8 > (int)(8 * m) - (int)bitlen(d)) { at = p + 1; m = m2; d = d2; }
  }
  tok = true; ti = at; tm = m; td = d;
  return at + m;
}

// The parse is a chain 0 -> next(0) -> ... cut into A.nseg segments of each block.  Every segment's walk from its
// own start, a lane a walk: it leaves the exact records of the positions that it visits in minfo, its tokens in the
// segment's slots, and where it leaves the segment, with the count, in seg_exit.  A warp takes `walks` (2 to 32)
// consecutive segments, its other lanes helping to finish records; no warp waits for another, so a launch
// of few blocks spreads over the whole GPU.  (Two or four segments a lane, handed out as lanes got done, kept more
// lanes busy, but the fewer warps took longer: 10.5, 10.8, 11.5 ms for 1 GiB of lz_mix in 512-byte segments.)
// Text in 512-byte segments is bound by L2 misses: 32 warps an SM are then in 296 blocks' candidate orders, 1.25 MiB
// each, 103 bytes read from memory a byte of input; lz_mix has few candidates and does not mind.
// The walks' own loads live on the L1, which has what 32 warps' lists leave of an SM's 256 KiB: two warps a CTA and
// 2688 bytes of lists a warp leave 128 KiB (1 GiB of lz_mix 8.7 ms, 64 MiB of text 1.62, 256 MiB at depth 256, then, 6.5);
// one, and 3584 bytes, left 64 (8.8, 1.68, 6.8).  40 or 48 warps in as many registers as that leaves: 8.9 and 9.4, text
// 1.9 and 2.5.
__global__ void __launch_bounds__(64, 16) k_enc_walk(EncArgs A, uint32_t walks) {
  __shared__ Finish Ws[2];
  Finish& W = Ws[threadIdx.x >> 5];
  const uint32_t per = A.nseg / walks, wi = blockIdx.x * 2 + (threadIdx.x >> 5);  // (per is even: 8 or more)
  const uint32_t b = wi / per, q = wi % per * walks + lane_id();
  const bool mine = lane_id() < walks;
  const uint32_t n = A.in_len[b];
  const size_t so = (size_t)b * A.B;
  ParseBlock P;
  P.in = A.in; P.base = A.in_off[b]; P.n = n; P.depth = (uint32_t)A.depth;
  P.minfo = A.minfo + so; P.srt = A.srt + so;
  const uint32_t S = seg_bytes(n, A.nseg), slots = S / 4 + 2;  // (a token takes at least 4 bytes: S / 4 + 1 at most)
  uint2* toks = A.tk_seg + (size_t)b * 2 * seg_tok_cap(A.B) + (size_t)q * slots;
  uint32_t p = mine ? min(q * S, n) : n, cnt = 0;
  const uint32_t e = min(p + S, n);
  bool t; uint32_t ta, tc, td;
  while (__any_sync(kFull, p < e)) {
    p = warp_step<false>(P, W, p, e, p < e, t, ta, tc, td);
    if (t) toks[cnt++] = tk_pack(ta, tc, td);
  }
  if (mine) A.seg_exit[(size_t)b * A.nseg + q] = make_uint2(p, cnt);
}

// One CTA per block, a lane a segment.  Each round follows the chain over the segments' exits as far as they are known,
// and a segment that it enters elsewhere than before is walked from there until that walk comes to a position of
// the first one (k_enc_walk's: its start, its tokens' ends, its exit); the segment's tokens are those of the steps
// before, then the first walk's.  A walk that starts at the wrong place meets the right one within a step or two.  The
// rounds end when no exit moves; a warp takes its part of the chain to its end before the next one.  (A whole walk from
// the true entry for the tokens: 2.26 ms per GiB of lz_mix at block 18, 0.52 for 64 MiB of text; now 0.35 and 0.17.)
// Where a match covers many segments, as in runs and periods, whose walks never meet, a step of the chain settles a
// match.  (Exits handed from each segment to the next, skipped ones among them, settled one segment a round: one block
// of 1 MiB of one value 6.5 ms, now 1.1; of 256 KiB 2.0, now 0.29.)
template <uint32_t T>
__global__ void __launch_bounds__(T, 1024 / T) k_enc_parse(EncArgs A) {
  const uint32_t b = blockIdx.x, q = threadIdx.x, lane = lane_id(), below = (1u << lane) - 1u;
  const uint32_t n = A.in_len[b];
  const size_t so = (size_t)b * A.B;
  __shared__ uint32_t hop[T], wsum[T / 32];
  extern __shared__ uint4 parse_sm[];
  Finish& W = reinterpret_cast<Finish*>(parse_sm)[q >> 5];
  ParseBlock P;
  P.in = A.in; P.base = A.in_off[b]; P.n = n; P.depth = (uint32_t)A.depth;
  P.minfo = A.minfo + so; P.srt = A.srt + so;
  const uint32_t S = seg_bytes(n, T);
  const uint32_t s = min(q * S, n), e = min(s + S, n);
  bool t; uint32_t ta, tc, td;
  const uint2 first = A.seg_exit[(size_t)b * T + q];  // the first walk's exit, its tokens
  uint32_t ent = s, ex = first.x;
  // the segment's tokens: cnt of its own slots, then the first walk's from the from-th on
  const uint32_t slots = S / 4 + 2;
  const uint2* old = A.tk_seg + (size_t)b * 2 * seg_tok_cap(A.B) + (size_t)q * slots;
  uint2* own = A.tk_seg + ((size_t)b * 2 + 1) * seg_tok_cap(A.B) + (size_t)q * slots;
  uint32_t cnt = 0, from = 0;
  // from each lane on, the warp's segments that the chain enters, the last of them, and the segment it enters after each
  uint32_t follow, far, goes;
  auto chain = [&]() {
    goes = ex >= n ? T : ex / S;  // (an exit lies past its segment)
    uint32_t nx = min(goes - (q & ~31u), 32u);
    follow = 1u << lane;
    far = lane;
#pragma unroll
    for (uint32_t o = 0; o < 5; ++o) {
      const uint32_t f = __shfl_sync(kFull, follow, nx & 31u), l = __shfl_sync(kFull, far, nx & 31u),
                     x = __shfl_sync(kFull, nx, nx & 31u);
      if (nx < 32u) { follow |= f; far = l; nx = x; }
    }
  };
  chain();
  bool entered;
  for (;;) {
    hop[q] = __shfl_sync(kFull, goes, far) | __shfl_sync(kFull, ex, far) << 11;  // (segment <= 1024, exit <= 2^20)
    __syncthreads();
    uint32_t g = 0, at = 0;  // the segment where the chain enters this warp, or a later one's, and its entry
    while (g < (q & ~31u)) {
      const uint32_t h = hop[g];
      g = h & 0x7FFu;
      at = h >> 11;
    }
    bool moved = false;
    for (;;) {  // (the warp's part of the chain to its end, then the next round)
      const uint32_t in = __shfl_sync(kFull, follow, g & 31u), prev = in & below;
      entered = (g & ~31u) == (q & ~31u) && (in >> lane & 1u);
      const uint32_t px = __shfl_sync(kFull, ex, prev ? 31u - __clz(prev) : 0u), want = prev ? px : at;
      const bool on = entered && want != ent;
      if (!__any_sync(kFull, on)) break;
      // the walk from there, and the first one's positions: its start, its tokens' ends, its exit
      uint32_t a = want, c = s, k = 0;
      Known kn;
      if (on) {
        ent = want;
        cnt = 0;
      }
      bool go = on;
      for (;;) {
        if (go) {
          while (c < a && k < first.y) {
            const uint2 f = old[k++];
            c = tk_i(f) + tk_m(f);
            kn.end = c;
            kn.dist = tk_i(f) <= a ? f.y : 0u;
          }
          if (c < a) { c = first.x; kn.end = 0; }
          go = a != c && a < e;
        }
        if (!__any_sync(kFull, go)) break;
        const uint32_t y = warp_step<true>(P, W, a, e, go, t, ta, tc, td, kn);
        if (go) {
          a = y;
          if (t) own[cnt++] = tk_pack(ta, tc, td);
        }
      }
      bool now = false;
      if (on) {
        from = a == c ? k : first.y;
        const uint32_t x = a == c ? first.x : a;
        now = x != ex;
        ex = x;
      }
      if (!__any_sync(kFull, now)) break;
      moved |= now;
      chain();
    }
    if (!__syncthreads_or(moved)) break;
  }
  if (!entered) { cnt = 0; from = first.y; }
  const uint32_t rest = first.y - from;
  const uint32_t incl = warp_incl_scan(cnt + rest);
  if (lane == 31) wsum[q >> 5] = incl;
  __syncthreads();
  // the warp's 32 segments' tokens lie one after another in the list: a lane a token, whose segment is the first with
  // a higher inclusive count
  uint32_t off = warp_sum(lane < (q >> 5) ? wsum[lane] : 0u);
  uint2* to = A.tk + (size_t)b * tok_cap(A.B) + off;
  const uint32_t all = __shfl_sync(kFull, incl, 31);
  const uint2* own0 = own - (size_t)lane * slots;
  const uint2* old0 = old - (size_t)lane * slots;
#pragma unroll 4
  for (uint32_t k0 = 0; k0 < all; k0 += 32) {
    const uint32_t k = k0 + lane;
    uint32_t l = 0;
#pragma unroll
    for (uint32_t h = 16; h; h >>= 1) l += __shfl_sync(kFull, incl, l + h - 1) <= k ? h : 0u;
    const uint32_t before = __shfl_sync(kFull, incl, l ? l - 1 : 0u), mine = __shfl_sync(kFull, cnt, l),
                   skip = __shfl_sync(kFull, from, l);
    const uint32_t j = k - (l ? before : 0u);
    const uint2* src = j < mine ? own0 + j : old0 + skip + (j - mine);
    if (k < all) to[k] = src[(size_t)l * slots];
  }
  if (q == T - 1) A.bcnt[b * 8 + 0] = off + all;
}

// ---------------------------------------------------------------- 4. tokens -> streams
constexpr uint32_t kWarpCopyRun = 32;

// n bytes from src, a range of the codec's input (16-byte aligned, 64 readable bytes after its end) or scratch, to
// dst by nth threads, this one thread t of them: 4-byte words stored aligned at dst, each built by a funnel shift from
// the two aligned input words that cover it (those may reach a few bytes past the range, into the
// input's slack, never before the input's start), four words a thread in flight.
__device__ __forceinline__ void copy_in(uint8_t* dst, const uint8_t* src, uint32_t n, uint32_t t, uint32_t nth) {
  const uint32_t head = min(n, (4u - ((uint32_t)(uintptr_t)dst & 3u)) & 3u);
  if (t < head) dst[t] = src[t];
  dst += head;
  src += head;
  n -= head;
  const uint32_t nw = n >> 2, sh = (uint32_t)(uintptr_t)src & 3u;
  const uint32_t* s = reinterpret_cast<const uint32_t*>(src - sh);
  uint32_t* d = reinterpret_cast<uint32_t*>(dst);
  if (sh) {
#pragma unroll 4
    for (uint32_t w = t; w < nw; w += nth) d[w] = __funnelshift_r(s[w], s[w + 1], 8u * sh);
  } else {
#pragma unroll 4
    for (uint32_t w = t; w < nw; w += nth) d[w] = s[w];
  }
  const uint32_t done = nw << 2;
  if (t < n - done) dst[done + t] = src[done + t];
}

// Tokens -> streams, a CTA of NW warps per block, 32 NW tokens a tile, a lane a token.
//
// Groups follow the rule of src/codec2.h:103-116: a group ends before a token whose match source starts before
// the token's own output and reaches past the group's first output byte, or once it holds 255 tokens.  A group
// opened at token g is read by token k exactly when the output start of g lies below k's source reach, and the
// output starts rise with the token index; so each token k whose source starts before its output gets
// theta_k = how many tokens start their output below its reach (at most k; only the last 255 matter), and a group
// opened at g ends at the first later token with theta > g, or at g + 255.  Within a warp's 32 tokens that is
// next(g), by a binary search over the running maximum of theta; doubling next() gives, for each lane, the group
// starts that follow if a group starts there, and the last of them.  One warp then goes through the tile's warps in
// order: the group open before a warp ends at the warp's first token that reads it, and the last start that
// follows from there is open after it.  A token's recent-offset symbols (250..252) name the offsets of the three
// tokens before its group's first token (src/codec2.h:121-137).
//
// All positions in the streams come from two packed scans (literals and group starts; ext bytes and offset bits).
// Offset bits (LSB first) are gathered in shared memory and stored as words, the last one carried to the next
// tile.
template <uint32_t NW>
struct StreamTile {
  static constexpr uint32_t NT = 32 * NW, RING = NT < 512 ? 1024 : 2 * NT;  // (a tile and the 257 tokens before it)
  uint32_t op[RING], d[RING];          // output start and offset of token k at k % RING
  uint32_t pm[NT];                     // running maximum of theta within the warp
  uint8_t last[NT];                    // the last start of the warp that follows one here
  uint32_t gin[NW], s1[NW];            // per warp: the group open before it, its first group start (32: none)
  uint32_t sum0[NW], sum1[NW];         // per warp: literals | starts << 21, ext bytes | offset bits << 16
  uint32_t bits[NT * 19 / 32 + 2];
  uint32_t big[NW * 32][3], nbig;      // literal runs that the whole CTA copies: destination, source, length
  uint32_t open;                       // the group open after the tile
};
constexpr uint32_t kCtaCopyRun = 2048;

template <uint32_t NW>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? 8 : NW == 16 ? 2 : 1) k_enc_streams(EncArgs A) {
  using T = StreamTile<NW>;
  constexpr uint32_t NT = T::NT, RM = T::RING - 1;
  __shared__ T S;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5, tid = threadIdx.x, b = blockIdx.x;
  const uint32_t n = A.in_len[b], nt = A.bcnt[b * 8 + 0];
  const uint8_t* src = A.in + A.in_off[b];
  const size_t TC = tok_cap(A.B);
  const uint2* TK = A.tk + (size_t)b * TC;
  uint8_t* lit = A.s_lit + (size_t)b * A.B;
  uint8_t* tok = A.s_tok + (size_t)b * TC;
  uint8_t* sym = A.s_sym + (size_t)b * TC;
  uint8_t* grp = A.s_grp + (size_t)b * TC;
  uint8_t* ext = A.s_ext + (size_t)b * ext_cap(A.B);
  uint32_t* bitw = reinterpret_cast<uint32_t*>(A.s_bits + (size_t)b * bits_cap(A.B));
  const uint32_t below = (1u << lane) - 1u;
  uint32_t li = 0, ei = 0, ng = 0;      // literals, ext bytes, group starts after the first, of the tiles before
  uint32_t bp = 0, cw = 0;              // offset bits of the tiles before, the last one's partly filled word
  if (tid == 0) S.open = 0;
  uint32_t ni = 0, nm = 4, nd = 1, ne = 0;  // the lane's token of the next tile, and the end of the one before it
  auto fetch = [&](uint32_t k) {
    ni = 0; nm = 4; nd = 1; ne = 0;
    if (k < nt) {
      const uint2 c = TK[k];
      ni = tk_i(c); nm = tk_m(c); nd = c.y;
      if (k) {
        const uint2 l = TK[k - 1];
        ne = tk_i(l) + tk_m(l);
      }
    }
  };
  fetch(tid);
  for (uint32_t t0 = 0; t0 < nt; t0 += NT) {
    const uint32_t k = t0 + tid;
    const bool on = k < nt;
    const uint32_t i = ni, m = nm, d = nd, opk = ne;
    S.op[k & RM] = on ? opk : 0xFFFFFFFFu;
    S.d[k & RM] = d;
    if (tid == 0) S.nbig = 0;
    for (uint32_t q = tid; q < sizeof S.bits / 4; q += NT) S.bits[q] = q ? 0u : cw;
    fetch(k + NT);
    __syncthreads();
    // theta, its running maximum, next() and what follows from each lane
    const uint32_t L = on ? i - opk : 0u;
    const uint32_t reach = i - d + min(m, d);
    uint32_t theta = 0;
    if (on && i - d < opk) {  // tokens [lo, theta) start below the reach, of the last 255
      uint32_t lo = k > 255u ? k - 255u : 0u, hi = k;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (S.op[mid & RM] < reach) lo = mid + 1; else hi = mid;
      }
      theta = lo;
    }
    uint32_t pm = theta;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, pm, o);
      if (lane >= o) pm = max(pm, v);
    }
    uint32_t nx = 0;  // the first lane with pm > k (32: none)
#pragma unroll
    for (uint32_t s = 16; s; s >>= 1)
      if (__shfl_sync(kFull, pm, nx + s - 1) <= k) nx += s;
    if (__shfl_sync(kFull, pm, nx) <= k) nx = 32;
    uint32_t follow = 1u << lane, far = lane;  // the starts from this lane on, the last of them
#pragma unroll
    for (uint32_t o = 0; o < 5; ++o) {
      const uint32_t f = __shfl_sync(kFull, follow, nx & 31u), l = __shfl_sync(kFull, far, nx & 31u),
                     x = __shfl_sync(kFull, nx, nx & 31u);
      if (nx < 32u) { follow |= f; far = l; nx = x; }
    }
    S.pm[tid] = on ? pm : 0u;
    S.last[tid] = (uint8_t)far;
    __syncthreads();
    if (w == 0) {  // the group that each warp meets, in order
      uint32_t g = S.open, p = S.pm[lane];
      for (uint32_t v = 0; v < NW; ++v) {
        const uint32_t at = t0 + 32 * v + lane;
        const unsigned e = __ballot_sync(kFull, at < nt && (p > g || at - g >= kMaxGroup) && at > g);
        if (v + 1 < NW) p = S.pm[32 * (v + 1) + lane];
        const uint32_t s = e ? (uint32_t)__ffs(e) - 1u : 32u;
        if (lane == 0) { S.gin[v] = g; S.s1[v] = s; }
        if (e) g = t0 + 32 * v + S.last[32 * v + s];
      }
      if (lane == 0) S.open = g;
    }
    __syncthreads();
    const uint32_t g0 = S.gin[w], s1 = S.s1[w];
    uint32_t starts = __shfl_sync(kFull, follow, s1 & 31u);
    if (s1 == 32u) starts = 0;
    starts &= __ballot_sync(kFull, on);
    const uint32_t mine = starts & (below | 1u << lane);
    const uint32_t gs = mine ? t0 + 32 * w + 31u - __clz(mine) : g0;
    // the offsets of tokens gs - 1, gs - 2, gs - 3, then 1, 4, 8
    const uint32_t r0 = gs >= 1 ? S.d[(gs - 1) & RM] : 1u;
    const uint32_t r1 = gs >= 2 ? S.d[(gs - 2) & RM] : gs == 1 ? 1u : 4u;
    const uint32_t r2 = gs >= 3 ? S.d[(gs - 3) & RM] : gs == 2 ? 1u : gs == 1 ? 4u : 8u;
    const uint32_t sv = d == r0 ? kSymRep : d == r1 ? kSymRep + 1 : d == r2 ? kSymRep + 2 : bitlen(d);
    if (on) {
      tok[k] = (uint8_t)((min(L, 15u) << 4) | min(m - 4u, 15u));
      sym[k] = (uint8_t)sv;
    }
    // ext bytes (src/codec2.h:120-121): L - 15 in 3 bytes when L >= 15, then m - 19 in 2 when m >= 19
    const uint32_t fl = on && L >= 15u, fm = on && m >= 19u;
    const uint32_t nbit = on && sv < kSymRep ? sv : 0u;
    const uint32_t v0 = L | (starts >> lane & 1u) << 21, v1 = 3u * fl + 2u * fm | nbit << 16;
    const uint32_t i0 = warp_incl_scan(v0), i1 = warp_incl_scan(v1);
    if (lane == 31) { S.sum0[w] = i0; S.sum1[w] = i1; }
    __syncthreads();
    const uint32_t w0 = lane < NW ? S.sum0[lane] : 0u, w1 = lane < NW ? S.sum1[lane] : 0u;
    const uint32_t c0 = warp_incl_scan(w0), c1 = warp_incl_scan(w1);
    const uint32_t p0 = __shfl_sync(kFull, c0 - w0, w) + i0 - v0, p1 = __shfl_sync(kFull, c1 - w1, w) + i1 - v1;
    const uint32_t all0 = __shfl_sync(kFull, c0, 31), all1 = __shfl_sync(kFull, c1, 31);
    if (starts >> lane & 1u) {  // a start closes the group before it
      const uint32_t before = starts & below;
      grp[ng + (p0 >> 21)] = (uint8_t)(k - (before ? t0 + 32 * w + 31u - __clz(before) : g0));
    }
    const uint32_t xq = ei + (p1 & 0xFFFFu);
    if (fl) { const uint32_t v = L - 15u; ext[xq] = (uint8_t)v; ext[xq + 1] = (uint8_t)(v >> 8); ext[xq + 2] = (uint8_t)(v >> 16); }
    if (fm) { const uint32_t v = m - 19u, y = xq + 3u * fl; ext[y] = (uint8_t)v; ext[y + 1] = (uint8_t)(v >> 8); }
    if (nbit) {
      const uint32_t at = (bp & 31u) + (p1 >> 16), x = d - (1u << nbit);
      atomicOr(&S.bits[at >> 5], x << (at & 31u));
      if ((at & 31u) + nbit > 32u) atomicOr(&S.bits[(at >> 5) + 1], x >> (32u - (at & 31u)));
    }
    // literals before each token: a lane copies its own short run, the warp a longer one, the CTA the longest
    const uint32_t lik = li + (p0 & 0x1FFFFFu);
    if (L < kWarpCopyRun) {
      for (uint32_t q = 0; q < L; ++q) lit[lik + q] = src[opk + q];
    } else if (L >= kCtaCopyRun) {
      const uint32_t q = atomicAdd(&S.nbig, 1u);
      S.big[q][0] = lik; S.big[q][1] = opk; S.big[q][2] = L;
    }
    for (unsigned lb = __ballot_sync(kFull, L >= kWarpCopyRun && L < kCtaCopyRun); lb; lb &= lb - 1) {
      const uint32_t r = (uint32_t)__ffs(lb) - 1u;
      const uint32_t rL = __shfl_sync(kFull, L, r), rd = __shfl_sync(kFull, lik, r), rs = __shfl_sync(kFull, opk, r);
      copy_in(lit + rd, src + rs, rL, lane, 32);
    }
    __syncthreads();
    for (uint32_t q = 0; q < S.nbig; ++q) copy_in(lit + S.big[q][0], src + S.big[q][1], S.big[q][2], tid, NT);
    const uint32_t end = (bp & 31u) + (all1 >> 16), full = end >> 5;  // words completed by this tile
    for (uint32_t q = tid; q < full; q += NT) bitw[(bp >> 5) + q] = S.bits[q];
    cw = S.bits[full];
    bp += all1 >> 16;
    li += all0 & 0x1FFFFFu;
    ng += all0 >> 21;
    ei += all1 & 0xFFFFu;
    __syncthreads();
  }
  __syncthreads();
  const uint32_t op = nt ? tk_i(TK[nt - 1]) + tk_m(TK[nt - 1]) : 0u;
  copy_in(lit + li, src + op, n - op, tid, NT);
  if (tid == 0) {
    if (nt) grp[ng] = (uint8_t)(nt - S.open);
    if (bp & 31u) bitw[bp >> 5] = cw;
    A.bcnt[b * 8 + 1] = li + n - op;
    A.bcnt[b * 8 + 2] = ei;
    A.bcnt[b * 8 + 3] = (bp + 7) / 8;
    A.bcnt[b * 8 + 4] = nt ? ng + 1 : 0;
  }
}

// ---------------------------------------------------------------- 5. rANS, per (block, stream)
__device__ __forceinline__ const uint8_t* stream_syms(const EncArgs& A, uint32_t b, uint32_t s) {
  const size_t TC = tok_cap(A.B);
  switch (s) {
    case 0: return A.s_lit + (size_t)b * A.B;
    case 1: return A.s_tok + (size_t)b * TC;
    case 2: return A.s_ext + (size_t)b * ext_cap(A.B);
    case 3: return A.s_sym + (size_t)b * TC;
    default: return A.s_grp + (size_t)b * TC;
  }
}
__device__ __forceinline__ uint32_t stream_len(const EncArgs& A, uint32_t b, uint32_t s) {
  const uint32_t* c = A.bcnt + b * 8;
  return s == 0 ? c[1] : s == 2 ? c[2] : s == 4 ? c[4] : c[0];
}

constexpr uint32_t kRansChunk = 4096;  // symbols staged per round: 64 per lane

__global__ void __launch_bounds__(64) k_enc_rans(EncArgs A) {
  const uint32_t b = blockIdx.x, s = blockIdx.y, k = threadIdx.x, g = b * 5 + s;
  const uint32_t ns = stream_len(A, b, s);
  uint32_t* info = A.sinfo + (size_t)g * 4;
  if (ns == 0) {
    if (k == 0) { info[0] = 0; info[1] = 0; info[2] = 0; info[3] = 0; }
    return;
  }
  const uint8_t* sym = stream_syms(A, b, s);
  // per symbol: fc = freq | cum << 13 | (ceil(log2 freq) - 1) << 25, rcp = ceil(2^(31 + ceil(log2 freq)) / freq)
  __shared__ uint32_t hist[2][256], fc[256], rcp[256], red[3];
  __shared__ __align__(16) uint8_t stage[kRansChunk];
  for (uint32_t i = k; i < 512; i += 64) (&hist[0][0])[i] = 0;
  __syncthreads();
  {  // counts, a warp's in its own half: 16 symbols a load (a byte a load was half the kernel's time on long streams)
    uint32_t* h = hist[k >> 5];
    const uint32_t nv = ((uintptr_t)sym & 15u) == 0 ? ns >> 4 : 0u;
#pragma unroll 4
    for (uint32_t i = k; i < nv; i += 64) {
      const uint4 v = reinterpret_cast<const uint4*>(sym)[i];
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 16; ++j) atomicAdd(&h[u[j >> 2] >> (8 * (j & 3)) & 0xFFu], 1u);
    }
    for (uint32_t i = 16 * nv + k; i < ns; i += 64) atomicAdd(&h[sym[i]], 1u);
  }
  __syncthreads();
  // normalisation (src/codec.h:41-66) by warp 0: lane l holds symbols 8l .. 8l+7
  if (k < 32) {
    uint32_t f[8], sum = 0, np = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t c = hist[0][k * 8 + q] + hist[1][k * 8 + q];
      f[q] = c ? max(1u, (uint32_t)(((uint64_t)c << kScaleBits) / ns)) : 0u;
      sum += f[q];
      np += c != 0;
    }
    sum = warp_sum(sum);
    np = warp_sum(np);
    // too many: one from the largest frequency above 1 (the lowest symbol on a tie), repeatedly
    while (sum > kScale) {
      uint32_t bv = 0, bi = 0xFFFFFFFFu;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (f[q] > 1 && f[q] > bv) { bv = f[q]; bi = k * 8 + q; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint32_t ov = __shfl_xor_sync(kFull, bv, o), oi = __shfl_xor_sync(kFull, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if ((bi >> 3) == k) {
#pragma unroll
        for (int q = 0; q < 8; ++q) if ((uint32_t)q == (bi & 7u)) --f[q];
      }
      --sum;
    }
    if (sum < kScale) {  // too few: the deficit to the largest (the lowest symbol on a tie)
      uint32_t bv = f[0], bi = k * 8;
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (f[q] > bv) { bv = f[q]; bi = k * 8 + q; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint32_t ov = __shfl_xor_sync(kFull, bv, o), oi = __shfl_xor_sync(kFull, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if ((bi >> 3) == k) {
#pragma unroll
        for (int q = 0; q < 8; ++q) if ((uint32_t)q == (bi & 7u)) f[q] += kScale - sum;
      }
    }
    uint32_t tot = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) tot += f[q];
    uint32_t c0 = warp_incl_scan(tot) - tot;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t sl = f[q] > 1 ? 32u - __clz(f[q] - 1u) : 1u;  // ceil(log2 f)
      fc[k * 8 + q] = f[q] | c0 << 13 | (sl - 1u) << 25;
      rcp[k * 8 + q] = f[q] > 1 ? (uint32_t)(((1ull << (31 + sl)) + f[q] - 1u) / f[q]) : 0u;
      A.freq[(size_t)g * 256 + k * 8 + q] = (uint16_t)f[q];
      c0 += f[q];
    }
    if (k == 0) red[0] = np;
  }
  __syncthreads();
  // lane k codes symbols k, k+64, ... last first, backwards into its scratch (src/codec.h:112-128)
  const uint32_t LC = lane_cap(A.B, s);
  uint8_t* end = A.lanes + (size_t)b * lanes_per_block(A.B) + lane_base(A.B, s) + (size_t)(k + 1) * LC;
  uint8_t* ptr = end;
  // output bytes go down from the lane's (16-byte aligned) end; they are gathered in acc, the first of its `pend` bytes
  // highest, and stored as aligned words
  uint64_t acc = 0;
  uint32_t pend = 0;
  uint32_t x = kRansLow;
  // The stream in chunks of kRansChunk symbols (a whole number of rounds of the 64 lanes), last chunk
  // first: the CTA stages a chunk in shared memory with coalesced loads, then lane k codes its symbols
  // c0 + k + 64 j of it, j descending -- the order of the whole-stream loop, without a global load on
  // the state's dependency chain.
  // (16-byte aligned streams: a chunk is loaded into registers while the one after it is coded)
  constexpr int kVecs = kRansChunk / 16 / kLanes;
  const bool al16 = ((uintptr_t)sym & 15u) == 0;
  const int32_t last = (int32_t)((ns - 1) / kRansChunk);
  uint4 ahead[kVecs];
  for (int32_t ch = last; ch >= 0; --ch) {
    const uint32_t c0 = (uint32_t)ch * kRansChunk, cn = min(kRansChunk, ns - c0);
    __syncthreads();  // (the previous chunk is coded)
    if (al16 && ch != last) {
#pragma unroll
      for (int j = 0; j < kVecs; ++j) reinterpret_cast<uint4*>(stage)[j * kLanes + k] = ahead[j];
    } else {
      const uint32_t n4 = ((uintptr_t)sym & 3u) == 0 ? cn >> 2 : 0u;
      for (uint32_t t = k; t < n4; t += kLanes)
        reinterpret_cast<uint32_t*>(stage)[t] = reinterpret_cast<const uint32_t*>(sym + c0)[t];
      for (uint32_t t = 4 * n4 + k; t < cn; t += kLanes) stage[t] = sym[c0 + t];
    }
    __syncthreads();
    if (al16 && ch > 0) {
#pragma unroll
      for (int j = 0; j < kVecs; ++j) ahead[j] = reinterpret_cast<const uint4*>(sym + c0 - kRansChunk)[j * kLanes + k];
    }
    if (k < cn) {
      // x' = (x / f) * 4096 + x % f + cum = x + cum + q * (4096 - f), with q = x / f by an exact
      // reciprocal: for x < 2^31 and s = ceil(log2 f), floor(x * ceil(2^(31+s) / f) / 2^(31+s)) = x / f
      // (the product's error is below x / 2^(31+s) < 2^-s <= 1/f, less than the gap to the next integer)
      // A symbol emits the state's low byte when it is at least f << 19, two when its upper bytes are too (never more:
      // x < 2^31).  Only that, the product and the sum are on the state's chain: the next symbol's table entries are
      // looked up before this one is coded.
      int32_t t = (int32_t)(k + (cn - 1 - k) / kLanes * kLanes);
      uint32_t e = fc[stage[t]], m = rcp[stage[t]];
      for (;;) {
        const uint32_t ce = e, cm = m;
        t -= (int32_t)kLanes;
        if (t >= 0) { e = fc[stage[t]]; m = rcp[stage[t]]; }
        const uint32_t f = ce & 0x1FFFu, xmax = f << (23 - kScaleBits + 8);
        const bool one = x >= xmax, two = x >> 8 >= xmax;
        const uint32_t b1 = x & 0xFFu, b2 = __byte_perm(x, 0, 0x4401);
        acc = two ? acc << 16 | b2 : one ? acc << 8 | b1 : acc;
        pend += (uint32_t)one + two;
        x = two ? x >> 16 : one ? x >> 8 : x;
        if (pend >= 4u) {
          pend -= 4u;
          ptr -= 4;
          *reinterpret_cast<uint32_t*>(ptr) = (uint32_t)(acc >> (8u * pend));
        }
        const uint32_t q = f == 1 ? x : __umulhi(x, cm) >> (ce >> 25);
        x += ((ce >> 13) & 0xFFFu) + q * (kScale - f);
        if (t < 0) break;
      }
    }
  }
  for (uint32_t i = pend; i > 0; --i) *--ptr = (uint8_t)(acc >> (8u * (i - 1u)));  // the bytes still gathered
  ptr -= 4;
  st32(ptr, x);
  const uint32_t ll = (uint32_t)(end - ptr);
  A.lanelen[(size_t)g * kLanes + k] = ll;
  const uint32_t lsum = warp_sum(ll);
  if (lane_id() == 0) red[1 + (k >> 5)] = lsum;
  __syncthreads();
  if (k == 0) {
    const uint32_t np = red[0];
    const uint32_t total = 32 + 2 * np + 4 * kLanes + red[1] + red[2];
    const uint32_t kind = total >= ns ? 0u : 1u;  // raw when rANS is not smaller (src/codec.h:130)
    info[0] = kind;
    info[1] = kind ? total : ns;
    info[2] = np;
    info[3] = ns;
  }
}

// ---------------------------------------------------------------- 6. the payload
// A CTA per (block, part): parts 0..4 are the streams' sections, part 5 the counts and the offset bits; each finds its
// place from the five sections' lengths.  Bytes are copied as aligned words (copy_in).  (One CTA per block, a byte a
// thread: 0.046 ms for one text block against 0.013, 0.39 for 1000 files against 0.10.)
__global__ void __launch_bounds__(256) k_enc_pack(EncArgs A) {
  const uint32_t b = blockIdx.x, s = blockIdx.y, tid = threadIdx.x;
  const uint32_t n = A.in_len[b];
  uint32_t* c = A.bcnt + b * 8;
  const uint32_t nob = c[3];
  uint64_t at = kHdrBytes, total = kHdrBytes + (uint64_t)nob;
  for (uint32_t k = 0; k < 5; ++k) {
    const uint32_t len = 5 + A.sinfo[(size_t)(b * 5 + k) * 4 + 1];
    if (k < s) at += len;
    total += len;
  }
  const bool stored = total >= n;  // (src/codec2.h:152, src/archive.h:394)
  uint8_t* o = A.slab + (size_t)b * A.B;
  if (s == 5) {
    if (tid == 0) { c[5] = stored ? n : (uint32_t)total; c[6] = stored ? 0 : 1; }
    if (stored) return;
    if (tid == 0) { st32(o, c[0]); st32(o + 4, c[1]); st32(o + 8, c[2]); st32(o + 12, nob); st32(o + 16, c[4]); }
    copy_in(o + at, A.s_bits + (size_t)b * bits_cap(A.B), nob, tid, 256);
    return;
  }
  if (stored) return;
  __shared__ uint32_t lofs[kLanes + 1];
  __shared__ uint32_t wcnt[8];
  const uint32_t g = b * 5 + s;
  const uint32_t* info = A.sinfo + (size_t)g * 4;
  const uint32_t kind = info[0], len = info[1], np = info[2], ns = info[3];
  uint8_t* d = o + at;
  if (tid == 0) { d[0] = (uint8_t)kind; st32(d + 1, len); }
  if (kind == 0) {
    copy_in(d + 5, stream_syms(A, b, s), ns, tid, 256);
    return;
  }
  const uint16_t* fq = A.freq + (size_t)g * 256;
  // present bitmap, then the frequencies of the present symbols in symbol order
  const uint32_t f = fq[tid];
  const uint32_t pres = f != 0;
  const unsigned bal = __ballot_sync(kFull, pres);
  if ((tid & 7u) == 0) d[5 + (tid >> 3)] = (uint8_t)((bal >> (tid & 31u)) & 0xFFu);
  if ((tid & 31u) == 0) wcnt[tid >> 5] = __popc(bal);
  const uint32_t* ll = A.lanelen + (size_t)g * kLanes;
  if (tid < 32) {
    const uint32_t a = ll[2 * tid], bb = ll[2 * tid + 1];
    const uint32_t inc = warp_incl_scan(a + bb);
    lofs[2 * tid] = inc - a - bb;
    lofs[2 * tid + 1] = inc - bb;
  }
  __syncthreads();
  uint32_t idx = __popc(bal & ((1u << (tid & 31u)) - 1u));
  for (uint32_t k = 0; k < (tid >> 5); ++k) idx += wcnt[k];
  if (pres) { d[5 + 32 + 2 * idx] = (uint8_t)f; d[5 + 32 + 2 * idx + 1] = (uint8_t)(f >> 8); }
  if (tid < kLanes) st32(d + 5 + 32 + 2 * np + 4 * tid, ll[tid]);
  const uint32_t data0 = 5 + 32 + 2 * np + 4 * kLanes;
  const uint32_t LC = lane_cap(A.B, s);
  const uint8_t* lb = A.lanes + (size_t)b * lanes_per_block(A.B) + lane_base(A.B, s);
  for (uint32_t jl = tid >> 5; jl < kLanes; jl += 8) {
    const uint32_t len_j = ll[jl];
    copy_in(d + data0 + lofs[jl], lb + (size_t)(jl + 1) * LC - len_j, len_j, lane_id(), 32);
  }
}

// ---------------------------------------------------------------- 7. record bodies back to back
__global__ void __launch_bounds__(1024) k_enc_scan(EncArgs A) {
  const uint32_t tid = threadIdx.x, nb = A.nb;
  const uint32_t per = (nb + 1023) / 1024;
  const uint32_t b0 = min(tid * per, nb), b1 = min(b0 + per, nb);
  uint64_t sum = 0;
  for (uint32_t b = b0; b < b1; ++b) {
    const uint32_t* c = A.bcnt + b * 8;
    sum += A.rec_hdr + (c[6] ? c[5] : (A.emit_stored ? A.in_len[b] : 0u));
  }
  __shared__ uint64_t ws[32];
  uint64_t incl = sum;
  const uint32_t l = lane_id();
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t t = __shfl_up_sync(kFull, incl, o);
    if (l >= (uint32_t)o) incl += t;
  }
  if (l == 31) ws[tid >> 5] = incl;
  __syncthreads();
  if (tid < 32) {
    uint64_t v = ws[tid], x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t t = __shfl_up_sync(kFull, x, o);
      if (l >= (uint32_t)o) x += t;
    }
    ws[tid] = x - v;
  }
  __syncthreads();
  uint64_t off = (A.rec_base ? *A.rec_base : 0ull) + ws[tid >> 5] + incl - sum;
  for (uint32_t b = b0; b < b1; ++b) {
    const uint32_t* c = A.bcnt + b * 8;
    const uint32_t method = c[6];
    const uint32_t len = method ? c[5] : A.in_len[b];
    off += A.rec_hdr;
    A.out_off[b] = off;
    A.out_len[b] = len;
    A.out_method[b] = (uint8_t)method;
    off += method ? len : (A.emit_stored ? len : 0u);
  }
  if (tid == 1023) *A.out_total = off;
}

__global__ void __launch_bounds__(256) k_enc_emit(EncArgs A) {
  const uint32_t b = blockIdx.x;
  const uint32_t method = A.bcnt[b * 8 + 6];
  if (!method && !A.emit_stored) return;
  const uint64_t off = A.out_off[b];
  const uint32_t len = A.out_len[b];
  if (off + len > A.out_cap) return;  // (the host checks out_total against out_cap)
  const uint8_t* s = method ? A.slab + (size_t)b * A.B : A.in + A.in_off[b];
  uint8_t* d = A.out + off;
  if (A.rec_hdr && threadIdx.x < 16) {  // the record header just before the body (off >= 16 here)
    const uint32_t t = threadIdx.x, w = t >> 2, sh = 8u * (t & 3u);
    const uint32_t v = w == 0 ? A.in_len[b] : w == 1 ? len : w == 2 ? method : A.rec_crc[b];
    d[(int)t - 16] = (w == 2 && t != 8) ? 0 : (uint8_t)(v >> sh);
  }
  uint32_t i = 0;
  if ((((uintptr_t)d ^ (uintptr_t)s) & 15u) == 0) {
    const uint32_t head = min(len, (uint32_t)((16u - ((uintptr_t)d & 15u)) & 15u));
    if (threadIdx.x < head) d[threadIdx.x] = s[threadIdx.x];
    i = head;
    const uint32_t nvec = (len - i) / 16;
    for (uint32_t v = threadIdx.x; v < nvec; v += blockDim.x)
      reinterpret_cast<uint4*>(d + i)[v] = reinterpret_cast<const uint4*>(s + i)[v];
    i += nvec * 16;
  } else {
    // not co-aligned (every record of an archive): 4-byte words stored aligned at d, each built by a funnel
    // shift from the two aligned source words that cover it (those reach at most 3 bytes past the body,
    // inside the input's slack or the slab's padding)
    const uint32_t head = min(len, (uint32_t)((4u - ((uintptr_t)d & 3u)) & 3u));
    if (threadIdx.x < head) d[threadIdx.x] = s[threadIdx.x];
    i = head;
    const uint32_t nw = (len - i) >> 2, sh = (uint32_t)((uintptr_t)(s + i) & 3u);
    const uint32_t* sw = reinterpret_cast<const uint32_t*>(s + i - sh);
    uint32_t* dw = reinterpret_cast<uint32_t*>(d + i);
    if (sh == 0) {
      for (uint32_t w = threadIdx.x; w < nw; w += blockDim.x) dw[w] = sw[w];
    } else {
      for (uint32_t w = threadIdx.x; w < nw; w += blockDim.x) dw[w] = __funnelshift_r(sw[w], sw[w + 1], 8u * sh);
    }
    i += nw * 4;
  }
  for (uint32_t k = i + threadIdx.x; k < len; k += blockDim.x) d[k] = s[k];
}

cudaError_t prepare_kernels() {  // with the device current, once per context
  cudaError_t e = cudaFuncSetAttribute(k_enc_parse<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, 512 / 32 * sizeof(Finish));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_enc_parse<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 / 32 * sizeof(Finish));
  return e == cudaSuccess ? prepare_fill() : e;
}

void launch_encode(const EncArgs& A, const CrcArgs& crc_in, cudaStream_t st, Stages& S) {
  if (!A.nb) return;
  launch_crc(crc_in, st, S, "k_crc_in");
  const dim3 sg((A.B + kSortTile - 1) / kSortTile, A.nb);
  const uint32_t scan_threads = sg.x > 16 ? 256 * kScanParts : 256;
  S.begin("k_sort_count", st);
  k_sort_count<0><<<sg, 256, 0, st>>>(A);
  S.end(st);
  S.begin("k_sort_scan", st);
  k_sort_scan<<<A.nb, scan_threads, 0, st>>>(A);
  S.end(st);
  S.begin("k_sort_scatter", st);
  k_sort_scatter<0><<<sg, kSortThreads, 0, st>>>(A);
  S.end(st);
  S.begin("k_sort_count", st);
  k_sort_count<1><<<sg, 256, 0, st>>>(A);
  S.end(st);
  S.begin("k_sort_scan", st);
  k_sort_scan<<<A.nb, scan_threads, 0, st>>>(A);
  S.end(st);
  S.begin("k_sort_scatter", st);
  k_sort_scatter<1><<<sg, kSortThreads, 0, st>>>(A);
  S.end(st);
  S.begin("k_enc_chain", st);
  k_enc_chain<<<dim3((A.B + kChainTile - 1) / kChainTile, A.nb), 256, 0, st>>>(A);
  S.end(st);
  S.begin("k_enc_walk", st);
  // Walks a warp: 32, or fewer while the launch has too few for every SM's 32 warps; a step takes as long as the chains
  // of its warp's walks together.  ms with 32 / 16 / 8 / 4 / 2: one block of text 0.38 / 0.25 / 0.17 / 0.13 / 0.12,
  // 16 blocks 0.41 / 0.29 / 0.22 / 0.21 / 0.32, 64 blocks 0.57 / 0.50 / 0.54 / 0.66 / 1.03, 128 blocks 0.82 / 0.87 /
  // 0.95 / 1.2 / 1.9.
  uint32_t walks = 32;
  while (walks > 2 && 2 * (A.nb * A.nseg / walks) <= 148 * 32) walks /= 2;
  k_enc_walk<<<A.nb * (A.nseg / walks) / 2, 64, 0, st>>>(A, walks);
  S.end(st);
  S.begin("k_enc_parse", st);
  const size_t fin = A.nseg / 32 * sizeof(Finish);
  if (A.nseg == 256) k_enc_parse<256><<<A.nb, 256, fin, st>>>(A);
  else if (A.nseg == 512) k_enc_parse<512><<<A.nb, 512, fin, st>>>(A);
  else k_enc_parse<1024><<<A.nb, 1024, fin, st>>>(A);
  S.end(st);
  S.begin("k_enc_streams", st);
  // A tile's barriers and the walk over its warps cost the same for any width, so a block is faster in wide tiles and a
  // full GPU in narrow ones.  ms with 32 / 16 / 8 warps: one text block 0.076 / 0.101 / 0.166, 64 MiB of text (256
  // blocks) 0.24 / 0.19 / 0.29, 256 blocks of 1 MiB 0.43 / 0.36 / 0.58, 1 GiB of lz_mix (4096 blocks) 1.56 / 1.24 /
  // 0.82.  (One warp a block, 32 tokens a round: 0.64, 1.09, 2.56 and 0.87.)
  if (A.nb <= 148) k_enc_streams<32><<<A.nb, 1024, 0, st>>>(A);
  else if (A.nb <= 3 * 148) k_enc_streams<16><<<A.nb, 512, 0, st>>>(A);
  else k_enc_streams<8><<<A.nb, 256, 0, st>>>(A);
  S.end(st);
  S.begin("k_enc_rans", st);
  k_enc_rans<<<dim3(A.nb, 5), 64, 0, st>>>(A);
  S.end(st);
  S.begin("k_enc_pack", st);
  k_enc_pack<<<dim3(A.nb, 6), 256, 0, st>>>(A);
  S.end(st);
  S.begin("k_enc_scan", st);
  k_enc_scan<<<1, 1024, 0, st>>>(A);
  S.end(st);
  S.begin("k_enc_emit", st);
  k_enc_emit<<<A.nb, 256, 0, st>>>(A);
  S.end(st);
}

}  // namespace zc
