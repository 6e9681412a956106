// zc_decode_fill.cu -- the ZB2 LZ replay in two kernels (src/codec2.h:155-203):
//
//   k_dec_tokens  one CTA per block: every token's literal run and match length (ext
//                 bytes), offset (offset bits), output start and literal start, from block-wide scans, in
//                 parallel over the tokens; which token holds each 128-byte line's first byte; then the groups
//                 (a scan of their counts) and the recent-offset symbols (each names an earlier token's offset,
//                 src/codec2.h:180-192), resolved by pointer jumping within each tile.  Every check of the reference
//                 decoder is made here; a failing one records a status and the block is not replayed.
//   k_dec_fill    one warp per block: fills the block in rounds of 128 output bytes (a 4-byte word a lane)
//                 straight through, group boundaries or not: a byte whose source lies earlier in the same
//                 round is read from the round's staged bytes once known; the token table is a 64-row ring in
//                 shared memory, refilled 32 tokens at a time from registers loaded one window ahead.
//   k_dec_fill_multi  the same with several warps a block, a line each, for launches of few blocks: words wait for
//                 their source words, which are published in shared memory.
// Stored blocks are copied by the fill.  The rANS streams come from k_dec_streams (zc_decode.cu).
#include <algorithm>
#include <type_traits>

#include "zc_internal.cuh"
#include "zc_kernels.h"

namespace zc {

namespace {

__device__ __forceinline__ void flag(uint32_t* err, uint32_t b, uint32_t code) { atomicCAS(err + b, 0u, code); }

// Scans over a CTA of 32 NW threads with one barrier each: every warp scans all the warps' totals for itself, and a
// scan's totals lie in the row of ws that the scan before it did not use, so none can still be read when they are
// written.
template <uint32_t NW>
struct CtaScan {
  uint64_t (*sums)[NW];
  uint32_t (*maxs)[NW];
  uint32_t row = 0;
  __device__ CtaScan(uint64_t (*s)[NW], uint32_t (*m)[NW]) : sums(s), maxs(m) {}
  // the sum over the threads before this one (`total`: over all), and the maximum of `top` over them
  __device__ __forceinline__ uint64_t operator()(uint64_t v, uint64_t& total, uint32_t top, uint32_t& top_before,
                                                 uint32_t& top_all) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint64_t inc = v;
    uint32_t mx = top;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(kFull, inc, o);
      const uint32_t z = __shfl_up_sync(kFull, mx, o);
      if (lane >= o) { inc += y; mx = max(mx, z); }
    }
    if (lane == 31) { sums[row][w] = inc; maxs[row][w] = mx; }
    __syncthreads();
    const uint64_t x = lane < NW ? sums[row][lane] : 0ull;
    const uint32_t xm = lane < NW ? maxs[row][lane] : 0u;
    uint64_t xi = x;
    uint32_t mi = xm;
#pragma unroll
    for (uint32_t o = 1; o < NW; o <<= 1) {
      const uint64_t y = __shfl_up_sync(kFull, xi, o);
      const uint32_t z = __shfl_up_sync(kFull, mi, o);
      if (lane >= o) { xi += y; mi = max(mi, z); }
    }
    row ^= 1u;
    total = __shfl_sync(kFull, xi, NW - 1);
    top_all = __shfl_sync(kFull, mi, NW - 1);
    const uint32_t warps = __shfl_sync(kFull, mi, w ? w - 1u : 0u), up = __shfl_up_sync(kFull, mx, 1);
    top_before = max(w ? warps : 0u, lane ? up : 0u);
    return __shfl_sync(kFull, xi - x, w) + inc - v;
  }
  __device__ __forceinline__ uint64_t operator()(uint64_t v, uint64_t& total) {
    uint32_t a, b;
    return (*this)(v, total, 0u, a, b);
  }
};

constexpr uint32_t kRepMark = 0x80000000u;  // a recent-offset symbol not resolved yet: kRepMark | the token it names

// A token's row: its output start and its literals' start before it (21 bits each: start - literal start is never
// negative), and its literal count (21 bits, split over the two words' upper bits).
__device__ __forceinline__ uint2 tok_row(uint32_t start, uint32_t lits, uint32_t lit0) {
  return make_uint2((start & 0x1FFFFFu) | lits << 21, ((start - lit0) & 0x1FFFFFu) | lits >> 11 << 21);
}
__device__ __forceinline__ uint32_t row_start(const uint2& r) { return r.x & 0x1FFFFFu; }
__device__ __forceinline__ uint32_t row_back(const uint2& r) { return r.y & 0x1FFFFFu; }  // start - literal start
__device__ __forceinline__ uint32_t row_lits(const uint2& r) { return r.x >> 21 | r.y >> 21 << 11; }

// `n` <= 26 bits from bit `at` of p on, from the one or two aligned words that hold them
__device__ __forceinline__ uint32_t bits_at(const uint8_t* p, uint32_t at, uint32_t n) {
  const uint8_t* q = p + (at >> 3);
  const uint32_t sh = (uint32_t)(uintptr_t)q & 3u, from = 8u * sh + (at & 7u);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(q - sh);
  uint64_t v = __ldg(w);
  if (from + n > 32u) v |= (uint64_t)__ldg(w + 1) << 32;
  return (uint32_t)(v >> from) & ((1u << n) - 1u);
}

}  // namespace

// A CTA of 512 threads per block, 2048 tokens a tile, four consecutive ones a thread (one load for their four bytes of
// a stream, vector stores for their rows).  A tile is a chain of loads and barriers whatever its size: its streams'
// bytes, the scan that places its ext bytes and offset bits, those, the scan that places its literals and output, and
// the offsets that its recent-offset symbols name.  (One token a thread, groups and recent offsets in passes of their
// own over the block's tokens in global memory: 0.49 ms per GiB of lz_mix at block 18 against 0.33, one text block 0.058
// against 0.037.)
//
// Recent offsets (src/codec2.h:179-199): symbol r of a group whose first token is gs names the offset of token
// gs - 1 - r (the last three offsets before the group, nearest first), or the initial 1, 4, 8 when r >= gs.  The group
// counts' scan sets a bit for each group's first token; the maximum of those up to a token is its gs.  A token named
// in an earlier tile is resolved; within the tile, by pointer jumping in shared memory (a chain halves each round).
//
// Many near copies make one long chain of the output if hardly a literal or hardly a farther copy ends it.  Several warps
// only hand such a chain's words to one another, 0.4 to 0.9 us a hop, so the block's line table says in its last row that
// one warp is to fill it.  ms shared / by one warp, one block of 256 KiB and 256: two values at random at level 1, 13
// near copies a 128-byte line and 3.2 hops, 5.53 / 2.65 and 7.42 / 3.01, at level 5, 4 a line and one hop, 1.74 / 1.83 and
// 2.44 / 2.13; four symbols at level 1, 2.4 a line, 0.92 / 2.01 and 1.36 / 2.51: so the line lies at 8.  Counters 8
// bytes apart at level 1, 16 a line, none farther and 14 hops, 10.5 / 8.0 and 16.4 / 8.5; at level 5, where one in twelve is
// farther and there are 0.6 hops, 0.96 / 5.5 and 1.55 / 5.9.  (Others pay 1 % of this kernel and 0.5 % of the fill for it.)
constexpr uint32_t kNearOffset = 128, kNearBytes = 16;  // more than one copy from at most 128 back in 16 bytes
constexpr uint32_t kTokThreads = 512, kTokPer = 4, kTokTile = kTokThreads * kTokPer;

__global__ void __launch_bounds__(kTokThreads, 2) k_dec_tokens(DecArgs A) {
  constexpr uint32_t NW = kTokThreads / 32;
  const uint32_t b = blockIdx.x, tid = threadIdx.x;
  if (A.method[b] != 1 || A.raw_len[b] > A.B || A.err[b]) return;
  __shared__ uint64_t sums[2][NW];
  __shared__ uint32_t maxs[2][NW];
  __shared__ uint32_t gbits[(1u << kMaxBlockLog) / 4 / 32 + 1];  // a bit for each group's first token
  __shared__ __align__(16) uint32_t jump[kTokTile];
  __shared__ uint32_t nears;
  const DecMeta m = A.meta[b];
  const uint32_t raw = A.raw_len[b], B = A.B;
  const size_t TC = tok_cap(B), EC = ext_cap(B);
  const uint32_t* tok = reinterpret_cast<const uint32_t*>(A.s_tok + (size_t)b * TC);  // (four symbols a word)
  const uint32_t* sym = reinterpret_cast<const uint32_t*>(A.s_sym + (size_t)b * TC);
  const uint32_t* grp = reinterpret_cast<const uint32_t*>(A.s_grp + (size_t)b * TC);
  const uint8_t* ext = A.s_ext + (size_t)b * EC;
  const uint8_t* bits = A.comp + A.comp_off[b] + m.bits_off;
  const uint64_t nbits = 8ull * m.nob;
  uint2* Tp = A.tk_pos + (size_t)b * TC;
  uint32_t* Td = A.tk_d + (size_t)b * TC;
  uint2* line = A.line ? A.line + (size_t)b * line_cap(B) : nullptr;  // (none for one warp a block)
  const uint32_t al = (uint32_t)(uintptr_t)(A.out + A.out_off[b]) & 127u;  // output byte q lies in line (q + al) / 128
  bool bad = false;
  CtaScan<NW> scan(sums, maxs);
  uint64_t sum;
  if (line)
    for (uint32_t k = tid; k < (raw + al + 127u) >> 7; k += kTokThreads) line[k] = make_uint2(0, 0);
  for (uint32_t k = tid; k < (m.nt >> 5) + 1; k += kTokThreads) gbits[k] = 0;
  if (tid == 0) nears = 0;
  __syncthreads();
  // ---- the groups' first tokens
  {
    uint32_t at = 0;
    for (uint32_t g0 = 0; g0 < m.ng; g0 += kTokTile) {
      const uint32_t g = g0 + kTokPer * tid, c4 = g < m.ng ? grp[g >> 2] : 0u;
      uint32_t c[kTokPer], mine = 0;
#pragma unroll
      for (uint32_t j = 0; j < kTokPer; ++j) {
        c[j] = g + j < m.ng ? c4 >> 8 * j & 0xFFu : 0u;
        mine += c[j];
      }
      uint32_t s = at + (uint32_t)scan(mine, sum);
#pragma unroll
      for (uint32_t j = 0; j < kTokPer; ++j) {
        if (g + j < m.ng) {
          if (c[j] == 0 || s + c[j] > m.nt) bad = true;  // (at most 2^20 counts of at most 255)
          else atomicOr(&gbits[s >> 5], 1u << (s & 31u));
        }
        s += c[j];
      }
      at += (uint32_t)sum;
    }
    if (at != m.nt) bad = true;
  }
  __syncthreads();
  // ---- the tokens
  uint32_t ei = 0, bp = 0, op = 0, li = 0, carry = 0, near = 0;
  uint32_t ntv = 0, nsv = 0;  // the next tile's tokens and symbols
  if (kTokPer * tid < m.nt) { ntv = tok[tid]; nsv = sym[tid]; }
  for (uint32_t t0 = 0; t0 < m.nt; t0 += kTokTile) {
    const uint32_t t = t0 + kTokPer * tid;  // the thread's first token
    const uint32_t n = t < m.nt ? min(kTokPer, m.nt - t) : 0u;
    const uint32_t tv4 = ntv, sv4 = nsv;
    ntv = 0; nsv = 0;
    if (t + kTokTile < m.nt) { ntv = tok[(t + kTokTile) >> 2]; nsv = sym[(t + kTokTile) >> 2]; }
    const uint32_t starts = n ? gbits[t >> 5] >> (t & 31u) & ((1u << n) - 1u) : 0u;
    uint32_t mine = 0;  // ext bytes | offset bits << 16 of the thread (each part of a tile's sum fits 16 bits)
#pragma unroll
    for (uint32_t j = 0; j < kTokPer; ++j) {
      if (j >= n) continue;
      const uint32_t tv = tv4 >> 8 * j & 0xFFu, sv = sv4 >> 8 * j & 0xFFu;
      if (sv > 19u && (sv < kSymRep || sv > kSymRep + 2)) bad = true;
      mine += ((tv >> 4) == 15u ? 3u : 0u) + ((tv & 15u) == 15u ? 2u : 0u) + (sv <= 19u ? sv << 16 : 0u);
    }
    uint32_t gbefore, gall;
    const uint32_t pre = (uint32_t)scan(mine, sum, starts ? t + 31u - __clz(starts) : 0u, gbefore, gall);
    uint32_t xq = ei + (pre & 0xFFFFu), bq = bp + (pre >> 16);
    ei += (uint32_t)sum & 0xFFFFu;
    bp += (uint32_t)sum >> 16;
    uint32_t L[kTokPer], M[kTokPer], D[kTokPer];
    uint64_t len = 0;  // literals, and output << 32 (a sum past 32 bits only where a token is bad by itself)
#pragma unroll
    for (uint32_t j = 0; j < kTokPer; ++j) {
      L[j] = 0; M[j] = 0; D[j] = 0;
      if (j >= n) continue;
      const uint32_t tv = tv4 >> 8 * j & 0xFFu, sv = sv4 >> 8 * j & 0xFFu;
      const uint32_t fl = (tv >> 4) == 15u, fm = (tv & 15u) == 15u, nx = 3u * fl + 2u * fm, nbit = sv <= 19u ? sv : 0u;
      if ((uint64_t)xq + nx > m.ne || (uint64_t)bq + nbit > nbits) bad = true;
      L[j] = tv >> 4;
      M[j] = (tv & 15u) + 4u;
      if (!bad) {
        if (fl) L[j] += (uint32_t)ext[xq] | (uint32_t)ext[xq + 1] << 8 | (uint32_t)ext[xq + 2] << 16;
        if (fm) { const uint32_t q = xq + 3u * fl; M[j] += (uint32_t)ext[q] | (uint32_t)ext[q + 1] << 8; }
        if (sv < kSymRep) {
          D[j] = (1u << sv) + (nbit ? bits_at(bits, bq, nbit) : 0u);
        } else {
          const uint32_t own = starts & (2u << j) - 1u, r = sv - kSymRep;
          const uint32_t gs = own ? t + 31u - __clz(own) : max(carry, gbefore);
          D[j] = r < gs ? kRepMark | (gs - 1u - r) : r - gs == 0 ? 1u : r - gs == 1 ? 4u : 8u;
          if (r < gs && gs - 1u - r < t0) D[j] = Td[gs - 1u - r];
        }
      }
      xq += nx;
      bq += nbit;
      len += (uint64_t)(L[j] + M[j]) << 32 | L[j];
    }
    carry = max(carry, gall);
    *reinterpret_cast<uint4*>(&jump[kTokPer * tid]) = make_uint4(D[0], D[1], D[2], D[3]);
    const uint64_t at = scan(len, sum);  // (its barrier also publishes jump)
    uint32_t opk = op + (uint32_t)(at >> 32), lik = li + (uint32_t)at;
    op += (uint32_t)(sum >> 32);
    li += (uint32_t)sum;
    uint2 row[kTokPer];
    uint32_t ms[kTokPer];
#pragma unroll
    for (uint32_t j = 0; j < kTokPer; ++j) {
      row[j] = tok_row(opk, L[j], lik);
      ms[j] = opk + L[j];
      if (j >= n) continue;
      if ((uint64_t)lik + L[j] > m.nl || (uint64_t)opk + L[j] + M[j] > raw) bad = true;
      const uint32_t end = opk + L[j] + M[j];
      if (line && !bad) {  // the lines whose first byte the token holds, and its own start inside a line
        for (uint32_t k = (opk + al + 127u) >> 7; k < (end + al + 127u) >> 7; ++k) line[k].x = t + j;
        if (t + j && ((opk + al) & 127u)) atomicOr(&line[(opk + al) >> 7].y, 1u << ((opk + al) >> 2 & 31u));
      }
      opk = end;
      lik += L[j];
    }
    for (;;) {  // (every thread has read jump before any writes it again)
      uint32_t more = 0;
#pragma unroll
      for (uint32_t j = 0; j < kTokPer; ++j) {
        if (D[j] & kRepMark) D[j] = jump[(D[j] & ~kRepMark) - t0];
        more |= D[j] & kRepMark;
      }
      if (!__syncthreads_or(more)) break;
      *reinterpret_cast<uint4*>(&jump[kTokPer * tid]) = make_uint4(D[0], D[1], D[2], D[3]);
      __syncthreads();
    }
    if (n) {
#pragma unroll
      for (uint32_t j = 0; j < kTokPer; ++j)
        if (j < n) {
          if (D[j] == 0 || D[j] > ms[j]) bad = true;
          near += D[j] <= kNearOffset;
        }
      *reinterpret_cast<uint4*>(Tp + t) = make_uint4(row[0].x, row[0].y, row[1].x, row[1].y);
      *reinterpret_cast<uint4*>(Tp + t + 2) = make_uint4(row[2].x, row[2].y, row[3].x, row[3].y);
      *reinterpret_cast<uint4*>(Td + t) = make_uint4(D[0], D[1], D[2], D[3]);
    }
  }
  near = warp_sum(near);
  if (lane_id() == 0) atomicAdd(&nears, near);
  const int any_bad = __syncthreads_or(bad);
  if (tid == 0) {
    Tp[m.nt] = tok_row(op, raw - op, li);  // token nt: the literal tail
    Td[m.nt] = 1;
    if (any_bad || op + (m.nl - li) != raw) flag(A.err, b, E_TOKEN);
    A.meta[b].op_total = op;
    A.meta[b].li_total = li;
    if (line)
      line[line_cap(B) - 1].x = nears > raw / kNearBytes && (m.nl <= raw / kNearBytes || m.nt - nears <= nears / 64);
  }
  if (line && !any_bad && op < raw) {  // the literal tail's lines and start (a line 0 that starts before the output: token 0)
    for (uint32_t k = ((op + al + 127u) >> 7) + tid; k < (raw + al + 127u) >> 7; k += kTokThreads) line[k].x = m.nt;
    if (tid == 0 && op && ((op + al) & 127u)) atomicOr(&line[(op + al) >> 7].y, 1u << ((op + al) >> 2 & 31u));
  }
}

namespace {

// The warp's token table: a ring of TR rows, token t in row t % TR.  start = the token's output start;
// tk = {match start, literal start - output start (mod 2^32), offset D, the reciprocal ceil(2^32 / D)
// for D >= 2 (0 for D = 1)}.  Token nt (one past the last) is the block's literal tail: it starts where
// the tokens' output ends and is literals up to the block's end; later rows start at kNoToken.
constexpr uint32_t kNoToken = 0x7FFFFFFFu;
template <uint32_t TR>
struct FillTable {
  uint32_t start[TR];
  uint4 tk[TR];
};
// per warp, for WPL output words a lane a round: the table's rows (a round's tokens and the one carried
// in), its bytes, and the round's staged bytes
__host__ __device__ constexpr uint32_t fill_rows(uint32_t wpl) { return 64 * wpl; }
__host__ __device__ constexpr uint32_t fill_table_bytes(uint32_t wpl) { return 20 * fill_rows(wpl); }
__host__ __device__ constexpr uint32_t fill_stage_bytes(uint32_t wpl) { return 256 * wpl; }

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// thread l of nth copies its share; no overlap
__device__ inline void copy_bytes(uint8_t* d, const uint8_t* s, uint32_t n, uint32_t l, uint32_t nth) {
  uint32_t i = 0;
  if ((((uintptr_t)d ^ (uintptr_t)s) & 15u) == 0) {
    const uint32_t head = (uint32_t)((16u - ((uintptr_t)d & 15u)) & 15u);
    if (l < head && l < n) d[l] = s[l];
    i = head < n ? head : n;
    for (uint32_t j = i + 16 * l; j + 16 <= n; j += 16 * nth)
      *reinterpret_cast<uint4*>(d + j) = *reinterpret_cast<const uint4*>(s + j);
    i += (n - i) & ~15u;
  }
  for (uint32_t j = i + l; j < n; j += nth) d[j] = s[j];
}

}  // namespace

// The replay of block b by one warp, in rounds of 128 * WPL output bytes: WPL 128-byte lines of the output
// address, lane k filling the aligned word at offset 4k of each.  Groups are not walked: a byte's value
// comes from its token's literals, from output before the round (the warp's shared-memory ring of the last
// R bytes, or global memory), or from an earlier byte of the same round.  The lanes first fill every byte
// of the first two kinds with their loads in flight together; the bytes of the third kind then read their
// sources from the round's bytes, staged 16 bits each, pass after pass until all are known (each source lies
// before its byte, so this ends; the format's groups keep those chains short).
//
// Bound by instruction issue, so the work of a byte is kept short: a round that lies wholly inside the block tests no
// bounds, ring loads are apart from loads of literals and far output (one generic load made the ring's slower), a
// byte's source stays as it was computed, and a staged byte carries its own flag.  lz_mix, 1 GiB, block 18: 3.69 ms
// with packed sources, bounds, generic loads and a flag array; 2.85 ms now.
//
// A token is at least 4 bytes long, so an aligned word holds at most one token start: a line's token
// starts form a 32-bit word mask (one OR-reduction), and a lane's bytes belong to the last token starting at
// or before its word's last byte, or the one before that.  A match byte's source is ms - D + ((q - ms) mod
// D) (src/codec2.h:194-197: an overlapping match repeats its D bytes before it), the quotient from a
// multiply-high by the reciprocal, exact to one step, which a compare corrects.
template <uint32_t WPL, uint32_t TR>
__device__ __forceinline__ void fill_block(const DecArgs& A, uint32_t b, FillTable<TR>& T, uint8_t* ring, uint32_t R,
                                           uint16_t* stage) {
  const uint32_t rmask = R - 1u;
  const uint32_t lane = lane_id();
  const uint32_t raw = A.raw_len[b], method = A.method[b], clen = A.comp_len[b], B = A.B;
  uint8_t* o = A.out + A.out_off[b];
  const uint8_t* p = A.comp + A.comp_off[b];
  if (raw > B) { if (lane == 0) flag(A.err, b, E_RAWLEN); return; }
  if (method == 0) {
    if (clen != raw) { if (lane == 0) flag(A.err, b, E_STORED); return; }
    copy_bytes(o, p, raw, lane, 32);
    return;
  }
  if (method != 1) { if (lane == 0) flag(A.err, b, E_METHOD); return; }
  if (A.err[b]) return;
  const DecMeta& m = A.meta[b];
  const uint32_t nt = m.nt, op_total = m.op_total, li_total = m.li_total;
  const size_t TC = tok_cap(B);
  const uint8_t* lit = A.s_lit + (size_t)b * B;
  const uint2* Tp = A.tk_pos + (size_t)b * TC;
  const uint32_t* Td = A.tk_d + (size_t)b * TC;
  const uint32_t ob = (uint32_t)(uintptr_t)o;
  // rows for tokens committed so far: [loaded - TR, loaded); row TR - 1 first holds a token "-1" (no byte
  // uses it).  The next 32 tokens wait in registers (lane k: token loaded + k), fetched one window ahead;
  // a match whose source lies beyond the ring has its first source lines brought into L2 then, and so
  // does each token's first literal line.
  uint32_t loaded = 0, ns, nm, nd, nl;
  auto fetch = [&](uint32_t base) {
    const uint32_t t = base + lane;
    ns = kNoToken; nm = kNoToken; nd = 1; nl = 0;
    if (t < nt) {
      const uint2 r = Tp[t];
      nd = Td[t];
      ns = row_start(r); nm = ns + row_lits(r); nl = 0u - row_back(r);
      prefetch_l2(lit + (ns + nl));
      if (nd >= R) {
        prefetch_l2(o + (nm - nd));
        prefetch_l2(o + (nm - nd) + 128);
      }
    } else if (t == nt) {
      ns = op_total; nm = raw; nl = li_total - op_total;
    }
  };
  auto commit = [&]() {
    const uint32_t t = loaded + lane;
    T.start[t % TR] = ns;
    T.tk[t % TR] = make_uint4(nm, nl, nd, nd >= 2 ? 0xFFFFFFFFu / nd + 1u : 0u);
    loaded += 32;
    fetch(loaded);
  };
  fetch(0);
  if (lane == 0) T.start[TR - 1] = 0;
  commit();
  __syncwarp();
  uint32_t before = 0;  // tokens starting before the round
  const uint32_t upto = 0xFFFFFFFFu >> (31u - lane);
  for (int32_t lb = -(int32_t)(ob & 127u); lb < (int32_t)raw; lb += 128 * WPL) {
    if (before + 32 * WPL > loaded) {  // (at most 32 tokens start in a line; the carried one keeps its row)
      do commit(); while (before + 32 * WPL > loaded);
      __syncwarp();
    }
    const int32_t rlo = lb - (int32_t)R;  // the ring holds output [lb - R, lb)
    uint32_t w[WPL], pend = 0;            // pend: bit 4h + j, byte j of word h is not known yet
    uint32_t srcs[WPL][4];                // its source
    uint32_t bh = before;
#pragma unroll
    for (uint32_t h = 0; h < WPL; ++h) {
      const int32_t lh = lb + 128 * (int32_t)h;
      const uint32_t ts = T.start[(bh + lane) % TR];
      const int32_t rel = (int32_t)(ts - (uint32_t)lh);
      const uint32_t mask = __reduce_or_sync(kFull, (uint32_t)rel < 128u ? 1u << (rel >> 2) : 0u);
      const uint32_t t1 = bh + __popc(mask & upto) - 1u, t0 = t1 - 1u;  // (mod 2^32: token -1 is row TR - 1)
      const uint32_t st1 = T.start[t1 % TR], st0 = T.start[t0 % TR];
      const uint4 a1 = T.tk[t1 % TR], a0 = T.tk[t0 % TR];
      bh += __popc(mask);
      const int32_t q0 = lh + 4 * (int32_t)lane;
      w[h] = 0;
      auto bytes = [&](auto whole) {
        constexpr bool inside = decltype(whole)::value;
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // every choice a select, the load predicated
          const int32_t qi = q0 + j;
          const bool valid = inside || (qi >= 0 && qi < (int32_t)raw);
          const uint32_t q = (uint32_t)qi;
          const bool hi = q >= st1;
          const uint32_t opk = hi ? st1 : st0, ms = hi ? a1.x : a0.x, ld = hi ? a1.y : a0.y, D = hi ? a1.z : a0.z,
                         mg = hi ? a1.w : a0.w;
          const uint32_t x = q - ms;
          uint32_t r = x - __umulhi(x, mg) * D;
          r = (int32_t)r < 0 ? r + D : r;
          r = mg ? r : 0u;
          const uint32_t s = q >= ms ? ms - D + r : q;
          const bool own = s >= opk;
          const bool inr = !own && (int32_t)s >= lb;
          const bool near = !own && (int32_t)s >= rlo;
          const uint8_t* src = (own ? lit : o) + (own ? s + ld : s);
          const bool take = valid && inr;
          pend |= (uint32_t)take << (4 * h + j);
          srcs[h][j] = s;
          uint32_t v = 0;
          if (valid && !near) v = *src;
          if (valid && near && !inr) v = ring[(ob + s) & rmask];
          w[h] |= v << (8 * j);
        }
      };
      if (lh >= 0 && lh + 128 <= (int32_t)raw) bytes(std::true_type{}); else bytes(std::false_type{});
    }
    // bytes from earlier in the round: the round's bytes staged, 16 bits each, bit 8 set while one is not known; each
    // pass takes the bytes whose sources are known
    __syncwarp();  // (every lane's loads from the ring come before any lane's stores into it)
    if (__any_sync(kFull, pend)) {
      for (;;) {
#pragma unroll
        for (uint32_t h = 0; h < WPL; ++h) {
          const uint32_t f = (pend >> (4 * h)) & 15u;  // (bits 0, 1 to bits 8, 24, then bits 2, 3)
          const uint32_t lo = __byte_perm(w[h], 0, 0x4140) | ((f & 3u) * 0x00800100u & 0x01000100u);
          const uint32_t hi = __byte_perm(w[h], 0, 0x4342) | ((f >> 2) * 0x00800100u & 0x01000100u);
          *reinterpret_cast<uint2*>(stage + 128 * h + 4 * lane) = make_uint2(lo, hi);
        }
        __syncwarp();
        uint32_t left = pend;
#pragma unroll
        for (uint32_t h = 0; h < WPL; ++h) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (!((pend >> (4 * h + j)) & 1u)) continue;
            const uint32_t c = stage[srcs[h][j] - (uint32_t)lb];
            if (c >> 8) continue;
            w[h] |= c << (8 * j);
            left &= ~(1u << (4 * h + j));
          }
        }
        pend = left;
        __syncwarp();
        if (!__any_sync(kFull, pend)) break;
      }
    }
    // stores: the ring always whole words; the output whole words inside the block, bytes at its edges
#pragma unroll
    for (uint32_t h = 0; h < WPL; ++h) {
      const int32_t q0 = lb + 128 * (int32_t)h + 4 * (int32_t)lane;
      *reinterpret_cast<uint32_t*>(ring + ((ob + (uint32_t)q0) & rmask)) = w[h];
      if (q0 >= 0 && q0 + 4 <= (int32_t)raw) {
        *reinterpret_cast<uint32_t*>(o + q0) = w[h];
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (q0 + j >= 0 && q0 + j < (int32_t)raw) o[q0 + j] = (uint8_t)(w[h] >> (8 * j));
      }
    }
    before = bh;
    __syncwarp();
  }
}

// Fed by a device work queue: every warp takes the next block from the work counter until none is left,
// so blocks of uneven sizes (a batch of many files) balance across warps.  A CTA holds blockDim.x / 32
// warps, each with its table, a ring of 2^ring_log bytes and its staged bytes in dynamic shared memory.
// The ring is read only at positions the warp has written in its current block.
template <uint32_t WPL>
__global__ void __maxnreg__(72) k_dec_fill(DecArgs A) {  // (72 registers: 28 warps an SM with 4-warp CTAs)
  constexpr uint32_t TR = fill_rows(WPL);
  extern __shared__ __align__(16) uint8_t fsm[];
  const uint32_t R = 1u << A.ring_log;
  const uint32_t wid = threadIdx.x >> 5;
  const size_t per = (size_t)fill_table_bytes(WPL) + R + fill_stage_bytes(WPL);
  uint8_t* mine = fsm + (size_t)wid * per;
  FillTable<TR>& T = *reinterpret_cast<FillTable<TR>*>(mine);
  uint8_t* ring = mine + fill_table_bytes(WPL);
  uint16_t* stage = reinterpret_cast<uint16_t*>(ring + R);
  for (;;) {
    uint32_t b = 0;
    if (lane_id() == 0) b = atomicAdd(A.work, 1u);
    b = __shfl_sync(kFull, b, 0);
    if (b >= A.nb) break;
    fill_block<WPL>(A, b, T, ring, R, stage);
    __syncwarp();
  }
}

// ---- several warps a block
// With fewer blocks than the GPU has room for warps, one warp a block leaves it idle and takes a block's 2^block_log
// / 128 rounds one after the other (about 0.55 us each: 1.1 ms for 256 KiB).  Here the CTA's NW warps share a block:
// warp w fills the 128-byte lines w, w + NW, ..., each looked up by itself in the token table (DecArgs.line gives
// the token that holds a line's first byte).  A word's bytes from literals and from lines that are complete are
// loaded at once; the others wait for their source words.  state[v] is the line that warp v is at, with a bit for
// each word of it that is done: a source word is there once its line lies below its warp's, or is its warp's
// line with the word's bit set.  A word's sources lie before it (or earlier in the word itself), so the first
// word not done never waits for another: all of them end; the polls are bounded all the same.
//
// Recent output is read from a ring of kMultiRing lines a warp.  A warp starts a line only within kMultiAhead * NW
// lines of the lowest incomplete one; a line then overwrites none that a warp may still read (a source at most
// (kMultiRing - kMultiAhead) * NW lines back is read from the ring, a farther one from the output itself, which
// its warp stored before it published its next line).
constexpr uint32_t kMultiWarps = 16, kMultiRing = 16, kMultiAhead = 4;
__host__ __device__ constexpr size_t multi_smem(uint32_t nw) { return nw * kMultiRing * 128; }

// a warp's state, read and published in the order of the CTA's memory: what was stored before it was published is
// there for who has read it
__device__ __forceinline__ uint64_t load_state(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.cta.shared.u64 %0, [%1];" : "=l"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
  return v;
}
__device__ __forceinline__ void store_state(uint64_t* p, uint64_t v) {
  asm volatile("st.release.cta.shared.u64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "l"(v) : "memory");
}

// a block by one warp, out of line: the shared form's registers stay its own
constexpr uint32_t kAloneRing = 4096;
static_assert(fill_table_bytes(1) + kAloneRing + fill_stage_bytes(1) <= 4 * kMultiRing * 128, "what four warps have");
__device__ __noinline__ void fill_alone(const DecArgs& A, uint32_t b, uint8_t* sm) {
  uint8_t* ring = sm + fill_table_bytes(1);
  fill_block<1>(A, b, *reinterpret_cast<FillTable<fill_rows(1)>*>(sm), ring, kAloneRing,
                reinterpret_cast<uint16_t*>(ring + kAloneRing));
}

// (Hasty: the polls' limit is A.polls, lowered for a test; read from there in every poll it cost all blocks 1 to 2 %, two
// values at random 22.1 -> 22.5 ms for 1 MiB, records 8.66 -> 8.86)
template <bool Hasty>
__global__ void __launch_bounds__(32 * kMultiWarps, 2) k_dec_fill_multi(const __grid_constant__ DecArgs A) {
  extern __shared__ __align__(16) uint8_t fsm[];
  __shared__ uint32_t next;
  __shared__ uint64_t state[kMultiWarps];
  const uint32_t NW = blockDim.x >> 5, w = threadIdx.x >> 5, lane = lane_id();
  const uint32_t RB = kMultiRing * 128 * NW, rmask = RB - 1u;
  uint8_t* ring = fsm;
  const uint32_t upto = 0xFFFFFFFFu >> (31u - lane);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) next = atomicAdd(A.work, 1u);
    if (threadIdx.x < kMultiWarps) state[threadIdx.x] = (uint64_t)threadIdx.x << 32;
    __syncthreads();
    const uint32_t b = next;
    if (b >= A.nb) break;
    const uint32_t raw = A.raw_len[b], method = A.method[b], clen = A.comp_len[b], B = A.B;
    const uint32_t alone = A.line[(size_t)(b + 1) * line_cap(B) - 1].x;  // (k_dec_tokens' choice, of a good block)
    uint8_t* o = A.out + A.out_off[b];
    if (raw > B || method > 1 || (method == 0 && clen != raw)) {
      if (threadIdx.x == 0) flag(A.err, b, raw > B ? E_RAWLEN : method > 1 ? E_METHOD : E_STORED);
      continue;
    }
    if (method == 0) {
      copy_bytes(o, A.comp + A.comp_off[b], raw, threadIdx.x, blockDim.x);
      continue;
    }
    if (A.err[b]) continue;
    if (alone) {
      if (w == 0) fill_alone(A, b, fsm);
      continue;
    }
    const DecMeta& m = A.meta[b];
    const size_t TC = tok_cap(B);
    const uint8_t* lit = A.s_lit + (size_t)b * B;
    const uint2* Tp = A.tk_pos + (size_t)b * TC;
    const uint32_t* Td = A.tk_d + (size_t)b * TC;
    const uint2* line = A.line + (size_t)b * line_cap(B);
    const uint32_t a = (uint32_t)(uintptr_t)o & 127u;  // output byte q lies in line (q + a) / 128
    const uint32_t NL = (raw + a + 127u) >> 7;
    const uint32_t back = (kMultiRing - kMultiAhead) * NW - 1u;  // lines before a line that the ring holds
    // The lane's word of a line: its last byte's token (row 1) and, where a token starts in the word, the one before
    // (row 0; the same one otherwise).  Loaded a line ahead.
    uint2 p1, p0;
    uint32_t d1, d0;
    auto fetch = [&](const uint2& l) {
      const uint32_t t1 = l.x + __popc(l.y & upto), t0 = t1 - (l.y >> lane & 1u);
      p1 = Tp[t1]; d1 = Td[t1];  // (t1 <= nt)
      p0 = Tp[t0]; d0 = Td[t0];
    };
    const uint2 none = make_uint2(m.nt, 0);
    uint2 lt = w < NL ? line[w] : none;
    fetch(lt);
    lt = w + NW < NL ? line[w + NW] : none;
    bool dead = false;
    for (uint32_t ln = w; ln < NL; ln += NW) {
      const uint32_t st1 = row_start(p1), st0 = row_start(p0);
      const uint32_t ms1 = st1 + row_lits(p1), ms0 = st0 + row_lits(p0);
      const uint32_t bk1 = row_back(p1), bk0 = row_back(p0), D1 = d1, D0 = d0;
      fetch(lt);
      lt = ln + 2 * NW < NL ? line[ln + 2 * NW] : none;
      // the lowest incomplete line; this one starts once it lies within the window
      uint32_t low;
      for (uint32_t k = 0;; ++k) {
        low = __reduce_min_sync(kFull, lane < NW ? (uint32_t)(load_state(&state[lane]) >> 32) : 0xFFFFFFFFu);
        if (ln < low + kMultiAhead * NW) break;
        if (k > (Hasty ? A.polls : kFillPolls)) { dead = true; break; }
      }
      if (dead) break;
      __syncwarp();
      const int32_t lb = (int32_t)(ln << 7) - (int32_t)a;
      const int32_t q0 = lb + 4 * (int32_t)lane;
      const int32_t rlo = lb - (int32_t)(back << 7);
      // A byte's source: itself for a literal, D before it for a match byte, its period's start for one that repeats
      // the match's own bytes (q - D - D * (x / D), x its offset in the match, x >= D: few lines hold one).  Bytes
      // from a token's own literals are read from the literals.
      uint32_t v[4], s[4], wait = 0, over = 0;  // bit j of wait: byte j's source may not be there yet
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t q = (uint32_t)(q0 + j);
        const bool hi = q >= st1;
        const uint32_t ms = hi ? ms1 : ms0, D = hi ? D1 : D0;
        const int32_t x = (int32_t)(q - ms);
        s[j] = x >= 0 ? q - D : q;
        over |= (uint32_t)(x >= (int32_t)D) << j;
      }
      if (__any_sync(kFull, over)) {
        // x / D for x, D < 2^20 by a float product, at most one too low; then D's multiples for the later bytes
        const uint32_t x1 = (uint32_t)max(q0 - (int32_t)ms1, 0), x0 = (uint32_t)max(q0 - (int32_t)ms0, 0);
        const uint32_t k1 = (uint32_t)__fdividef((float)x1, (float)D1) * D1;
        const uint32_t k0 = (uint32_t)__fdividef((float)x0, (float)D0) * D0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t q = (uint32_t)(q0 + j);
          const bool hi = q >= st1;
          const uint32_t ms = hi ? ms1 : ms0, D = hi ? D1 : D0;
          uint32_t r = q - ms - (hi ? k1 : k0);
#pragma unroll
          for (int t = 0; t < 4; ++t) r = r >= D ? r - D : r;
          if (over >> j & 1u) s[j] = ms - D + r;
        }
      }
      const int32_t lows = (int32_t)(low << 7) - (int32_t)a;  // the first output byte that may not be there
      auto bytes = [&](auto whole) {  // (a line inside the block needs no bounds)
        constexpr bool inside = decltype(whole)::value;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int32_t qi = q0 + j;
          const bool valid = inside || (qi >= 0 && qi < (int32_t)raw);
          const bool hi = (uint32_t)qi >= st1;
          const bool own = s[j] >= (hi ? st1 : st0);
          const bool later = !own && (int32_t)s[j] >= lows;
          const bool near = !own && (int32_t)s[j] >= rlo;
          wait |= (uint32_t)(valid && later) << j;
          v[j] = 0;
          const uint8_t* from = own ? lit : o;
          const uint32_t off = own ? s[j] - (hi ? bk1 : bk0) : s[j];
          if (valid && !near) v[j] = from[off];
          if (valid && near && !later) v[j] = ring[(s[j] + a) & rmask];
        }
      };
      if (lb >= 0 && lb + 128 <= (int32_t)raw) bytes(std::true_type{}); else bytes(std::false_type{});
      uint32_t word = v[0] | v[1] << 8 | v[2] << 16 | v[3] << 24;
      uint32_t* const slot = reinterpret_cast<uint32_t*>(ring + (((ln << 7) + 4 * lane) & rmask));
      if (!wait) *slot = word;
      uint32_t done = __ballot_sync(kFull, !wait);
      // The bytes that wait come from one or two source words (sa, sb, by the output's word number) in most words:
      // those are taken once both are there; the others byte by byte, as are bytes from earlier in the word itself.
      const uint32_t here = (ln << 5) + lane;
      auto there = [&](uint32_t sw) {  // is output word sw done?
        const uint64_t st = load_state(&state[sw >> 5 & (NW - 1u)]);
        const uint32_t l = (uint32_t)(st >> 32), sl = sw >> 5;
        return l > sl || (l == sl && ((uint32_t)st >> (sw & 31u) & 1u));
      };
      uint32_t sa = 0, sb = 0;
      bool mixed = false;
      if (done != kFull && wait) {
        const int j0 = __ffs(wait) - 1, j1 = 31 - __clz(wait);
        sa = (j0 == 0 ? s[0] : j0 == 1 ? s[1] : j0 == 2 ? s[2] : s[3]) + a >> 2;
        sb = (j1 == 3 ? s[3] : j1 == 2 ? s[2] : j1 == 1 ? s[1] : s[0]) + a >> 2;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t sw = (s[j] + a) >> 2;
          mixed |= (wait >> j & 1u) && ((sw != sa && sw != sb) || sw == here);
        }
      }
      uint32_t shown = 0;
      for (uint32_t k = 0; done != kFull; ++k) {
        __syncwarp();
        if (lane == 0 && done != shown) store_state(&state[w], (uint64_t)ln << 32 | done);
        shown = done;
        if (wait && !mixed && there(sa) && there(sb)) {  // (a line not complete at the start is in the ring)
          const uint32_t wa = reinterpret_cast<const uint32_t*>(ring)[sa & (rmask >> 2)];
          const uint32_t wb = reinterpret_cast<const uint32_t*>(ring)[sb & (rmask >> 2)];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t at = s[j] + a;
            const uint32_t c = ((at >> 2 == sa ? wa : wb) >> 8 * (at & 3u) & 0xFFu) << 8 * j;
            word |= wait >> j & 1u ? c : 0u;
          }
          wait = 0;
          *slot = word;
        }
        if (__any_sync(kFull, mixed)) {
          if (mixed) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (!(wait >> j & 1u)) continue;
              const uint32_t at = s[j] + a;
              if (at >> 2 == here) {  // earlier in this word
                if (wait >> (at & 3u) & 1u) continue;
                word |= (word >> 8 * (at & 3u) & 0xFFu) << 8 * j;
              } else {
                if (!there(at >> 2)) continue;
                word |= (uint32_t)ring[at & rmask] << 8 * j;
              }
              wait &= ~(1u << j);
            }
            if (!wait) { mixed = false; *slot = word; }
          }
        }
        done = __ballot_sync(kFull, !wait);
        if (k > (Hasty ? A.polls : kFillPolls)) { dead = true; break; }
      }
      if (dead) break;
      __syncwarp();
      if (lane == 0) store_state(&state[w], (uint64_t)(ln + NW) << 32);
      if (q0 >= 0 && q0 + 4 <= (int32_t)raw) {
        *reinterpret_cast<uint32_t*>(o + q0) = word;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (q0 + j >= 0 && q0 + j < (int32_t)raw) o[q0 + j] = (uint8_t)(word >> (8 * j));
      }
    }
    __syncwarp();
    if (lane == 0) store_state(&state[w], (uint64_t)0x7FFFFFFFu << 32);
    if (dead && lane == 0) flag(A.err, b, E_GAVE_UP);
  }
}

size_t fill_smem_bytes(uint32_t ring_log, uint32_t warps, uint32_t words) {
  return (size_t)warps * (fill_table_bytes(words) + (1u << ring_log) + fill_stage_bytes(words));
}

cudaError_t prepare_fill() {
  const int cap = (int)kMaxFillSmem;
  cudaError_t e = cudaFuncSetAttribute(k_dec_fill<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_dec_fill<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_dec_fill<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  return e;
}

constexpr uint32_t kFillSms = 148;

void launch_decode_fill(const DecArgs& args, cudaStream_t st, Stages& S) {
  DecArgs A = args;
  if (!A.nb) return;
  // A warp a block beyond six blocks an SM, else 4 to kMultiWarps warps a block, as many as the GPU holds (32 an SM).
  // Block 18, ms with 1 / 4 / 8 / 16 warps, lz_mix: 256 blocks 1.16 / 0.76 / 0.56 / 0.51, 1024 blocks 1.41 / 1.57 /
  // 1.55 / 1.65, 1600 blocks 1.63 / 2.27 / 2.55 / 2.56; block 16, 768 blocks: lz_mix 0.34 / 0.36 / 0.35 / 0.38, text
  // 0.43 / 0.34 / 0.35 / 0.43; 1200 blocks: text 0.49 / 0.47 / 0.52 / 0.63.  Sharing a block costs waits on its
  // source words, so it pays while warps are few: the line lies where lz_mix loses as little as text gains.
  uint32_t nw = 1;
  if (A.line && A.nb <= kFillSms * 6)
    for (nw = 4; nw < kMultiWarps && 2 * nw * A.nb <= kFillSms * 32;) nw *= 2;
  if (nw == 1) A.line = nullptr;
  launch_dec_streams(A, st, S);
  S.begin("k_dec_tokens", st);
  k_dec_tokens<<<A.nb, kTokThreads, 0, st>>>(A);
  S.end(st);
  cudaMemsetAsync(A.work, 0, sizeof(uint32_t), st);
  if (nw > 1) {
    S.begin("k_dec_fill", st);
    if (A.polls < kFillPolls) k_dec_fill_multi<true><<<A.nb, 32 * nw, multi_smem(nw), st>>>(A);
    else k_dec_fill_multi<false><<<A.nb, 32 * nw, multi_smem(nw), st>>>(A);
    S.end(st);
    return;
  }
  const uint32_t W = A.fill_warps;
  const size_t sm = fill_smem_bytes(A.ring_log, W, A.fill_words);
  const uint32_t grid = (A.nb + W - 1) / W;  // (as many warps as blocks; the counter balances them)
  S.begin("k_dec_fill", st);
  if (A.fill_words == 4) k_dec_fill<4><<<grid, 32 * W, sm, st>>>(A);
  else if (A.fill_words == 2) k_dec_fill<2><<<grid, 32 * W, sm, st>>>(A);
  else k_dec_fill<1><<<grid, 32 * W, sm, st>>>(A);
  S.end(st);
}

}  // namespace zc
