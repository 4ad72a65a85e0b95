// The symbol chain of the entropy stage: a tile's interleaved rANS decoder
// (ebiv/rans.go:222-304) driving the part of the macroblock grammar that picks
// the next context (ebiv/decode_intra.go:121-167, ebiv/decode_inter.go:8-62,
// ebiv/residual.go:79-126, ebiv/mv.go:75-128), and the log it leaves for
// kParseMB.  Device code; compiled by a host compiler too, for tests.
#pragma once

#include <cstddef>
#include <cstdint>

#include "ebiv_format.h"

#ifdef __CUDACC__
#define EBIV_DEV __device__ __forceinline__
#else  // the few device names the chain uses, for host tests
#include <algorithm>
#define EBIV_DEV inline
struct uint4 {
  uint32_t x, y, z, w;
};
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return uint4{x, y, z, w}; }
template <class T>
inline T __ldg(const T* p) {
  return *p;
}
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t n) {
  return (n & 31) ? hi << (n & 31) | lo >> (32 - (n & 31)) : hi;
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t n) {
  return (n & 31) ? lo >> (n & 31) | hi << (32 - (n & 31)) : lo;
}
using std::min;
#endif

namespace ebiv {
namespace dev {

// ---------------------------------------------------------------------------
// Symbol tables, built once per CTA for the frame whose tiles it decodes
// ---------------------------------------------------------------------------
// One 16-byte entry per context and bucket of 64 slots, for the symbol s that
// holds the bucket's first slot.  A bucket's entries of the three
// previous-value classes of a plane, transform size and band lie side by
// side, with one of the other contexts in the fourth place; its 64 bytes are
// where bits 6-11 of the state point, so an entry's offset is the masked
// state or-ed with its row: group (4 KB each) and place.  The signs have a
// group of their own with the same entry in three places, so that a row of it
// keeps the class that the token before the sign leaves, and in the fourth
// place as the last symbol of a block (kEEnd).
//
// The words are masks and numbers that the chain uses as they are:
//   x  frequency - 4096: the next state is x * (state >> 12) + state - start
//   y  start
//   z  kEAdvance when the next symbol's position in the block is the next one
//      (tokens, signs, modes), else 0; or, in bit 31, kEStop with the reason:
//      kEEnd (end of block, last sign and transform size, these with kEBlock,
//      escape, a mode that is not skip),
//      kEImpure (a later symbol starts inside the bucket; y is the index, in
//      entries from the first, of the symbol's own one, from where resolve()
//      goes on, and x the class of a sign's row) or kEUnused (an unused
//      context; the entry is the identity)
//   w  the log entry (bits 0-15; a nonzero token has bit 2 set and the class
//      it leaves in bits 4-5), and kENonzero for a token of magnitude one to
//      four
constexpr uint32_t kEStop = 1u << 31, kEEnd = 1u << 30, kEImpure = 1u << 29, kEUnused = 1u << 28, kEBlock = 1u << 27;
constexpr uint32_t kGroupBytes = 4096, kClassBytes = 16, kBucketMask = 0xFC0, kClassMask = 0x30;
constexpr uint32_t kGroupMask = 0x1F000;                         // the group in a row
constexpr uint32_t kERest = 1u << 8;                             // ChainOf::z: the edge is not the block's end
constexpr uint32_t kECount = 1u << 20;                           // one position, in ChainOf::z
constexpr uint32_t kEAdvance = kECount | kGroupBytes | 1u;       // a position, a band's step, a shift by one
constexpr uint32_t kENonzero = 1u << 31 | kGroupMask | kEAdvance;
constexpr int kTokenGroups = 4 * kNumBands;
constexpr uint32_t kSignRow = kTokenGroups * kGroupBytes, kLastSignRow = kSignRow | kClassMask;
constexpr int kSymbols = 18;  // own entries of a context: its symbols, then sentinels past the last slot
static_assert(kNumContexts == ctxTokenBase + 3 * kTokenGroups && ctxTokenBase <= kTokenGroups && kTokenGroups < 32,
              "entry layout");
// What follows a block: the row of the next one's first symbol (x), the values
// that ChainOf::z and ::bands start with (y, z) and z's count past position
// 19 (w), for blocks of a kind.  Kinds 0-2: luma by transform size, 3 chroma,
// + 4 with an intra mode in front.
constexpr int kBlockKinds = 8;
struct EntropyTables {
  uint4 entry[(kTokenGroups + 1) * 64 * 4];
  uint4 symbol[kNumContexts * kSymbols];
  uint4 block[kBlockKinds];
};
static_assert(kSDHMinSpan == 4, "bit 2 of ChainOf::since");
// The row of context c (of the signs: with class 0 to keep).
EBIV_DEV uint32_t rowOf(int c) {
  if (c == ctxSign) return kSignRow;
  return c < ctxTokenBase ? (uint32_t)c * kGroupBytes + 3 * kClassBytes
                          : (uint32_t)((c - ctxTokenBase) / 3) * kGroupBytes + (uint32_t)((c - ctxTokenBase) % 3) * kClassBytes;
}

// The log: 16 bits per symbol that name its kind (bits 6-7) and its value
// (from bit 8), so that kParseMB's lanes can read one each.  A macroblock that
// is not skip has its mode (inter frames), an inter one its reference,
// partition, vector components and pattern, then the transform size when it
// has luma; per coded block the intra mode if it has one, every token, each
// nonzero token but the block's first followed by its sign (after an escape's
// value), tEOB also where the block ends without one, and the first nonzero
// token's sign when it is coded.  Vector components and escape values (class
// values of 15 bits) are two entries of eight bits, the high ones first.
constexpr uint32_t kLogToken = 0, kLogSign = 1u << 6, kLogMode = 2u << 6, kLogValue = 3u << 6, kLogKind = 3u << 6;
constexpr int kLogShift = 8;
constexpr uint32_t kLogNonzero = 4;               // token flag, where ChainOf::far looks
constexpr uint32_t kSkipOffset = 0xFFFFFFFFu;     // a skip macroblock: it has no log
constexpr uint32_t kDecodedOffset = 0xFFFFFFFEu;  // one that the full chain has decoded, or that is not reached
// The most entries of a block of n positions (the mode in front is one): a
// token and a sign for each position and the end; a block has a last sign only
// when its nonzero tokens are four at most, so that others have no sign.  Of a
// macroblock without escapes: the header (mode, reference, partition, eight
// vector components, pattern, transform size) and the blocks, 17 with a mode.
// An escape adds its value.
EBIV_DEV constexpr int blockEntries(int n) { return 2 * n + 1; }
constexpr int kHeaderEntries = 5 + 8 * 2, kEscapeEntries = 2;
constexpr int kPlainMBEntries = kHeaderEntries + 2 * 384 + 17;
constexpr int kLastEntries = 4;  // kept free: the next macroblock's transform size, once
constexpr int kMBEntries = kPlainMBEntries + kEscapeEntries * 384 + kLastEntries;

// The entry of symbol s of context c, which starts at st and has frequency
// freq, in a row that keeps class cls (signs).
EBIV_DEV uint4 symbolEntry(int c, int s, uint32_t st, uint32_t freq, uint32_t cls) {
  uint32_t z = 0, w = (uint32_t)s << kLogShift;
  if (c >= ctxTokenBase) {
    z = s < tEscape ? kEAdvance : kEStop | kEEnd | (s == tEOB ? kEBlock : 0u);
    if (s >= tOne && s <= tFour) w |= kENonzero;
    if (s >= tOne && s <= tEscape) w |= kLogNonzero | (s == tOne ? kClassBytes : 2 * kClassBytes);
  } else if (c == ctxSign) {
    const bool last = cls == kClassMask;
    z = last ? kEStop | kEEnd | kEBlock : kEAdvance;
    w |= last ? kLogSign : kLogSign | cls;
  } else if (c == ctxLumaMode || c == ctxChromaMode) {
    z = kEAdvance;
    w |= kLogMode;
  } else {
    if (c == ctxMBMode && s != mbSkip) z = kEStop | kEEnd;
    if (c == ctxTxSize) z = kEStop | kEEnd | kEBlock;
    w |= kLogValue;
  }
  return make_uint4(freq - kM, st, z, w);
}
EBIV_DEV uint4 unusedEntry() { return make_uint4(0u, 0u, kEStop | kEUnused, 0u); }
EBIV_DEV uint4 sentinelEntry() { return make_uint4(0u, kM, 0u, 0u); }

// The entry of bucket b of context c, whose symbol s, the last one that
// starts at or before the bucket's first slot, covers [st, nx).
EBIV_DEV uint4 bucketEntry(int c, int s, uint32_t st, uint32_t nx, uint32_t b, uint32_t cls) {
  if (nx < ((b + 1) << 6))
    return make_uint4(cls, (uint32_t)(offsetof(EntropyTables, symbol) / 16) + (uint32_t)(c * kSymbols + s),
                      kEStop | kEImpure, 0u);
  return symbolEntry(c, s, st, nx - st, cls);
}

// The row of the token after the next symbol's is a band further after
// positions 1, 7 and 19 (bandOf(i + 2)).  With a mode in front, which moves on
// like a token, `bands` holds the first two, up to position 18: then there is
// an edge, as there is at the block's end.
EBIV_DEV uint4 blockEntry(int kind) {
  const bool mode = kind >= 4;
  const uint32_t plane = (uint32_t)kind & 3u, total = plane == 3 ? 64u : 16u << (2 * plane);
  const uint32_t row = plane * kNumBands * kGroupBytes;
  const bool rest = mode && total > 19;
  const uint32_t edge = mode ? 1 + (rest ? 19 : total) : total;
  return make_uint4(mode ? rowOf(plane == 3 ? ctxChromaMode : ctxLumaMode) : row,
                    (mode ? row : row + kGroupBytes) + (2048 - edge) * kECount + (rest ? kERest : 0u),
                    mode ? (1u | 1u << 2 | 1u << 8) << 12 : (1u << 1 | 1u << 7 | 1u << 19) << 12,
                    rest ? (2048 - (total - 19)) * kECount : 0u);
}

// Where a tile's rANS decoder stands between two symbols: its states in use
// order and the stream bytes not taken yet (it reads them backwards).
struct ChainState {
  uint32_t x0, x1, x2, x3;
  int32_t pos;
};
// Where a run of the symbol chain failed: the macroblocks surely complete, the
// first one behind those that it leaves, and the stream bytes left.
struct ChainFailure {
  int reached, next, pos;
};
// The state at a tile's start, from the end of its len >= 16 bytes
// (ransDecoder.reset, ebiv/rans.go:236-250).
EBIV_DEV ChainState initialState(const uint8_t* buf, uint32_t len) {
  uint32_t st[kStates];
  int pos = (int)len;
#pragma unroll
  for (int i = kStates - 1; i >= 0; i--) {
    st[i] = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) st[i] = st[i] << 8 | (uint32_t)__ldg(buf + --pos);
  }
  return ChainState{st[0], st[1], st[2], st[3], pos};
}

// A tile's chain, run by one thread.
//
// A symbol's context is known only when the symbol before it is, so the chain
// is serial; what it costs is set by what one warp alone on its scheduler
// pays: 23 cycles for a shared-memory load, 4 for an instruction that needs
// the one before (1 to 2 for one that does not), and for a branch 10 not
// taken, 15 to 20 taken (measured).  A decoder written with branches for
// tokens, signs, bands and stream bytes took 67 instructions, 9 of them
// branches, and 270 cycles a symbol.  So the symbols of a macroblock's blocks
// all take the same straight line (tokens()), four of them, one per rANS
// state, in a loop: the entry's words turn the state of the grammar into the
// next by masks, the next entry's address is two logic operations away from
// this one's entry, and one test per symbol finds everything else.  The ends
// of blocks, last signs, buckets with a boundary and, in a frame of intra
// macroblocks, the transform sizes then go through a stub beside the line and
// join it again (one for each state, so that no register moves); escapes,
// edges and second stream bytes leave it.  Measured: 91 cycles a symbol on the
// line, 105 to 120 with everything (720p key frame of one tile at q18, 448
// thousand symbols: 61 ms before, 25 ms), 31 a skip (77 before).  Issuing the
// next entry's load before the test instead of after it: 107 on the line; four
// symbols to a test: 70, but what follows an end in its group is lost and
// undone, 170 with everything.
//
// kRooms: the macroblocks' logs lie in rooms of their own, as the kernel has
// them in the coefficient regions, else one behind the other.
template <bool kRooms>
struct ChainOf {
  uint32_t x0, x1, x2, x3;  // states in use order: x0 decodes the next symbol
  // The stream, read backwards: hi and lo are its next words, off the bits of
  // hi that are used, nw the word after lo, wp its address; rem counts the
  // bits left, below 0 when a symbol has taken a byte before the tile's first
  // one.  The words read ahead are up to 15 bytes before that byte, in the
  // packet: 78 bytes of headers and tables at least precede a tile.
  uint32_t hi, lo, off, nw;
  const uint32_t* wp;
  int32_t rem;
  const EntropyTables* t;
  // The log of `entries` entries, or rooms of as many: the tile's rows (of
  // `width`) lie `gap` more than their rooms apart, and log moves on by that
  // with the rows; macroblock mb, before rowEnd, has those from log + mb *
  // entries.
  uint16_t* log;
  uint16_t* lp;     // the next entry
  uint16_t* first;  // the macroblock's first one
  int32_t width, entries, gap, rowEnd;
  int32_t escaped;  // the macroblock has an escape
  int32_t stop;    // macroblocks to decode; 0 after a failure
  // The grammar inside a macroblock's blocks.  kind: its block entry; left:
  // the blocks after this one that have the same, -1 past the macroblock's
  // last; queue: the kinds after those, a byte each, kind + 1 and in the high
  // half the blocks less one.  z: the row of the token at the position after
  // the next symbol's (class 0), and in bits 20-31 the positions up to an edge,
  // counted up to a set sign bit.  bands: bit 12 is set when the row after that
  // is a band further, the bits above it for the positions that follow.  seen:
  // kClassMask, and kENonzero after a nonzero token.  since: a set bit for each
  // position after the first nonzero token's and before this one (unary, the
  // oldest lost).  far: bit 2 is set once a nonzero token was kSDHMinSpan or
  // more positions after the first.
  // The macroblocks: mb is the current one, mbOff where their logs begin or
  // how many entries they have; intraOnly: no mode in front of a macroblock.
  uint4 kind;
  int32_t left;
  int32_t mb;
  bool intraOnly;
  uint32_t* mbOff;
  uint32_t queue, z, bands, seen, since, far;

  EBIV_DEV uint4 entryAt(uint32_t offset) const {
#ifdef __CUDACC__
    uint4 e;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(e.x), "=r"(e.y), "=r"(e.z), "=r"(e.w)
                 : "r"((uint32_t)__cvta_generic_to_shared(t->entry) + offset));
    return e;
#else
    return *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(t->entry) + offset);
#endif
  }
  EBIV_DEV int count() const { return (int)(lp - log); }
  EBIV_DEV void put(uint32_t v) { *lp++ = (uint16_t)v; }
  EBIV_DEV void putValue(uint32_t v) {
    put(kLogValue | (v >> 8) << kLogShift);
    put(kLogValue | (v & 255u) << kLogShift);
  }
  // A symbol that cannot be decoded (an unused context, a byte before the
  // tile's first), or one with no room: the macroblock is left to the full chain.
  EBIV_DEV void fail() { stop = 0; }
  // The log's part for macroblock mb.
  EBIV_DEV void open() {
    if (kRooms) {
      while (mb >= rowEnd) {
        rowEnd += width;
        log += gap;
      }
      lp = log + (ptrdiff_t)mb * entries;
    }
    first = lp;
    escaped = 0;
  }
  // All of macroblock mb is in the log.
  EBIV_DEV void close() { mbOff[mb] = (uint32_t)(kRooms ? lp - first : first - log); }
  // And the next one follows (without a branch).
  EBIV_DEV void step() {
    close();
    mb++;
    if (kRooms) {
      const bool row = mb == rowEnd;
      rowEnd += row ? width : 0;
      log += row ? gap : 0;
      first += row ? entries + gap : entries;
      lp = first;
    }
    first = lp;
    escaped = 0;
  }
  // The entries left from lp on.
  EBIV_DEV int room() const { return entries - (int)(lp - (kRooms ? first : log)); }
  // Keeps off below 32.
  EBIV_DEV void refill() {
#ifdef __CUDACC__  // without a branch
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ge.u32 p, %2, 32;\n"
        "@p add.u32 %2, %2, -32;\n"
        "@p mov.b32 %0, %1;\n"
        "@p mov.b32 %1, %3;\n"
        "@p add.u64 %4, %4, -4;\n"
        "@p ld.global.nc.u32 %3, [%4];\n}"
        : "+r"(hi), "+r"(lo), "+r"(off), "+r"(nw), "+l"(wp));
#else
    if (off >= 32) {
      off -= 32;
      hi = lo;
      lo = nw;
      nw = __ldg(--wp);
    }
#endif
  }
  // A state below kLower takes the next byte of cur, the next stream bits.
  static EBIV_DEV void take(uint32_t& v, uint32_t& cur, int32_t& rem) {
#ifdef __CUDACC__  // predicated: a branch costs more
    asm("{\n.reg .pred p;\n"
        "setp.lt.u32 p, %0, 8388608;\n"
        "@p shf.l.wrap.b32 %0, %1, %0, 8;\n"
        "@p shl.b32 %1, %1, 8;\n"
        "@p add.s32 %2, %2, -8;\n}"
        : "+r"(v), "+r"(cur), "+r"(rem));
#else
    if (v < kLower) {
      v = __funnelshift_l(cur, v, 8);
      cur <<= 8;
      rem -= 8;
    }
#endif
  }
  // Stream bytes for the state v.
  EBIV_DEV uint32_t fill(uint32_t v) {
#pragma unroll 1
    while (v < kLower) {
      if (rem < 8) {
        fail();
        return v | kLower;
      }
      v = v << 8 | __funnelshift_l(lo, hi, off) >> 24;
      off += 8;
      rem -= 8;
      refill();
    }
    return v;
  }

  // The entry of the symbol that holds state x's slot, for one with kEImpure.
  EBIV_DEV uint4 resolve(const uint4& e, uint32_t x) const {
    const uint32_t slot = x & (kM - 1);
    uint32_t q = 16 * e.y;
    const uint4 r0 = entryAt(q), r1 = entryAt(q + 16);
    uint32_t end = entryAt(q + 32).y;
    uint4 r = slot < r1.y ? r0 : r1;  // most buckets hold two symbols
#pragma unroll 1
    while (slot >= end) {
      r = entryAt(q += 32);
      end = entryAt(q + 16).y;
      q -= 16;
    }
    const bool last = e.x == kClassMask;  // the last sign's row; else the row's class (0 but for signs)
    r.z = last ? kEStop | kEEnd | kEBlock : r.z;
    r.w |= last ? 0u : e.x;
    return r;
  }
  // One symbol with everything that can happen to it, from its entry; it is
  // not yet in the log.  A symbol of an unused context fails.
  EBIV_DEV uint4 symbolOf(uint4 e) {
    if (e.z & kEUnused) fail();
    if (e.z & kEImpure) e = resolve(e, x0);
    const uint32_t v = fill(e.x * (x0 >> kScaleBits) + x0 - e.y);
    x0 = x1;
    x1 = x2;
    x2 = x3;
    x3 = v;
    return e;
  }
  EBIV_DEV uint32_t sym(int ctx) { return (symbolOf(entryAt(rowOf(ctx) | (x0 & kBucketMask))).w >> kLogShift) & 15u; }
  // getClassValue with getRawBits — ebiv/mv.go:75-103.
  EBIV_DEV uint32_t classValue(int ctx) {
    const uint32_t cls = sym(ctx);
    uint32_t v = min(cls, 1u);
#pragma unroll 1
    for (uint32_t k = 1; k < cls; k++) v = v << 1 | sym(ctxBypass);
    return v;
  }

  // The offset of the symbol after the one of entry e, when state xn decodes
  // it.  A nonzero token after the first goes to the sign's row, all else to
  // z's row; both keep the class.
  EBIV_DEV uint32_t nextAt(const uint4& e, uint32_t xn) const {
    const uint32_t row = z & kGroupMask;
    const uint32_t to = (row ^ (kSignRow | kClassMask)) & seen;
    return (row ^ (xn & kBucketMask)) ^ (e.w & to);
  }
  // The rest of the grammar's state after it.  A nonzero token that a sign
  // follows leaves the position to the sign.
  EBIV_DEV void follow(const uint4& e) {
    const uint32_t adv = e.z & ~(e.w & seen);
    far |= since & e.w;
    since = __funnelshift_l(seen, since, adv);
    seen |= e.w & kENonzero;
    z += (bands | kECount) & adv;
    bands = __funnelshift_r(bands, 0u, adv);
  }

  // The blocks of the queue's next byte, behind the entry lp[j].  Without an
  // escape before it in the macroblock there is room for them.
  EBIV_DEV void nextKind(int j) {
    kind = entryAt((uint32_t)offsetof(EntropyTables, block) - 16 + 16 * (queue & 15u));
    left = (int32_t)((queue >> 4) & 15u);
    queue >>= 8;
    if (escaped && room() - (j + 1) < (left + 1) * blockEntries(positions(kind.y)) + kLastEntries) {
      fail();
      left = -1;
    }
  }
  // Up to the edge and behind it: the positions of a block whose z or kind is at v.
  EBIV_DEV int positions(uint32_t v) const {
    return 2048 - (int)(v >> 20) + (v & kERest ? 2048 - (int)(kind.w >> 20) : 0);
  }
  // The blocks of an intra macroblock of transform size tx.
  static EBIV_DEV uint32_t intraQueue(uint32_t tx) {
    return (tx + 5u) | ((16u >> (2 * tx)) - 1) << 4 | (8u | 4u << 8) << 8;
  }
  // After the last block of a kind: the next kind; in a frame of intra
  // macroblocks only, the next one's transform size, which is the first entry
  // of its log, and then its blocks (e is the symbol of lp[j]).
  EBIV_DEV void endedKind(const uint4& e, int j) {
    if ((e.w & kLogKind) == kLogValue) {
      queue = intraQueue(min((e.w >> kLogShift) & 15u, 2u));  // alphabet size 3
      lp += j;
      step();
      *lp = (uint16_t)e.w;
      lp -= j;
    } else if (queue == 0) {
      if (!intraOnly || mb + 1 >= stop || (!kRooms && room() < kPlainMBEntries + 2 * kLastEntries)) return;
      kind = make_uint4(rowOf(ctxTxSize), 0u, 0u, 0u);
      left = 0;
      return;
    }
    nextKind(j);
  }
  // The grammar after a block's end, its last sign, or a transform size (the
  // symbol of entry e, at lp[j]): the offset of the next symbol, which state
  // xn decodes.
  EBIV_DEV uint32_t ended(const uint4& e, int j, uint32_t xn) {
    const bool sign = (seen & kGroupMask) != 0 && !(far & kLogNonzero);
    seen = kClassMask;
    since = far = 0;
    left -= sign ? 0 : 1;
    if (left < 0) endedKind(e, j);
    z = left < 0 ? 1u << 31 : kind.y;
    bands = kind.z;
    return (sign ? kLastSignRow : kind.x) | (xn & kBucketMask);
  }

  // The symbols of a macroblock's blocks (decodeBlock, ebiv/residual.go:79-126),
  // which `blocks` lists as `queue` does, and with intraOnly those of the
  // macroblocks after it.
  EBIV_DEV void tokens(uint32_t blocks) {
    queue = blocks;
    nextKind(-1);
    z = kind.y;
    bands = kind.z;
    seen = kClassMask;
    since = far = 0;
    uint4 e = entryAt(kind.x | (x0 & kBucketMask)), f;
    // Sign bits: the last state, and the one before it, need another byte.  It
    // is looked at one symbol late, so that the test does not wait for it.
    uint32_t small = 0, small1 = 0;
    int n;
    int32_t had = rem, had1 = rem;  // bits left at the window, and before the last symbol
    uint32_t cur = __funnelshift_l(lo, hi, off);
    // One symbol, of entry E, with the state X, the next one's being XN and
    // its entry F; and its stub for what needs more than the line has.
#define EBIV_UPDATE(J, X, E)                  \
  small1 = small;                             \
  had1 = rem;                                 \
  X = E.x * (X >> kScaleBits) + X - E.y;      \
  take(X, cur, rem);                          \
  small = X - kLower;                         \
  lp[J] = (uint16_t)E.w;
#ifdef __CUDACC__  // keeps the symbol's work here, beside the next entry's load
#define EBIV_PIN(X) asm volatile("" : "+r"(X), "+r"(z), "+r"(bands), "+r"(seen));
#else
#define EBIV_PIN(X)
#endif
#define EBIV_PLAIN(J, X, XN, E, F)                                                            \
  go##J : F = entryAt(nextAt(E, XN));                                                         \
  EBIV_UPDATE(J, X, E)                                                                        \
  follow(E);                                                                                  \
  EBIV_PIN(X)
#define EBIV_MORE(E) __builtin_expect((int32_t)(E.z | z | small1) < 0, 0)
#define EBIV_STUB(J, X, XN, E, F)                                                             \
  if ((int32_t)(E.z << 4 & ~(z | small1)) < 0) { /* kEBlock */                                \
    EBIV_UPDATE(J, X, E)                                                                      \
    F = entryAt(ended(E, J, XN));                                                             \
  } else {                                                                                    \
    n = J;                                                                                    \
    if ((int32_t)(z | small1) < 0 || !(E.z & kEImpure)) goto stopped;                         \
    E = resolve(E, X);                                                                        \
    if ((int32_t)E.z < 0) goto stopped;                                                       \
    goto go##J;                                                                               \
  }
    for (;;) {
      if (EBIV_MORE(e)) goto stub0;
      EBIV_PLAIN(0, x0, x1, e, f)
      if (EBIV_MORE(f)) goto stub1;
      EBIV_PLAIN(1, x1, x2, f, e)
      if (EBIV_MORE(e)) goto stub2;
      EBIV_PLAIN(2, x2, x3, e, f)
      if (EBIV_MORE(f)) goto stub3;
      EBIV_PLAIN(3, x3, x0, f, e)
    next3:
      lp += 4;
      off += (uint32_t)(had - rem);
      if (rem < 0) return fail();
      refill();
      had = rem;
      cur = __funnelshift_l(lo, hi, off);
      continue;
    stub0:
      EBIV_STUB(0, x0, x1, e, f)
      if (!EBIV_MORE(f)) goto go1;
    stub1:
      EBIV_STUB(1, x1, x2, f, e)
      if (!EBIV_MORE(e)) goto go2;
    stub2:
      EBIV_STUB(2, x2, x3, e, f)
      if (!EBIV_MORE(f)) goto go3;
    stub3:
      EBIV_STUB(3, x3, x0, f, e)
      goto next3;
    stopped:
      lp += n;
      off += (uint32_t)(had - rem);
      refill();
      if (n & 1) {  // the states in use order again
        const uint32_t v = x0;
        x0 = x1;
        x1 = x2;
        x2 = x3;
        x3 = v;
        e = f;
      }
      if (n & 2) {
        uint32_t v = x0;
        x0 = x2;
        x2 = v;
        v = x1;
        x1 = x3;
        x3 = v;
      }
      if (rem < 0) return fail();
      if ((int32_t)(small | small1) < 0) {
        if ((int32_t)small1 < 0) {  // x2's byte comes before the one that x3 may have taken
          if (had1 != rem) {
            if (off == 0) {  // it was the last of the word before
              nw = lo;
              lo = hi;
              hi = x3 & 255u;
              off = 32;
              wp++;
            }
            x3 >>= 8;
            off -= 8;
            rem += 8;
          }
          x2 = fill(x2);
        }
        x3 = fill(x3);
        small = small1 = 0;
      }
      if (left < 0 || stop == 0) return;
      if ((int32_t)z < 0) {  // an edge
        if (z & kERest) {
          z = (z & kGroupMask) + kind.w;
          bands = 1u << 12;
        } else {
          put(tEOB << kLogShift);
          e = entryAt(ended(make_uint4(0u, 0u, 0u, 0u), -1, x0));
          if (left < 0) return;
        }
      } else if (e.z & kEBlock) {
        e = symbolOf(e);
        put(e.w);
        e = entryAt(ended(e, -1, x0));
        if (left < 0) return;
      } else if ((e.z & (kEUnused | kEEnd)) != 0) {
        // A failure, or an escape: its value, then the sign unless it is the
        // first nonzero token.
        e = symbolOf(e);
        escaped = 1;
        if (room() < kEscapeEntries + blockEntries(positions(z)) + left * blockEntries(positions(kind.y)) + kLastEntries)
          return fail();
        put(e.w);
        putValue(classValue(ctxEscClass));
        if (seen & kGroupMask) put(kLogSign | sym(ctxSign) << kLogShift);
        if (stop == 0) return;
        e = entryAt((z & kGroupMask) | 2 * kClassBytes | (x0 & kBucketMask));
        far |= since & kLogNonzero;
        since = __funnelshift_l(seen, since, kEAdvance);
        seen |= kENonzero;
        z += (bands | kECount) & kEAdvance;
        bands >>= 1;
      }
      had = rem;
      cur = __funnelshift_l(lo, hi, off);
    }
#undef EBIV_STUB
#undef EBIV_MORE
#undef EBIV_PLAIN
#undef EBIV_PIN
#undef EBIV_UPDATE
  }

  // Skip macroblocks from `from` on, up to the next other mode, which it
  // returns, or up to `stop` (mbSkip); *at is the macroblock it stopped at.
  // Four modes are looked up at once.
  EBIV_DEV uint32_t skips(int from, int* at) {
    const uint32_t row = rowOf(ctxMBMode);
    int k = from;
    uint32_t mode = mbSkip;
#pragma unroll 1
    while (k < stop) {
      uint32_t x[4] = {x0, x1, x2, x3}, bad = (uint32_t)(stop - 4 - k);
      uint32_t cur = __funnelshift_l(lo, hi, off);
      int32_t after = rem;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint4 e = entryAt(row | (x[j] & kBucketMask));
        x[j] = e.x * (x[j] >> kScaleBits) + x[j] - e.y;
        take(x[j], cur, after);
        bad |= e.z | (x[j] - kLower);
      }
      if ((int32_t)(bad | (uint32_t)after) >= 0) {
        x0 = x[0];
        x1 = x[1];
        x2 = x[2];
        x3 = x[3];
        off += (uint32_t)(rem - after);
        rem = after;
        refill();
        k += 4;
        continue;
      }
      mode = sym(ctxMBMode);
      if (stop == 0) return mbSkip;
      if (mode != mbSkip) break;
      k++;
    }
    *at = k;
    return mode;
  }

  // Takes up a tile's decoding (buf: its bytes); false when a state is below
  // kLower or at 2^31 and above, as no encoder leaves it (a symbol of one in
  // between takes at most two bytes and leaves one).  The bytes down to the
  // first aligned word are read one by one, so no load reaches past the tile.
  EBIV_DEV bool set(const uint8_t* buf, const ChainState& s, const EntropyTables* tables) {
    t = tables;
    x0 = s.x0;
    x1 = s.x1;
    x2 = s.x2;
    x3 = s.x3;
    int pos = s.pos;
    if (min(min(x0, x1), min(x2, x3)) < kLower || ((x0 | x1 | x2 | x3) >> 31) != 0) return false;
    rem = 8 * pos;
    const int head = min(pos, (int)((uintptr_t)(buf + pos) & 3));  // bytes above the last aligned word
    hi = 0;
    for (int k = 0; k < head; k++) hi = hi << 8 | (uint32_t)__ldg(buf + --pos);
    off = 32 - 8 * (uint32_t)head;
    wp = reinterpret_cast<const uint32_t*>((uintptr_t)(buf + pos) & ~(uintptr_t)3) - 1;
    lo = __ldg(wp);
    nw = __ldg(--wp);
    refill();
    return true;
  }

  // The chain of a whole tile: len bytes at buf, its log into tileLog.
  EBIV_DEV bool run(const uint8_t* buf, uint32_t len, const EntropyTables& tables, int inter, int total,
                    uint16_t* tileLog, int logEntries, uint32_t* offsets, int tileWidth = 0, int stride = 0) {
    return len >= (uint32_t)(kStates * 4) &&
           run(buf, initialState(buf, len), tables, inter, 0, total, tileLog, logEntries, offsets, tileWidth, stride);
  }
  // The chain of a tile's macroblocks from `from` on, where its decoder stands
  // at s, up to macroblock `total`.  Its log goes into tileLog, which has
  // logEntries entries, or as many for each macroblock (kRooms; the tile is
  // tileWidth macroblocks wide, the frame `stride`, and tileLog the room of the
  // tile's first).  offsets (kSkipOffset everywhere before) gets the first entry
  // of each macroblock that is not skip, or the number of its entries (kRooms).
  // False when macroblocks (failure()) are left to the full chain: a
  // symbol failed, or there was no room for the most entries that could follow.
  EBIV_DEV bool run(const uint8_t* buf, const ChainState& s, const EntropyTables& tables, int inter, int from, int total,
                    uint16_t* tileLog, int logEntries, uint32_t* offsets, int tileWidth = 0, int stride = 0) {
    log = lp = first = tileLog;
    entries = logEntries;
    width = rowEnd = tileWidth;
    gap = (stride - tileWidth) * entries;
    mbOff = offsets;
    stop = total;
    intraOnly = !inter;
    mb = from;
    if (!set(buf, s, &tables)) return false;
#pragma unroll 1
    for (; mb < stop; mb++) {
      uint32_t mode = mbIntra;
      if (inter) {
        mode = skips(mb, &mb);
        if (mode == mbSkip) break;
      }
      open();
      if (!kRooms && room() < kPlainMBEntries + kLastEntries) return false;
      if (inter) put(kLogValue | mode << kLogShift);
      uint32_t cbp = kNumCBP - 1;
      if (mode != mbIntra) {
        put(kLogValue | sym(ctxRef) << kLogShift);
        const uint32_t part = sym(ctxPart);
        put(kLogValue | part << kLogShift);
        const int nv = part == partWhole ? 2 : (part == part8x8 ? 8 : 4);
#pragma unroll 1
        for (int i = 0; i < nv; i++) putValue(classValue((i & 1) ? ctxMVClassY : ctxMVClassX));
        cbp = sym(ctxCBP);
        put(kLogValue | cbp << kLogShift);
      }
      // The coded blocks in bitstream order: luma, Cb, Cr; an intra one's mode
      // before each luma block and before Cb.
      uint32_t tx = 0, blocks = 0;
      if (cbp & cbpLuma) {
        tx = min(sym(ctxTxSize), 2u);  // alphabet size 3
        put(kLogValue | tx << kLogShift);
        blocks = (tx + 1) | ((16u >> (2 * tx)) - 1) << 4;
      }
      const uint32_t chroma = (cbp & cbpCb ? 1u : 0u) + (cbp & cbpCr ? 1u : 0u);
      if (chroma) blocks |= (4u | (chroma - 1) << 4) << (cbp & cbpLuma ? 8 : 0);
      if (mode == mbIntra) blocks = intraQueue(tx);
      if (blocks != 0 && stop != 0) tokens(blocks);
      if (stop == 0) return false;
      close();
    }
    return stop == total;
  }
  // After run(): where the decoder stands behind the last macroblock.
  EBIV_DEV ChainState state() const { return ChainState{x0, x1, x2, x3, rem >> 3}; }
  // After a run() from macroblock `from` on that failed.  In a frame of intra
  // macroblocks only, the failing symbol may be up to three before the one
  // where that was noticed, at the end of the macroblock before.
  EBIV_DEV ChainFailure failure(int from) const {
    return ChainFailure{intraOnly && mb > from ? mb - 1 : mb, mb + 1, rem >> 3};
  }
};
using Chain = ChainOf<false>;

}  // namespace dev
}  // namespace ebiv
