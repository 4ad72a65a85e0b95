// The symbol chain of the entropy kernel (govid_gb300/csrc/symbol_chain.h, the
// same code compiled for the host) against a plain restatement of the decoder
// it speeds up (ebiv/rans.go:222-304 and the grammar's context choices,
// ebiv/decode_intra.go:121-167, ebiv/decode_inter.go:8-62,
// ebiv/residual.go:79-126, ebiv/mv.go:75-128): for every tile of every packet
// the planner accepts, the log and each macroblock's first entry are the same,
// or the chain leaves the tile to the full chain for a reason that the plain
// decoder confirms, with the decoder's own log size and with one that some
// tiles overflow.  The packet, the log and
// the offsets are allocated at their exact sizes, so a sanitizer sees every
// access outside them.
//
// Input (binary, little endian): u32 streams; per stream u32 packets; per
// packet u32 length, bytes.  Output: one summary line.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <vector>

#include "container.h"
#include "gpu_types.h"
#include "symbol_chain.h"

using namespace ebiv;

namespace {

struct Plain {
  const DeviceTables& t;
  const uint8_t* buf;
  int pos;
  uint32_t x[4];
  int at = 0;
  bool err = false, low = false;  // a symbol failed; a state started out of range
  std::vector<uint16_t> log;
  std::vector<uint32_t> off;

  Plain(const DeviceTables& tables, const uint8_t* b, int len) : t(tables), buf(b), pos(len) {
    if (len < 16) {
      err = true;
      return;
    }
    for (int i = 3; i >= 0; i--) {
      pos -= 4;
      x[i] = rd32(buf + pos);
      low = low || x[i] < kLower || x[i] >> 31;
    }
  }
  int fail() {
    err = true;
    return 0;
  }
  int sym(int c) {
    if (err) return 0;
    if (!t.used[c]) return fail();
    uint32_t& v = x[at & 3];
    const uint32_t slot = v & (kM - 1);
    int s = 0;
    while (t.start[c][s + 1] <= slot) s++;
    uint32_t n = (uint32_t)(t.start[c][s + 1] - t.start[c][s]) * (v >> kScaleBits) + slot - t.start[c][s];
    while (n < kLower) {
      if (pos == 0) return fail();
      n = n << 8 | buf[--pos];
    }
    v = n;
    at++;
    return s;
  }
  void put(unsigned v) { log.push_back((uint16_t)v); }
  int logged(int c, unsigned kind) {
    const int s = sym(c);
    put(kind | (unsigned)s << dev::kLogShift);
    return s;
  }
  void value(int c) {
    const int cls = sym(c);
    unsigned v = cls > 0;
    for (int k = 1; k < cls; k++) v = v << 1 | (unsigned)sym(ctxBypass);
    put(dev::kLogValue | v >> 8 << dev::kLogShift);
    put(dev::kLogValue | (v & 255u) << dev::kLogShift);
  }
  void block(int plane, int tx) {
    int first = -1, last = -1, pc = 0, kept = 0;
    for (int i = 0; i < 16 << (2 * tx) && !err; i++) {
      const int k = sym(tokenCtx(plane, plane == kPlaneLuma ? tx : 0, bandOf(i), pc));
      if (k == tEOB) break;
      pc = classForMag(k);
      // A token's entry holds the masks of its table entry's low half.
      put((unsigned)k << dev::kLogShift | (unsigned)pc << 4 |
          (k == tZero ? 0u : dev::kLogNonzero | (k == tEscape ? 0u : dev::kENonzero)));
      if (k == tZero) continue;
      if (k == tEscape) value(ctxEscClass);
      // A sign's entry names the class that it keeps, but for an escape's.
      kept = k == tEscape ? 0 : pc;
      if (first >= 0) logged(ctxSign, dev::kLogSign | (unsigned)kept << 4);
      if (first < 0) first = i;
      last = i;
    }
    put(tEOB << dev::kLogShift);
    if (first >= 0 && last - first < kSDHMinSpan) logged(ctxSign, dev::kLogSign);
  }
  void run(bool inter, int total) {
    for (int k = 0; k < total && !err; k++) {
      const int mode = inter ? sym(ctxMBMode) : (int)mbIntra;
      off.push_back(mode == mbSkip ? dev::kSkipOffset : (uint32_t)log.size());
      if (mode == mbSkip) continue;
      if (inter) put(dev::kLogValue | (unsigned)mode << dev::kLogShift);
      int cbp = kNumCBP - 1;
      if (mode == mbInter) {
        logged(ctxRef, dev::kLogValue);
        const int n = kPartCount[logged(ctxPart, dev::kLogValue)];
        for (int i = 0; i < n; i++) {
          value(ctxMVClassX);
          value(ctxMVClassY);
        }
        cbp = logged(ctxCBP, dev::kLogValue);
      }
      if (cbp & cbpLuma) {
        const int tx = logged(ctxTxSize, dev::kLogValue);
        for (int b = 0; b < 16 >> (2 * tx) && !err; b++) {
          if (mode == mbIntra) logged(ctxLumaMode, dev::kLogMode);
          block(kPlaneLuma, tx);
        }
      }
      if (mode == mbIntra) logged(ctxChromaMode, dev::kLogMode);
      if (cbp & cbpCb) block(kPlaneChroma, 1);
      if (cbp & cbpCr) block(kPlaneChroma, 1);
    }
  }
};

long tiles = 0, failing = 0, left = 0, overflowing = 0, entries = 0;

bool sameTile(const PayloadPlan& p, const TileRange& r, const uint8_t* pkt, bool inter, const dev::EntropyTables& tables) {
  const int total = (r.mbX1 - r.mbX0) * (r.mbY1 - r.mbY0);
  Plain want(p.tables, pkt + r.offset, (int)r.length);
  want.run(inter, total);
  tiles++;
  failing += want.err;
  entries += (long)want.log.size();
  for (const int perMB : {kSymPerMB, 24}) {
    const int cap = total * perMB / 2;
    std::unique_ptr<uint16_t[]> log(new uint16_t[(size_t)cap]);
    std::vector<uint32_t> off((size_t)total, dev::kSkipOffset);
    dev::Chain d;
    if (!d.run(pkt + r.offset, r.length, tables, inter, total, log.get(), cap, off.data())) {
      // Left to the full chain: a tile that fails, starts with a state that no
      // encoder leaves, or whose log has no room for the most that a
      // macroblock can take.
      const bool fits = (int)want.log.size() + dev::kMBEntries < cap;
      overflowing += !want.err && !fits;
      left += !want.err && fits;
      if (!want.err && fits && !want.low) return false;
      continue;
    }
    if (want.err || want.off != off || d.count() != (int)want.log.size()) return false;
    if (!want.log.empty() && std::memcmp(log.get(), want.log.data(), 2 * want.log.size())) return false;
  }
  return true;
}

}  // namespace

int main(int argc, char** argv) {
  std::FILE* f = argc == 2 ? std::fopen(argv[1], "rb") : nullptr;
  if (!f) return 2;
  auto u32 = [&] {
    uint32_t v = 0;
    if (std::fread(&v, 4, 1, f) != 1) std::exit(2);
    return v;
  };
  std::unique_ptr<dev::EntropyTables> tables(new dev::EntropyTables);
  for (uint32_t streams = u32(); streams; streams--) {
    TableHistory hist;
    Geometry geo;
    bool ready = false;
    for (uint32_t packets = u32(); packets; packets--) {
      const uint32_t n = u32();
      std::unique_ptr<uint8_t[]> pkt(new uint8_t[n ? n : 1]);
      if (n && std::fread(pkt.get(), 1, n, f) != n) return 2;
      FrameHeader fh;
      if (parseFrameHeader(pkt.get(), n, &fh) || fh.goldenOverride || fh.coding == kCodingRaw) continue;
      const bool key = fh.type == kFrameKey;
      if (!key && !ready) continue;
      if (key && (int64_t)fh.width * fh.height > 1 << 22) continue;
      if (key) geo = Geometry::of(fh.width, fh.height);
      ready = true;
      PayloadPlan p;
      if (planPayload(pkt.get(), fh.bodyOffset, n - fh.bodyOffset, key, geo.mbCols, geo.mbRows, hist, &p)) continue;
      for (int k = 0; k < dev::kBlockKinds; k++) tables->block[k] = dev::blockEntry(k);
      for (int c = 0; c < kNumContexts; c++) {
        const uint16_t* st = p.tables.start[c];
        const bool used = p.tables.used[c] != 0;
        for (int k = 0; k < dev::kSymbols; k++)
          tables->symbol[c * dev::kSymbols + k] =
              used && k < 17 && st[k] < kM ? dev::symbolEntry(c, k, st[k], (uint32_t)(st[k + 1] - st[k]), 0) : dev::sentinelEntry();
        for (uint32_t b = 0; b < 64; b++) {
          int k = 0;
          while (used && st[k + 1] <= b << 6) k++;
          for (uint32_t place = 0; place < (c == ctxSign ? 4u : 1u); place++)
            tables->entry[dev::rowOf(c) / 16 + 4 * b + place] =
                used ? dev::bucketEntry(c, k, st[k], st[k + 1], b, dev::kClassBytes * place) : dev::unusedEntry();
        }
      }
      for (const TileRange& r : p.tiles)
        if (!sameTile(p, r, pkt.get(), fh.coding == kCodingInter, *tables)) {
          std::printf("tile differs: packet of %u bytes, tile at %u of %u bytes\n", n, r.offset, r.length);
          return 1;
        }
    }
  }
  std::printf("tiles %ld failing %ld left %ld overflowing %ld entries %ld\n", tiles, failing, left, overflowing, entries);
  return 0;
}
