// The symbol chain with the log as the entropy kernel has it: each macroblock's
// entries in a room of their own inside the frame's coefficient regions
// (kSymPerMB bytes), for every tile of every packet the planner accepts,
// against the plain decoder of chain_test.cpp.  Rooms of other tiles and of
// skip macroblocks, and a room behind its entries, stay as they were; the
// frame's regions are allocated at their exact size.
//
// Input as chain_test.cpp's.  Output: one summary line.
#define main chainTestMain
#include "chain_test.cpp"
#undef main

namespace {

constexpr int kRoom = kSymPerMB / 2;
constexpr uint16_t kUntouched = 0xBEEF;
// A macroblock of at most this many entries always has room: 21 of its header,
// then at most 560 without escapes, and 115 escapes more (345 entries) fit.
constexpr int kAlwaysFits = 345;

struct Rooms {
  int cols;
  std::unique_ptr<uint16_t[]> log;
  Rooms(int c, int rows) : cols(c), log(new uint16_t[(size_t)c * rows * kRoom]) {
    std::fill_n(log.get(), (size_t)c * rows * kRoom, kUntouched);
  }
  uint16_t* at(int x, int y) { return log.get() + ((size_t)y * cols + x) * kRoom; }
};

long compared = 0, small = 0, macroblocks = 0, dense = 0;

const char* sameRooms(const PayloadPlan& p, const TileRange& r, const uint8_t* pkt, bool inter,
                      const dev::EntropyTables& tables, const Geometry& geo) {
  const int tw = r.mbX1 - r.mbX0, total = tw * (r.mbY1 - r.mbY0);
  Plain want(p.tables, pkt + r.offset, (int)r.length);
  want.run(inter, total);
  tiles++;
  failing += want.err;
  int largest = 0, at = (int)want.log.size();
  for (size_t k = want.off.size(); k-- > 0;)
    if (want.off[k] != dev::kSkipOffset) {
      largest = std::max(largest, at - (int)want.off[k]);
      at = (int)want.off[k];
    }
  Rooms rooms(geo.mbCols, geo.mbRows);
  std::vector<uint32_t> entries((size_t)total, dev::kSkipOffset);
  dev::Chain d;
  const bool whole = d.run(pkt + r.offset, r.length, tables, inter, total, rooms.at(r.mbX0, r.mbY0), kRoom,
                           entries.data(), tw, geo.mbCols);
  if (!whole) {
    if (!want.err && !want.low && largest <= kAlwaysFits) return "left although it fits";
    dense += !want.err && !want.low;
  } else {
    if (want.err) return "a failing tile decoded";
    compared++;
    small += total <= 6 && !want.log.empty();
  }
  std::vector<uint32_t> next(want.off);
  next.push_back((uint32_t)want.log.size());
  for (size_t k = next.size() - 1; k-- > 0;)
    if (next[k] == dev::kSkipOffset) next[k] = next[k + 1];  // where macroblock k's entries would begin
  for (int y = 0; y < geo.mbRows; y++)
    for (int x = 0; x < geo.mbCols; x++) {
      const bool inside = x >= r.mbX0 && x < r.mbX1 && y >= r.mbY0 && y < r.mbY1;
      const int k = inside ? (y - r.mbY0) * tw + x - r.mbX0 : 0;
      const uint16_t* const room = rooms.at(x, y);
      int used = 0;
      if (inside && whole) {
        if ((want.off[(size_t)k] == dev::kSkipOffset) != (entries[(size_t)k] == dev::kSkipOffset)) return "skip differs";
        if (want.off[(size_t)k] != dev::kSkipOffset) {
          used = (int)entries[(size_t)k];
          macroblocks++;
          if (used != (int)(next[(size_t)k + 1] - want.off[(size_t)k])) return "number of entries differs";
          if (std::memcmp(room, want.log.data() + want.off[(size_t)k], 2 * (size_t)used)) return "entries differ";
          used = std::min(kRoom, used + 1);  // the next macroblock's transform size may stand there
        }
      }
      if (!inside || whole)
        for (int i = used; i < kRoom; i++)
          if (room[i] != kUntouched) return "written outside the macroblock's entries";
    }
  return nullptr;
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
      if ((!key && !ready) || (key && (int64_t)fh.width * fh.height > 1 << 20)) continue;
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
        if (const char* what = sameRooms(p, r, pkt.get(), fh.coding == kCodingInter, *tables, geo)) {
          std::printf("%s: packet of %u bytes, tile at %u of %u bytes\n", what, n, r.offset, r.length);
          return 1;
        }
    }
  }
  std::printf("tiles %ld failing %ld dense %ld compared %ld small %ld macroblocks %ld\n", tiles, failing, dense, compared,
              small, macroblocks);
  return 0;
}
