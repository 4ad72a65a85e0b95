// The symbol chain with the log as the entropy kernel has it: each macroblock's
// entries in a room of their own inside the frame's coefficient regions
// (kSymPerMB bytes), for every tile of every packet the planner accepts, and
// taken up again behind macroblocks that it leaves, against the plain decoder
// of chain_test.cpp.  Rooms of other tiles and of
// skip macroblocks, and a room behind its entries, stay as they were; the
// frame's regions are allocated at their exact size.
//
// Input as chain_test.cpp's.  Output: one summary line.
#define main chainTestMain
#include "chain_test.cpp"
#undef main

#include <algorithm>

namespace {

using dev::ChainState;

constexpr int kRoom = kSymPerMB / 2;
constexpr uint16_t kUntouched = 0xBEEF;
// A macroblock of at most this many entries always has room, however many of
// them are escapes: behind u entries of a 16x16 block's escapes, four each,
// there are u / 4 positions done, and the rest takes 515 - u / 2 at most.
constexpr int kAlwaysFits = 345;

struct Rooms {
  int cols;
  std::unique_ptr<uint16_t[]> log;
  Rooms(int c, int rows) : cols(c), log(new uint16_t[(size_t)c * rows * kRoom]) {
    std::fill_n(log.get(), (size_t)c * rows * kRoom, kUntouched);
  }
  uint16_t* at(int x, int y) { return log.get() + ((size_t)y * cols + x) * kRoom; }
};

long compared = 0, small = 0, logged = 0, dense = 0, stopped = 0, resumed = 0;

ChainState stateOf(const Plain& p) {
  auto x = [&](int i) { return p.x[(p.at + i) & 3]; };
  return ChainState{x(0), x(1), x(2), x(3), p.pos};
}
bool same(const ChainState& a, const ChainState& b) {
  return a.x0 == b.x0 && a.x1 == b.x1 && a.x2 == b.x2 && a.x3 == b.x3 && a.pos == b.pos;
}

// As the kernel decodes a tile: the chain as far as it goes, the plain decoder
// for the macroblocks that it leaves, the chain again behind them.
const char* sameRooms(const PayloadPlan& p, const TileRange& r, const uint8_t* pkt, bool inter,
                      const dev::EntropyTables& tables, const Geometry& geo) {
  const int tw = r.mbX1 - r.mbX0, total = tw * (r.mbY1 - r.mbY0);
  const uint8_t* const buf = pkt + r.offset;
  Plain want(p.tables, buf, (int)r.length);
  tiles++;
  if (want.err) {  // too short for the states: nothing runs
    failing++;
    return nullptr;
  }
  std::vector<ChainState> before;  // where the plain decoder stands before each macroblock
  std::vector<size_t> at;
  for (int k = 0; k < total && !want.err; k++) {
    before.push_back(stateOf(want));
    at.push_back(want.log.size());
    want.run(inter, 1);
  }
  failing += want.err;
  const int good = (int)before.size() - (want.err ? 1 : 0);  // macroblocks without an error
  before.push_back(stateOf(want));
  at.push_back(want.log.size());
  int largest = 0;
  for (int k = 0; k < good; k++) largest = std::max(largest, (int)(at[(size_t)k + 1] - at[(size_t)k]));
  Rooms rooms(geo.mbCols, geo.mbRows);
  std::vector<uint32_t> entries((size_t)total, dev::kSkipOffset);
  std::vector<char> mine((size_t)total, 0);  // logged by the chain
  ChainState st = before[0];
  int done = 0;
  long left = 0;
  while (done < total) {
    int upTo = total, next = 0;
    dev::ChainOf<true> d;
    bool again = false;
    while (!d.run(buf, st, tables, inter, done, upTo, rooms.at(r.mbX0, r.mbY0), kRoom, entries.data(), tw, geo.mbCols)) {
      if (again) return "the second run failed";
      next = d.failure(done).next;
      upTo = d.failure(done).reached;
      if (upTo < done || upTo >= next || next - upTo > 2) return "no progress";
      if (upTo == done) break;
      again = true;
    }
    if (upTo > good) return "decoded beyond an error";
    if (upTo > done) {
      if (!same(d.state(), before[(size_t)upTo])) return "another state behind the last macroblock";
      std::fill(mine.begin() + done, mine.begin() + upTo, 1);
    }
    resumed += done > 0 && upTo > done;
    done = upTo;
    if (done == total) break;
    left += next - done;
    if (next > good) {  // the plain decoder meets the error there
      if (!want.err) return "left behind the end";
      stopped++;
      break;
    }
    std::fill(entries.begin() + done, entries.begin() + next, dev::kDecodedOffset);
    done = next;
    st = before[(size_t)done];
  }
  if (want.err && done > good) return "no error";
  // Without an error only macroblocks with no room are left, and in a frame of intra macroblocks the one before.
  if (!want.err && !want.low && left && largest <= kAlwaysFits) return "left although it fits";
  dense += !want.err && !want.low && left;
  compared++;
  small += total <= 6 && std::count(mine.begin(), mine.end(), 1) == total && !want.log.empty();
  for (int y = 0; y < geo.mbRows; y++)
    for (int x = 0; x < geo.mbCols; x++) {
      const bool inside = x >= r.mbX0 && x < r.mbX1 && y >= r.mbY0 && y < r.mbY1;
      const size_t k = inside ? (size_t)((y - r.mbY0) * tw + x - r.mbX0) : 0;
      if (inside && !mine[k]) continue;
      const uint16_t* const room = rooms.at(x, y);
      int used = 0;
      if (inside) {
        const bool skip = want.off[k] == dev::kSkipOffset;
        if (skip != (entries[k] == dev::kSkipOffset)) return "skip differs";
        if (!skip) {
          used = (int)entries[k];
          logged++;
          if (used != (int)(at[k + 1] - at[k])) return "number of entries differs";
          if (std::memcmp(room, want.log.data() + at[k], 2 * (size_t)used)) return "entries differ";
          used = std::min(kRoom, used + 1);  // the next macroblock's transform size may stand there
        }
      }
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
  std::printf("tiles %ld failing %ld dense %ld compared %ld small %ld logged %ld stopped %ld resumed %ld\n", tiles, failing,
              dense, compared, small, logged, stopped, resumed);
  return 0;
}
