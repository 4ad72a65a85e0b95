// GB300 (sm_103a) EBIV decode kernels.
//
// Stage A  kEntropy   one warp per tile, up to four tiles of one frame per
//                     CTA sharing the frame's symbol tables: one thread runs
//                     the tile's symbol chain (symbol_chain.h) into the
//                     macroblocks' logs, from which kParseMB makes one MBRec
//                     per macroblock plus sparse levels; macroblocks that the
//                     chain leaves (a symbol fails, no room for the log) are
//                     decoded by the whole warp in lockstep, records and
//                     levels included (leftTile, fullChain).
// Stage B1 kInterRecon one warp per macroblock of an inter frame: motion
//                     compensation (ebiv/motioncomp.go) from the last or
//                     golden reference plus dequantized inverse DCT residual
//                     (ebiv/quant.go:72-80, ebiv/transform.go:129-194).
// Stage B2 kIntraRecon one or two CTAs per tile: intra macroblocks along
//                     their true dependencies only, a dataflow schedule over
//                     the 4x4-block diagonal steps (ebiv/predict.go:50-219).
//
// Waits are __syncwarp/__syncthreads barriers inside one CTA, and in
// kIntraRecon polls of progress bytes written by warps of the same CTA, each
// bounded (IntraSync); no kernel spins on memory written by another CTA.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "gpu_types.h"
#include "symbol_chain.h"

namespace ebiv {
namespace dev {

constexpr unsigned kFull = 0xffffffffu;

// Per transform size and scan position: row-major index (bits 0-7) and the
// offset of the position's band in the symbol-table rows, bandOf(i) *
// kGroupBytes (from bit 8).  One entry past each scan is zero, so the next
// position's entry can always be loaded.
__constant__ uint32_t cScanRow[3][257];
// The same positions for lanes that read different ones.
__device__ uint8_t gScan[3][256];
// 2^13-scaled DCT-II basis, [k*n + i], per transform size.  Global memory:
// the transforms read it with a different index in every lane, which the
// L1 path serves in one pass and the constant cache would serialise.
__device__ __align__(16) int32_t gDct[3][256];
__constant__ int32_t cTaps[4][4] = {{0, 64, 0, 0}, {-6, 55, 18, -3}, {-8, 40, 40, -8}, {-3, 18, 55, -6}};

__device__ __forceinline__ int clampByteD(int32_t v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }
__device__ __forceinline__ int32_t wadd(int32_t a, int32_t b) { return (int32_t)((uint32_t)a + (uint32_t)b); }
__device__ __forceinline__ int32_t wmul(int32_t a, int32_t b) { return (int32_t)((uint32_t)a * (uint32_t)b); }
__device__ __forceinline__ int clampC(int v, int hi) { return v < 0 ? 0 : (v >= hi ? hi - 1 : v); }
__device__ __forceinline__ int16_t clampMV(int v) {
  return (int16_t)(v < -kMVClampRange ? -kMVClampRange : (v > kMVClampRange ? kMVClampRange : v));
}

// ---------------------------------------------------------------------------
// Stage A: entropy decode
// ---------------------------------------------------------------------------
// One warp per context in turn: lane s holds where symbol s starts and
// writes its entry, then each lane finds two buckets' symbols among them.
__device__ __forceinline__ void buildTables(EntropyTables& T, const DeviceTables& src, int tid, int nthreads) {
  const int lane = tid & 31;
  if (tid < kBlockKinds) T.block[tid] = blockEntry(tid);
  for (int c = tid >> 5; c < kNumContexts; c += nthreads >> 5) {
    const int places = c == ctxSign ? 4 : 1;
    uint4* const e = T.entry + rowOf(c) / 16 + 4 * lane;
    if (!src.used[c]) {
      for (int k = 0; k < places; k++) e[k] = e[4 * 32 + k] = unusedEntry();
      continue;
    }
    const uint32_t start = lane < 17 ? (uint32_t)src.start[c][lane] : 0xFFFFu;
    const uint32_t after = __shfl_down_sync(kFull, start, 1);
    if (lane < kSymbols)
      T.symbol[c * kSymbols + lane] = start < kM ? symbolEntry(c, lane, start, after - start, 0u) : sentinelEntry();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t b = (uint32_t)(lane + 32 * h);
      uint32_t s = 0, st = 0, nx = kM;
#pragma unroll
      for (int k = 1; k < 16; k++) {
        const uint32_t v = __shfl_sync(kFull, start, k);
        if (v <= b << 6) {
          s = (uint32_t)k;
          st = v;
        } else {
          nx = min(nx, v);
        }
      }
      for (int k = 0; k < places; k++) e[4 * 32 * h + k] = bucketEntry(c, (int)s, st, nx, b, kClassBytes * (uint32_t)k);
    }
  }
  __syncthreads();
}

// A tile's rANS decoder as the full chain runs it (ebiv/rans.go:222-304).
// All fields are warp-uniform; the two next stream bytes are prefetched so
// renormalisation rarely waits.  After the first error every symbol decodes
// as 0.
struct WarpChain {
  const uint8_t* buf;
  int32_t pos;
  uint32_t x0, x1, x2, x3;  // states in use order: x0 decodes the next symbol
  uint32_t b1, b2;          // buf[pos-1], buf[pos-2] when present
  int32_t err;
  const EntropyTables* t;

  __device__ __forceinline__ uint32_t byteAt(int i) const { return i >= 0 ? (uint32_t)__ldg(buf + i) : 0u; }
  __device__ __forceinline__ int fail(int e) {
    err = e;
    return 0;
  }

  __device__ __forceinline__ uint4 entryAt(uint32_t offset) const {
    return *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(t->entry) + offset);
  }
  // The next symbol of the context at a row (rowOf).
  __device__ __forceinline__ int symAt(uint32_t row) {
    if (err) return 0;
    const uint32_t x = x0;
    uint4 e = entryAt(row | (x & kBucketMask));
    if (e.z & (kEImpure | kEUnused)) {
      if (e.z & kEUnused) return fail(kErrCorrupt);  // symbol decoded from an unused context
      uint32_t q = 16 * e.y;
      e = entryAt(q);
      for (uint4 n = entryAt(q += 16); (x & (kM - 1)) >= n.y; n = entryAt(q += 16)) e = n;
    }
    return renew(e.x * (x >> kScaleBits) + x - e.y, (int)((e.w >> kLogShift) & 15u));
  }
  // A symbol of ctxBypass, whose two symbols have half of the range each
  // (installBypass, ebiv/rans.go:317-322).
  __device__ __forceinline__ int bypass() {
    if (err) return 0;
    return renew((x0 >> kScaleBits << (kScaleBits - 1)) + (x0 & (kM / 2 - 1)), (int)(x0 >> (kScaleBits - 1) & 1u));
  }
  // Stream bytes for the state behind symbol s, which it returns.
  __device__ __forceinline__ int renew(uint32_t xn, int s) {
    if (xn < kLower) {
      if (pos >= 2 && xn >= (kLower >> 16)) {
        if (xn < (kLower >> 8)) {  // two bytes
          xn = (xn << 16) | (b1 << 8) | b2;
          pos -= 2;
          b1 = byteAt(pos - 1);
          b2 = byteAt(pos - 2);
        } else {  // one byte
          xn = (xn << 8) | b1;
          pos -= 1;
          b1 = b2;
          b2 = byteAt(pos - 2);
        }
      } else {
        while (xn < kLower) {
          if (pos == 0) return fail(kErrCorrupt);  // stream underrun
          pos--;
          xn = (xn << 8) | b1;
          b1 = b2;
          b2 = byteAt(pos - 2);
        }
      }
    }
    x0 = x1;
    x1 = x2;
    x2 = x3;
    x3 = xn;
    return s;
  }
  __device__ __forceinline__ int sym(int ctx) { return symAt(rowOf(ctx)); }
  // Takes up a tile's decoding (b: its bytes).
  __device__ __forceinline__ void set(const uint8_t* b, const ChainState& s, const EntropyTables* tables) {
    buf = b;
    err = 0;
    t = tables;
    x0 = s.x0;
    x1 = s.x1;
    x2 = s.x2;
    x3 = s.x3;
    pos = s.pos;
    b1 = byteAt(pos - 1);
    b2 = byteAt(pos - 2);
  }
  __device__ __forceinline__ ChainState state() const { return ChainState{x0, x1, x2, x3, pos}; }
};

// getRawBits / getClassValue / getMVComponent — ebiv/mv.go:75-128.
__device__ __forceinline__ uint32_t classValue(WarpChain& d, int classCtx) {
  const int cls = d.sym(classCtx);
  uint32_t v = (uint32_t)min(cls, 1);
  for (int i = 1; i < cls; i++) v = v << 1 | (uint32_t)d.bypass();
  return v;
}
__device__ __forceinline__ int unzigzag(uint32_t u) { return (int)(u >> 1) ^ -(int)(u & 1); }
__device__ __forceinline__ int mvComponent(WarpChain& d, int classCtx) { return unzigzag(classValue(d, classCtx)); }

// decodeBlock (ebiv/residual.go:79-126): the block's nonzero levels are
// written as packed entries after a count word (by lane 0).  row is the row of
// the block's token contexts at band 0 and previous class 0; the band and
// previous class add their offsets.  Returns the count.
__device__ __forceinline__ int entropyBlock(WarpChain& d, uint32_t row, int sz, uint32_t* region, int lane) {
  const uint32_t* sb = cScanRow[sz];
  const int total = 16 << (2 * sz);
  int first = -1, last = -1, count = 0;
  int32_t sumAbs = 0;
  uint32_t pc = 0;  // previous class * kClassBytes
  uint32_t firstPos = 0;
  int32_t firstMag = 0;
  uint32_t cur = sb[0];
  for (int i = 0; i < total; i++) {
    const uint32_t nxt = sb[i + 1];  // next position's entry, loaded early (the table is padded)
    const int t = d.symAt(row + (cur >> 8) + pc);
    if (t == tEOB) break;
    if (t == tZero) {
      pc = 0;
      cur = nxt;
      continue;
    }
    int mag;
    if (t == tEscape) {
      mag = 5 + (int)classValue(d, ctxEscClass);
      pc = 2 * kClassBytes;
    } else {
      mag = t;
      pc = t == tOne ? kClassBytes : 2 * kClassBytes;
    }
    sumAbs = wadd(sumAbs, mag);
    const uint32_t pos = cur & 0xFFu;
    if (first < 0) {
      first = i;
      firstPos = pos;
      firstMag = mag;
    } else {
      if (d.sym(ctxSign) == 1) mag = -mag;
      if (lane == 0) region[1 + count] = pos | ((uint32_t)mag << 8);
    }
    count++;
    last = i;
    cur = nxt;
  }
  if (first >= 0) {
    const bool neg = (last - first >= kSDHMinSpan) ? (sumAbs & 1) == 1 : d.sym(ctxSign) == 1;
    if (lane == 0) region[1] = firstPos | ((uint32_t)(neg ? -firstMag : firstMag) << 8);
  }
  if (lane == 0) region[0] = (uint32_t)count;
  return count;
}

__device__ __forceinline__ uint32_t packMV(int x, int y) { return (uint32_t)(uint16_t)x | ((uint32_t)(uint16_t)y << 16); }
__device__ __forceinline__ int mvX(uint32_t v) { return (int16_t)(v & 0xFFFFu); }
__device__ __forceinline__ int mvY(uint32_t v) { return (int16_t)(v >> 16); }

// The macroblock record being assembled, in registers (see MBRec: word 0
// mode|ref<<8|part<<16|cbp<<24, 1 tx|cmode<<8, 2-5 vectors, 6-9 luma modes,
// 10 nzmask, 11 wmask).
struct Rec {
  uint32_t w0, w1, mv0, mv1, mv2, mv3, lm0, lm1, lm2, lm3, nz, wm;
  __device__ __forceinline__ void clear() { w0 = w1 = mv0 = mv1 = mv2 = mv3 = lm0 = lm1 = lm2 = lm3 = nz = wm = 0; }
  __device__ __forceinline__ void lumaMode(int k, uint32_t m) {
    const uint32_t v = m << ((k & 3) * 8);
    const int w = k >> 2;
    if (w == 0) lm0 |= v;
    else if (w == 1) lm1 |= v;
    else if (w == 2) lm2 |= v;
    else lm3 |= v;
  }
  __device__ __forceinline__ void setMV(int i, uint32_t v) {
    if (i == 0) mv0 = v;
    else if (i == 1) mv1 = v;
    else if (i == 2) mv2 = v;
    else mv3 = v;
  }
  // Lanes 0-2 store the 48-byte record as three 16-byte words.
  __device__ __forceinline__ void store(MBRec* dst, int lane) const {
    uint4 v;
    if (lane == 0) v = make_uint4(w0, w1, mv0, mv1);
    else if (lane == 1) v = make_uint4(mv2, mv3, lm0, lm1);
    else v = make_uint4(lm2, lm3, nz, wm);
    if (lane < 3) reinterpret_cast<uint4*>(dst)[lane] = v;
  }
};

// Neighbourhood of the macroblock being decoded: availability within the
// tile, the left neighbour's vector/level (registers) and the row above.
struct Nbr {
  bool aOK, bOK, arOK;
  uint32_t mvA, mvB, mvC;  // left, above, above-right (or above-left)
  bool cOK;
};

// predictMV — ebiv/mv.go:21-52 (neighbours within the tile).  The median of
// three runs on both packed 16-bit components at once: median(a, b, c) =
// max(min(a, b), min(max(a, b), c)); unavailable neighbours are zero.
__device__ __forceinline__ uint32_t predictMV(const Nbr& n) {
  if (!n.aOK && !n.bOK && !n.cOK) return 0;
  if (n.aOK && !n.bOK && !n.cOK) return n.mvA;
  if (!n.aOK && n.bOK && !n.cOK) return n.mvB;
  const uint32_t lo = __vmins2(n.mvA, n.mvB), hi = __vmaxs2(n.mvA, n.mvB);
  return __vmaxs2(lo, __vmins2(hi, n.mvC));
}

// The coded blocks of one macroblock in bitstream order: nLuma luma blocks
// (each preceded by its intra mode when intra), then Cb (preceded by the
// chroma intra mode when intra) and Cr when present.
struct BlockPlan {
  int nLuma, tx;
  bool intra, cb, cr;
};

// The block loop of a macroblock.  Returns how many blocks completed before
// an error; *nzOut gets the nonzero mask (bit k luma block k, 16 Cb, 17 Cr).
__device__ __forceinline__ int entropyBlocks(WarpChain& d, Rec& r, const BlockPlan& p, uint32_t* coef, int lane,
                                             uint32_t* nzOut) {
  const int nEnt = p.nLuma + (p.cb ? 1 : 0) + (p.cr ? 1 : 0);
  const int bw = (16 << (2 * p.tx)) + 1;  // words per luma block region
  const uint32_t lumaRow = (uint32_t)(p.tx * kNumBands) * kGroupBytes;
  int done = 0;
  uint32_t nz = 0;
#pragma unroll 1
  for (int e = 0; e < nEnt; e++) {
    uint32_t row;
    int sz;
    uint32_t* region;
    uint32_t bit;
    if (e < p.nLuma) {
      sz = p.tx;
      if (p.intra) r.lumaMode(e, (uint32_t)d.sym(ctxLumaMode));
      row = lumaRow;
      region = coef + e * bw;
      bit = 1u << e;
    } else {
      sz = 1;
      const bool isCb = p.cb && e == p.nLuma;
      if (isCb && p.intra) r.w1 |= (uint32_t)d.sym(ctxChromaMode) << 8;
      row = rowOf(ctxTokenBase + kLumaTokenCtx);
      region = coef + (isCb ? kCoefCb : kCoefCr);
      bit = isCb ? (1u << 16) : (1u << 17);
    }
    const int cnt = entropyBlock(d, row, sz, region, lane);
    if (d.err) break;
    if (cnt) nz |= bit;
    done++;
  }
  *nzOut = nz;
  return done;
}

// Intra macroblock header (decodeLumaMB, ebiv/decode_intra.go:137-150): the
// transform size; the blocks follow.
__device__ __forceinline__ void intraHeader(WarpChain& d, Rec& r, BlockPlan* p) {
  int tx = d.sym(ctxTxSize);
  if (tx >= 3) tx = 0;  // alphabet size 3: unreachable
  r.w0 = kRecIntra;
  r.w1 = (uint32_t)tx;
  p->tx = tx;
  p->nLuma = 16 >> (2 * tx);
  p->intra = p->cb = p->cr = true;
}

// Inter-frame macroblock header after the mode (decodeInterMB,
// ebiv/decode_inter.go:8-62): reference, partition, vector deltas,
// coded-block pattern, transform size.  The vectors are stored as deltas
// (x, y as int16) in the record; predictVectors turns them into vectors
// (no context depends on a vector, so the chain never needs them).  Returns
// 1 when the blocks of *p follow, 0 when the macroblock ends here (an error).
__device__ __forceinline__ int interHeader(WarpChain& d, Rec& r, int mode, BlockPlan* p, bool* intra) {
  if (mode == mbIntra) {
    *intra = true;
    intraHeader(d, r, p);
    return d.err ? 0 : 1;
  }
  if (mode != mbInter) {
    d.err = kErrCorrupt;
    return 0;
  }
  const int refSel = d.sym(ctxRef);
  int part = d.sym(ctxPart);
  if (part >= kNumPartModes) part = 0;  // alphabet size 4: unreachable
  const int np = part == partWhole ? 1 : (part == part8x8 ? 4 : 2);
#pragma unroll 1
  for (int i = 0; i < np; i++) {
    const int dx = mvComponent(d, ctxMVClassX);
    const int dy = mvComponent(d, ctxMVClassY);
    r.setMV(i, packMV(dx, dy));
  }
  if (d.err) return 0;
  const int cbp = d.sym(ctxCBP);
  r.w0 = kRecInter | ((uint32_t)refSel << 8) | ((uint32_t)part << 16) | ((uint32_t)cbp << 24);
  if (d.err) return 0;
  int tx = 0, nb = 0;
  if (cbp & cbpLuma) {
    tx = d.sym(ctxTxSize);
    if (tx >= 3) tx = 0;
    if (d.err) return 0;
    r.w1 = (uint32_t)tx;
    nb = 16 >> (2 * tx);
  }
  p->tx = tx;
  p->nLuma = nb;
  p->intra = false;
  p->cb = (cbp & cbpCb) != 0;
  p->cr = (cbp & cbpCr) != 0;
  return 1;
}

// Write mask after the blocks (decodeLumaMB/decodeChromaMB and
// reconInterMB, ebiv/decode_intra.go:150-187, ebiv/decode_inter.go:63-118):
// an intra macroblock keeps the blocks completed before an error; an inter
// macroblock whose coded luma failed writes only the luma blocks decoded.
__device__ __forceinline__ uint32_t writeMask(const BlockPlan& p, int done) {
  const int nb = p.nLuma;
  if (p.intra) {
    uint32_t w = (1u << min(done, nb)) - 1;
    if (done > nb) w |= 1u << 16;
    if (done > nb + 1) w |= 1u << 17;
    return w;
  }
  if (done < nb) return (1u << done) - 1;
  const int cbEntry = p.cb ? nb : -1;
  const int crEntry = p.cr ? nb + (p.cb ? 1 : 0) : -1;
  uint32_t w = 0xFFFFu;  // coded luma complete, or motion-compensated luma
  if (cbEntry < 0 || done > cbEntry) w |= 1u << 16;
  if (crEntry < 0 || done > crEntry) w |= 1u << 17;
  return w;
}

// Vector prediction over a tile whose chain is done (predictMV,
// ebiv/mv.go:21-52, neighbours inside the tile; decodeInterMB's use of it,
// ebiv/decode_inter.go:8-62).  A macroblock's vector needs the final
// vectors of its left, above and above-right (or above-left) neighbours, so
// the tile runs as a wavefront: in a pass of 32 rows lane k takes row k and,
// at step t, column t - 2k.  The left neighbour is the lane's own result of
// the step before; the row above comes from lane k-1 by shuffle (its
// results of the last three steps are columns x-1, x, x+1), and for lane 0
// from the previous pass's last row, in the frame's vector grid.  A skip
// macroblock takes the prediction; an inter one adds its deltas (partition 0 to
// the prediction, zero for the golden reference; later partitions to partition
// 0), clamped as the chain would have.  Records past `done` are not touched.
// For tiles wider than kRowMax; predictVectorsShared has the others.
__device__ void predictVectors(const FrameDesc* fp, int tile, int done, int lane) {
  const int mbCols = fp->mbCols;
  MBRec* const recs = fp->mbrec;
  uint32_t* const gmv = reinterpret_cast<uint32_t*>(fp->mvgrid);
  const TileRange tr = fp->tiles[tile];
  const int x0 = tr.mbX0, y0 = tr.mbY0, tw = tr.mbX1 - x0, th = tr.mbY1 - y0;
  for (int p0 = 0; p0 < th; p0 += 32) {
    const int ry = p0 + lane;
    const int nrows = min(32, th - p0);
    const int steps = tw + 2 * (nrows - 1);
    const bool lastRowOfPass = lane == 31 && p0 + 32 < th;
    const uint32_t* upRow = gmv + (size_t)(y0 + p0 - 1) * mbCols + x0;
    uint32_t* nextUp = gmv + (size_t)(y0 + p0 + 31) * mbCols + x0;
    // Records of this lane's row; written by this warp's chain, so read
    // with coherent loads (never through the read-only path).
    MBRec* const rowRec = recs + (size_t)(y0 + min(ry, th - 1)) * mbCols + x0;
    const int rowDone = ry < th ? min(tw, done - ry * tw) : 0;  // columns of this row the chain reached
    uint32_t h1 = 0, h2 = 0, h3 = 0;  // this lane's results of steps t-1, t-2, t-3
    // Record words 0-3 of a step's macroblock, loaded four steps ahead into
    // one of four registers that nothing touches until its step, so the
    // global-memory latency overlaps the steps between.
    auto recAt = [&](int x) {
      return x >= 0 && x < rowDone ? reinterpret_cast<const uint4*>(rowRec + x)[0] : make_uint4(0u, 0u, 0u, 0u);
    };
    auto step = [&](int t, const uint4& cur) {
      const int rx = t - 2 * lane;
      const bool act = t < steps && rx >= 0 && rx < rowDone;
      uint32_t above = __shfl_up_sync(kFull, h2, 1);
      uint32_t ar = __shfl_up_sync(kFull, h1, 1);
      uint32_t al = __shfl_up_sync(kFull, h3, 1);
      uint32_t out = 0;
      if (act) {
        if (lane == 0 && p0 > 0) {
          above = upRow[rx];
          ar = rx + 1 < tw ? upRow[rx + 1] : 0u;
          al = rx > 0 ? upRow[rx - 1] : 0u;
        }
        uint32_t* const rw = reinterpret_cast<uint32_t*>(rowRec + rx);
        const uint32_t w0 = cur.x;
        const int mode = (int)(w0 & 0xFF);
        if (mode == kRecSkip || mode == kRecInter) {
          Nbr n;
          n.aOK = rx > 0;
          n.bOK = ry > 0;
          n.arOK = n.bOK && rx + 1 < tw;
          n.cOK = n.arOK || (n.bOK && n.aOK);
          n.mvA = h1;
          n.mvB = n.bOK ? above : 0u;
          n.mvC = n.cOK ? (n.arOK ? ar : al) : 0u;
          uint32_t pred = predictMV(n);
          if (mode == kRecSkip) {
            rw[2] = pred;
            out = pred;
          } else {
            const bool golden = ((w0 >> 8) & 0xFF) == refGolden;
            const int part = (int)((w0 >> 16) & 0xFF);
            if (golden) pred = 0;
            const uint32_t v0 = packMV(clampMV(mvX(pred) + mvX(cur.z)), clampMV(mvY(pred) + mvY(cur.z)));
            rw[2] = v0;
            if (part != partWhole) {
              rw[3] = packMV(clampMV(mvX(v0) + mvX(cur.w)), clampMV(mvY(v0) + mvY(cur.w)));
              if (part == part8x8) {
                const uint32_t d2 = rw[4], d3 = rw[5];
                rw[4] = packMV(clampMV(mvX(v0) + mvX(d2)), clampMV(mvY(v0) + mvY(d2)));
                rw[5] = packMV(clampMV(mvX(v0) + mvX(d3)), clampMV(mvY(v0) + mvY(d3)));
              }
            }
            out = golden ? 0u : v0;
          }
        }
        if (lastRowOfPass) nextUp[rx] = out;
      }
      h3 = h2;
      h2 = h1;
      h1 = out;
    };
    const int base = -2 * lane;
    uint4 q0 = recAt(base), q1 = recAt(base + 1), q2 = recAt(base + 2), q3 = recAt(base + 3);
    for (int t = 0; t < steps; t += 4) {
      step(t, q0);
      q0 = recAt(base + t + 4);
      step(t + 1, q1);
      q1 = recAt(base + t + 5);
      step(t + 2, q2);
      q2 = recAt(base + t + 6);
      step(t + 3, q3);
      q3 = recAt(base + t + 7);
    }
    __syncwarp();  // the pass's last row is read by the next pass's lane 0
  }
}

constexpr int kEntropyWarps = kEntropyTilesPerJob;

// One macroblock's grammar (decodeInterMB, ebiv/decode_inter.go:8-62;
// decodeLumaMB / decodeChromaMB, ebiv/decode_intra.go:137-187), run by a warp
// together; the record is written by lanes 0-2 and the coefficient regions by
// lane 0.  Returns 1 when the macroblock is intra and written (an entry of
// the tile's intra list).
__device__ __forceinline__ int decodeMB(WarpChain& d, int inter, MBRec* rec, uint32_t* coef, int lane) {
  int mode = 0;
  if (inter) {
    mode = d.sym(ctxMBMode);
    if (mode == mbSkip) {
      // Skip macroblock (most of an inter frame): a fixed record whose
      // vector predictVectors fills in; nothing else to decode.
      const uint4 a = make_uint4(kRecSkip, 0u, 0u, 0u), z = make_uint4(0u, 0u, 0u, 0u),
                  c = make_uint4(0u, 0u, 0u, kWriteAll);
      if (lane < 3) reinterpret_cast<uint4*>(rec)[lane] = lane == 0 ? a : (lane == 1 ? z : c);
      return 0;
    }
  }
  Rec r;
  r.clear();
  bool intra = !inter;
  uint32_t w = 0;
  BlockPlan p;
  int blocks;
  if (inter) {
    blocks = interHeader(d, r, mode, &p, &intra);
  } else {
    intraHeader(d, r, &p);
    blocks = d.err ? 0 : 1;
  }
  if (blocks) {
    uint32_t nz;
    const int nd = entropyBlocks(d, r, p, coef, lane, &nz);
    r.nz = nz;
    w = writeMask(p, nd);
  }
  r.wm = w;
  r.store(rec, lane);
  return intra && w ? 1 : 0;
}

// A macroblock's log, and the same as 16-byte words: its coefficient region.
constexpr int kLogEntries = kSymPerMB / 2, kLogWords = kSymPerMB / 16;
static_assert(kSymPerMB % 16 == 0 && kPlainMBEntries + kLastEntries <= kLogEntries, "a macroblock's log");
__device__ __forceinline__ uint32_t* coefRegion(const FrameDesc* fp, int idx) {
  return fp->coef + (size_t)idx * kCoefPerMB;
}

// The full chain, by one warp (the frame's tables are in sT): the rANS symbols
// drive the macroblock grammar from macroblock `from` of the tile on, where
// the decoder stands at *st, up to `to`, and every macroblock reached gets its
// record (inter vectors as deltas), its coefficient regions and its flags.
// Returns the macroblocks reached, with *st behind the last one, or with
// st->pos -1 after an error, the macroblock where it came counted.
__device__ __noinline__ int fullChain(const FrameDesc* fp, int tile, const EntropyTables& sT, int lane, ChainState* st,
                                      int from, int to) {
  const TileRange tr = fp->tiles[tile];
  const int tw = tr.mbX1 - tr.mbX0;
  uint8_t* const flags = reinterpret_cast<uint8_t*>(fp->lvgrid) + tr.mbBase;
  WarpChain d;
  d.set(fp->pkt + tr.offset, *st, &sT);
  int k = from;
  while (k < to && !d.err) {
    const int idx = (tr.mbY0 + k / tw) * fp->mbCols + tr.mbX0 + k % tw;
    const int f = decodeMB(d, fp->inter, fp->mbrec + idx, coefRegion(fp, idx), lane);
    if (lane == 0) {
      flags[k] = (uint8_t)f;
      fp->symOff[tr.mbBase + k] = kDecodedOffset;
    }
    k++;
  }
  *st = d.state();
  if (d.err) st->pos = -1;
  return k;
}

// The symbol chain of a tile's macroblocks from `from` to `to`, into their logs.
__device__ __forceinline__ bool runChain(ChainOf<true>& d, const FrameDesc* fp, const TileRange& tr, const EntropyTables& sT,
                                         const ChainState& st, int from, int to) {
  uint16_t* const log = reinterpret_cast<uint16_t*>(coefRegion(fp, tr.mbY0 * fp->mbCols + tr.mbX0));
  return d.run(fp->pkt + tr.offset, st, sT, fp->inter, from, to, log, kLogEntries, fp->symOff + tr.mbBase,
               tr.mbX1 - tr.mbX0, fp->mbCols);
}

// A tile that the symbol chain left, by one warp: the symbol chain as far as
// it goes, the full chain for the macroblocks that it leaves (one with no room
// for its log; one where a symbol fails, which ends the tile), and so on.
// Where the chain failed (f: in its run over the whole tile), the decoder's
// state is not known; another run up to the last complete macroblock finds it.
//
// Two runs take 250 cycles a symbol where the full chain takes 340, and what
// the first one lost in the macroblock where it failed another 125: they pay
// when they got some way.  While it is not four times as far as what was lost,
// as where macroblocks with no room for their log follow one another, the full
// chain is left 1, 3, 7 and more macroblocks behind that one (hold).  Of 1, 2,
// 4 and 8 times, 4 is the best or as good on frames at q0 to q6, by up to 3 %.
// 920 macroblocks of 384 escapes each: 251 ms without this, 169 now (and bypass
// symbols without a table).
__device__ __noinline__ void leftTile(const FrameDesc* fp, int tile, const EntropyTables& sT, int lane, ChainFailure f) {
  const TileRange tr = fp->tiles[tile];
  const int tw = tr.mbX1 - tr.mbX0, total = tw * (tr.mbY1 - tr.mbY0);
  ChainState st = {0u, 0u, 0u, 0u, -1};
  if (tr.length >= (uint32_t)(kStates * 4)) st = initialState(fp->pkt + tr.offset, tr.length);
  int done = 0, hold = 0, upTo = f.reached;
  while (st.pos >= 0 && done < total) {
    if (lane == 0) {
      const int start = st.pos;
      ChainOf<true> d;
#pragma unroll 1
      while (upTo > done) {
        if (runChain(d, fp, tr, sT, st, done, upTo)) {
          st = d.state();
          break;
        }
        f = d.failure(done);
        upTo = f.reached;
      }
      if (upTo < total) {
        hold = start - st.pos >= 4 * (st.pos - f.pos) ? 0 : min(2 * hold + 1, 255);
        f.next = min(total, f.next + hold);
      }
      done = upTo;
    }
    done = __shfl_sync(kFull, done, 0);
    if (done == total) break;
    f.next = __shfl_sync(kFull, f.next, 0);
    st.x0 = __shfl_sync(kFull, st.x0, 0);
    st.x1 = __shfl_sync(kFull, st.x1, 0);
    st.x2 = __shfl_sync(kFull, st.x2, 0);
    st.x3 = __shfl_sync(kFull, st.x3, 0);
    st.pos = __shfl_sync(kFull, st.pos, 0);
    done = fullChain(fp, tile, sT, lane, &st, done, f.next);
    upTo = total;
  }
  const bool err = st.pos < 0;
  // Macroblocks the tile never reached are left untouched by reconstruction.
  for (int k = done + lane; k < total; k += 32) {
    MBRec* r = fp->mbrec + (size_t)(tr.mbY0 + k / tw) * fp->mbCols + tr.mbX0 + k % tw;
    r->mode = kRecNone;
    r->wmask = 0;
    fp->symOff[tr.mbBase + k] = kDecodedOffset;
  }
  if (lane == 0) {
    fp->tileStat[tile] = TileStat{err ? kErrCorrupt : 0, 0, done, 0};
    if (err) atomicExch(fp->status, kErrCorrupt);
  }
}

// A tile, by one warp.
__device__ __forceinline__ void decodeTile(const FrameDesc* fp, int tile, const EntropyTables& sT, int lane) {
  const TileRange tr = fp->tiles[tile];
  const int total = (tr.mbX1 - tr.mbX0) * (tr.mbY1 - tr.mbY0);
  for (int k = lane; k < total; k += 32) fp->symOff[tr.mbBase + k] = kSkipOffset;
  __syncwarp();
  ChainFailure f = {0, 0, 0};
  bool whole = false;
  if (lane == 0 && tr.length >= (uint32_t)(kStates * 4)) {
    ChainOf<true> d;
    whole = runChain(d, fp, tr, sT, initialState(fp->pkt + tr.offset, tr.length), 0, total);
    if (whole) fp->tileStat[tile] = TileStat{0, 0, total, 0};
    else f = d.failure(0);
  }
  if (!__shfl_sync(kFull, whole ? 1 : 0, 0)) leftTile(fp, tile, sT, lane, f);
}

// Entropy jobs: up to kEntropyWarps tiles of one frame per job, one warp per
// tile, sharing the frame's symbol tables.  With a queue counter the grid is
// persistent: each CTA takes jobs (longest first, as listed) until none are
// left, so a round with more jobs than resident CTAs has no second-wave
// tail; without one, CTA b runs job b.  The tables stay for a CTA's next job
// when that is of the same frame: built for every four of the 8160 tiles of a
// 1080p frame, six such frames took 3.14 ms, now 2.81.
__global__ void __launch_bounds__(32 * kEntropyWarps, 2) kEntropy(const FrameDesc* frames, const int4* jobs, int njobs,
                                                                   int* next) {
  extern __shared__ __align__(16) uint8_t sTables[];
  EntropyTables& sT = *reinterpret_cast<EntropyTables*>(sTables);
  __shared__ int sJob;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int frame = -1;  // the frame whose tables sT holds
  for (;;) {
    if (threadIdx.x == 0) sJob = next ? atomicAdd(next, 1) : (int)blockIdx.x;
    __syncthreads();
    const int jb = sJob;
    if (jb >= njobs) return;  // the same for the whole CTA
    const int4 job = jobs[jb];
    const FrameDesc* fp = frames + job.x;
    if (job.x != frame) buildTables(sT, *fp->tables, threadIdx.x, blockDim.x);
    frame = job.x;
    if (warp < job.z) decodeTile(fp, job.y + warp, sT, lane);
    if (!next) return;
    __syncthreads();  // every warp is done with sT and sJob before the next job
  }
}

// Rebuilds the records of the logged macroblocks, one warp per macroblock over
// every macroblock of the launch's tiles (grid.x: job * kEntropyTilesPerJob +
// tile within the job; grid.y * kParseWarps: the macroblock's raster index
// within its tile).  A skip macroblock's record is
// fixed; of another one the warp takes the log out of the macroblock's
// coefficient region into shared memory, whole, before it writes levels there;
// then all of it reads the header, and each lane one log entry at a time of
// its blocks: the entries name their kind, so a lane finds its block, its
// position and its place among the block's levels by counting the ends and
// tokens before it.  A flag per macroblock marks the intra ones for
// kTileFinish.
constexpr int kParseWarps = 8;

struct ParseBlocks {
  uint32_t nz;     // blocks with levels (bit k luma block k, 16 Cb, 17 Cr)
  uint32_t cmode;  // the chroma intra mode
};

// The blocks of plan p whose entries start at entry `from` of the log's first
// 32 (lane's entry of them: v); the log has `end` entries.  Levels go to coef,
// luma modes to lmode (log and lmode in shared memory).
__device__ __forceinline__ ParseBlocks parseBlocks(const uint16_t* log, int end, int from, uint32_t v,
                                                   const BlockPlan& p, uint32_t* coef, uint8_t* lmode, int lane) {
  ParseBlocks out = {0u, 0u};
  const int blocks = p.nLuma + (p.cb ? 1 : 0) + (p.cr ? 1 : 0);
  const int perBlock = (16 << (2 * p.tx)) + 1;  // words per luma block region
  const unsigned before = (1u << lane) - 1u;
  auto entry = [&](int i) { return i < end ? (uint32_t)log[i] : 0u; };
  // The block that is open at the start of a pass: its tokens and nonzero ones
  // so far, the first one's position and magnitude, the last one's position
  // and the parity of the magnitudes.
  int off = 0, done = 0, openTokens = 0, openCount = 0, openFirst = 0, openMag = 0, openLast = 0, openOdd = 0;
  while (done < blocks) {
    const uint32_t kind = v & kLogKind;
    const int sym = (int)((v >> kLogShift) & 7u);
    const bool isEnd = kind == kLogToken && sym == tEOB;
    // The entries of this pass that count: from `from` up to the last block's end.
    unsigned valid = ~((1u << from) - 1u);
    unsigned ends = __ballot_sync(kFull, isEnd) & valid;
    const unsigned last = __ballot_sync(kFull, ((ends >> lane) & 1u) && done + __popc(ends & before) == blocks - 1);
    if (last) {
      valid &= last | (last - 1u);
      ends &= valid;
    }
    const unsigned tokens = __ballot_sync(kFull, kind == kLogToken && !isEnd) & valid;
    const unsigned levels = __ballot_sync(kFull, kind == kLogToken && (v & kLogNonzero) != 0) & valid;
    const bool isLevel = (levels >> lane) & 1u, ends_here = (ends >> lane) & 1u;
    // The entry after this one: a token's sign, the last sign of an end, or an
    // escape's value, whose second half and sign follow.
    const int at = off + lane;
    uint32_t next = isLevel || ends_here ? entry(at + 1) : 0u;
    int mag = sym;
    if (isLevel && sym == tEscape) {
      mag = 5 + (int)((next & 0xFF00u) | entry(at + 2) >> kLogShift);
      next = entry(at + 3);
    }
    const bool minus = (next >> kLogShift) & 1u;
    const unsigned odd = __ballot_sync(kFull, isLevel && (mag & 1));
    // This lane's block and, of the entries before the lane in this pass,
    // those of the block.
    const unsigned endsBefore = ends & before;
    const int blk = done + __popc(endsBefore);
    const bool opened = endsBefore == 0;  // the block may have begun in an earlier pass
    const unsigned mine = opened ? before : before & ~((2u << (31 - __clz(endsBefore))) - 1u);
    const int pos = __popc(tokens & mine) + (opened ? openTokens : 0);
    const unsigned mineLevels = levels & mine;
    const int index = __popc(mineLevels) + (opened ? openCount : 0);
    const int firstLane = (__ffs(mineLevels) - 1) & 31, lastLane = (31 - __clz(mineLevels)) & 31;
    int firstPos = __shfl_sync(kFull, pos, firstLane), firstMag = __shfl_sync(kFull, mag, firstLane);
    int lastPos = __shfl_sync(kFull, pos, lastLane);
    if (opened && openCount) {
      firstPos = openFirst;
      firstMag = openMag;
      if (!mineLevels) lastPos = openLast;
    }
    const bool isLuma = blk < p.nLuma;
    const bool isCb = p.cb && blk == p.nLuma;
    uint32_t* const region = coef + (isLuma ? blk * perBlock : (isCb ? kCoefCb : kCoefCr));
    const uint8_t* const scan = gScan[isLuma ? p.tx : 1];
    uint32_t bit = 0;
    if (isLevel) {
      if (index > 0) region[1 + index] = (uint32_t)scan[pos] | (uint32_t)(minus ? -mag : mag) << 8;
    } else if (ends_here) {
      region[0] = (uint32_t)index;
      if (index > 0) {
        const bool hidden = lastPos - firstPos >= kSDHMinSpan;
        const bool neg = hidden ? ((__popc(odd & mine) + (opened ? openOdd : 0)) & 1) != 0 : minus;
        region[1] = (uint32_t)scan[firstPos] | (uint32_t)(neg ? -firstMag : firstMag) << 8;
        bit = isLuma ? 1u << blk : (isCb ? 1u << 16 : 1u << 17);
      }
    } else if (kind == kLogMode && ((valid >> lane) & 1u) && isLuma) {
      lmode[blk] = (uint8_t)((v >> kLogShift) & 15u);
    }
    const unsigned modes = __ballot_sync(kFull, kind == kLogMode && !isLuma) & valid;
    if (modes) out.cmode = (__shfl_sync(kFull, v, __ffs(modes) - 1) >> kLogShift) & 15u;
    out.nz |= __reduce_or_sync(kFull, bit);
    done += __popc(ends);
    if (last) break;
    // What is open after this pass.
    unsigned tail = valid;
    if (ends) {
      tail &= ~((2u << (31 - __clz(ends))) - 1u);
      openTokens = openCount = openOdd = 0;
    }
    const unsigned tailLevels = levels & tail;
    if (tailLevels) {
      const int f = __shfl_sync(kFull, pos, __ffs(tailLevels) - 1), m = __shfl_sync(kFull, mag, __ffs(tailLevels) - 1);
      if (!openCount) {
        openFirst = f;
        openMag = m;
      }
      openLast = __shfl_sync(kFull, pos, 31 - __clz(tailLevels));
      openCount += __popc(tailLevels);
      openOdd ^= __popc(odd & tail) & 1;
    }
    openTokens += __popc(tokens & tail);
    off += 32;
    from = 0;
    if (off >= end) break;  // unreachable: the log holds every block's end
    v = entry(off + lane);
  }
  return out;
}

__global__ void __launch_bounds__(32 * kParseWarps) kParseMB(const FrameDesc* frames, const int4* jobs, int njobs) {
  __shared__ __align__(16) uint8_t sMode[kParseWarps][16];
  __shared__ uint4 sLog[kParseWarps][kLogWords];
  const int jb = (int)blockIdx.x / kEntropyTilesPerJob, tj = (int)blockIdx.x % kEntropyTilesPerJob;
  if (jb >= njobs) return;
  const int4 job = jobs[jb];
  if (tj >= job.z) return;
  const FrameDesc* fp = frames + job.x;
  const int tile = job.y + tj;
  const TileRange tr = fp->tiles[tile];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tw = tr.mbX1 - tr.mbX0, total = tw * (tr.mbY1 - tr.mbY0);
  const int k = (int)blockIdx.y * kParseWarps + warp;
  if (k >= total) return;
  const int idx = (tr.mbY0 + k / tw) * fp->mbCols + tr.mbX0 + k % tw;
  uint4* const words = reinterpret_cast<uint4*>(fp->mbrec + idx);
  uint8_t* const flags = reinterpret_cast<uint8_t*>(fp->lvgrid) + tr.mbBase;
  const uint32_t entries = fp->symOff[tr.mbBase + k];
  if (entries == kDecodedOffset) return;
  if (entries == kSkipOffset) {
    if (lane < 3) words[lane] = make_uint4(lane ? 0u : (uint32_t)kRecSkip, 0u, 0u, lane == 2 ? kWriteAll : 0u);
    if (lane == 0) flags[k] = 0;
    return;
  }
  uint32_t* const coef = coefRegion(fp, idx);
  const int end = (int)min(entries, (uint32_t)kLogEntries);
  const uint4* const from = reinterpret_cast<const uint4*>(coef);
  for (int i = lane; 8 * i < end; i += 32) sLog[warp][i] = from[i];
  __syncwarp();
  const uint16_t* const log = reinterpret_cast<const uint16_t*>(sLog[warp]);
  const uint32_t v = lane < end ? (uint32_t)log[lane] : 0u;
  int n = 0;
  auto next = [&]() -> uint32_t { return (__shfl_sync(kFull, v, n++) >> kLogShift) & 255u; };
  auto value = [&]() -> uint32_t {
    const uint32_t high = next();
    return high << 8 | next();
  };
  const int mode = fp->inter ? (int)next() : (int)mbIntra;
  uint32_t w0 = kRecIntra, cbp = kNumCBP - 1;
  uint32_t mv[4] = {0u, 0u, 0u, 0u};
  if (mode != mbIntra) {
    const uint32_t ref = next(), part = next();
    const int np = part == partWhole ? 1 : (part == part8x8 ? 4 : 2);
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (i < np) {
        const int x = unzigzag(value()), y = unzigzag(value());
        mv[i] = packMV(x, y);
      }
    cbp = next();
    w0 = kRecInter | ref << 8 | part << 16 | cbp << 24;
  }
  BlockPlan p;
  p.tx = 0;
  p.nLuma = 0;
  p.intra = mode == mbIntra;
  p.cb = (cbp & cbpCb) != 0;
  p.cr = (cbp & cbpCr) != 0;
  if (cbp & cbpLuma) {
    p.tx = (int)min(next(), 2u);
    p.nLuma = 16 >> (2 * p.tx);
  }
  uint8_t* const lmode = sMode[warp];
  if (lane < 4) reinterpret_cast<uint32_t*>(lmode)[lane] = 0;
  __syncwarp();
  const ParseBlocks b = parseBlocks(log, end, n, v, p, coef, lmode, lane);
  __syncwarp();
  if (lane < 3) {
    // Every block is there, so all of the macroblock is written (of an intra
    // one, the blocks that its transform size has).
    const uint32_t wm = p.intra ? ((1u << p.nLuma) - 1u) | 3u << 16 : kWriteAll;
    const uint32_t* lm = reinterpret_cast<const uint32_t*>(lmode);
    words[lane] = lane == 0   ? make_uint4(w0, (uint32_t)p.tx | b.cmode << 8, mv[0], mv[1])
                  : lane == 1 ? make_uint4(mv[2], mv[3], lm[0], lm[1])
                              : make_uint4(lm[2], lm[3], b.nz, wm);
  }
  if (lane == 0) flags[k] = p.intra ? 1 : 0;
}

constexpr int kRowMax = 128;  // tiles at most this many macroblocks wide have their vectors in shared memory
// The same wavefront for a tile of at most kRowMax macroblocks' width, by a
// CTA: the records of a pass of 32 rows are read into shared memory by all
// threads, one warp runs the wavefront there, and all threads write the
// vectors back, those of the partitions after the first added then.  A step
// of the wavefront costs its latency only (a shuffle and a dozen dependent
// instructions), not a record's way from memory: a 30x22 tile took 52 us by
// the old kernel and 18.6 us by this one (cold, the intra list included).
constexpr int kFinishThreads = 256;
struct FinishVectors {
  uint32_t mv[32 * (kRowMax + 1)];  // delta, then vector; rows an odd number of words apart (lane k reads column t - 2k)
  uint8_t kind[32 * kRowMax];       // 0: no vector, 1 skip, 2 + partition shape, + 4 for the golden reference
  uint32_t above[kRowMax];          // the row above the pass
};
__device__ void predictVectorsShared(const FrameDesc* fp, const TileRange& tr, int done, FinishVectors& S, int tid) {
  const int mbCols = fp->mbCols;
  const int tw = tr.mbX1 - tr.mbX0, th = tr.mbY1 - tr.mbY0, pitch = tw | 1;
  MBRec* const recs = fp->mbrec + (size_t)tr.mbY0 * mbCols + tr.mbX0;
  for (int p0 = 0; p0 < th; p0 += 32) {
    const int rows = min(32, th - p0), n = rows * tw;
    for (int i = tid; i < n; i += kFinishThreads) {
      const int r = i / tw, x = i - r * tw;
      uint32_t kind = 0, delta = 0;
      if ((p0 + r) * tw + x < done) {
        const uint4 q = *reinterpret_cast<const uint4*>(recs + (size_t)(p0 + r) * mbCols + x);
        const uint32_t mode = q.x & 0xFF;
        if (mode == kRecSkip) kind = 1;
        if (mode == kRecInter) {
          kind = 2 + ((q.x >> 16) & 3u) + (((q.x >> 8) & 0xFF) == refGolden ? 4 : 0);
          delta = q.z;
        }
      }
      S.mv[r * pitch + x] = delta;
      S.kind[i] = (uint8_t)kind;
    }
    __syncthreads();
    if (tid < 32) {
      const int lane = tid, ry = p0 + lane;
      const bool mine = lane < rows, rowAbove = ry > 0;
      uint32_t left = 0, ar = 0, above = 0, al = 0;  // the row above at columns x + 1, x, x - 1
      const int steps = tw + 2 * (rows - 1);
      for (int t = 0; t < steps; t++) {
        const int x = t - 2 * lane;
        const bool act = mine && x >= 0 && x < tw;
        const uint32_t kind = act ? S.kind[lane * tw + x] : 0u;
        const uint32_t delta = act ? S.mv[lane * pitch + x] : 0u;
        al = above;
        above = ar;
        ar = __shfl_up_sync(kFull, left, 1);
        if (lane == 0 && p0 > 0) {
          al = x > 0 && x <= tw ? S.above[x - 1] : 0u;
          above = x < tw ? S.above[x] : 0u;
          ar = x + 1 < tw ? S.above[x + 1] : 0u;
        }
        uint32_t out = 0;
        if (kind) {
          Nbr n;
          n.aOK = x > 0;
          n.bOK = rowAbove;
          n.arOK = rowAbove && x + 1 < tw;
          n.cOK = n.arOK || (n.bOK && n.aOK);
          n.mvA = left;
          n.mvB = n.bOK ? above : 0u;
          n.mvC = n.cOK ? (n.arOK ? ar : al) : 0u;
          uint32_t v = predictMV(n);
          if (kind > 1) {
            if (kind >= 6) v = 0;
            v = packMV(clampMV(mvX(v) + mvX(delta)), clampMV(mvY(v) + mvY(delta)));
          }
          S.mv[lane * pitch + x] = v;
          out = kind >= 6 ? 0u : v;
        }
        left = out;
      }
    }
    __syncthreads();
    for (int i = tid; i < n; i += kFinishThreads) {
      const int r = i / tw, x = i - r * tw;
      const uint32_t kind = S.kind[i], v0 = S.mv[r * pitch + x];
      if (r == 31) S.above[x] = kind == 0 || kind >= 6 ? 0u : v0;
      if (!kind) continue;
      uint32_t* const w = reinterpret_cast<uint32_t*>(recs + (size_t)(p0 + r) * mbCols + x);
      const int part = kind == 1 ? (int)partWhole : (int)((kind - 2) & 3u);
      auto add = [&](uint32_t d) { return packMV(clampMV(mvX(v0) + mvX(d)), clampMV(mvY(v0) + mvY(d))); };
      w[2] = v0;
      if (part != partWhole) w[3] = add(w[3]);
      if (part == part8x8) {
        w[4] = add(w[4]);
        w[5] = add(w[5]);
      }
    }
    __syncthreads();
  }
}

// After kParseMB: per tile (one CTA per tile of a job) the written intra
// macroblocks listed in raster order, and (inter frames) the tile's vector
// wavefront.
constexpr int kFlagsPerThread = 8;
__global__ void __launch_bounds__(kFinishThreads) kTileFinish(const FrameDesc* frames, const int4* jobs, int njobs) {
  __shared__ FinishVectors sV;
  __shared__ int sWarp[kFinishThreads / 32];
  const int jb = blockIdx.x;
  if (jb >= njobs) return;
  const int4 job = jobs[jb];
  if ((int)blockIdx.y >= job.z) return;
  const FrameDesc* fp = frames + job.x;
  const int tile = job.y + (int)blockIdx.y;
  const TileRange tr = fp->tiles[tile];
  const TileStat st = fp->tileStat[tile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mbCols = fp->mbCols, tw = tr.mbX1 - tr.mbX0;
  const int done = st.done;
  // Each thread counts the flags of eight macroblocks in a row, a warp and
  // then the CTA add the counts up, and each thread lists its own.
  const uint8_t* const flags = reinterpret_cast<const uint8_t*>(fp->lvgrid) + tr.mbBase;
  int base = 0;
  for (int k0 = 0; k0 < done; k0 += kFinishThreads * kFlagsPerThread) {
    const int k = k0 + tid * kFlagsPerThread;
    uint32_t set = 0;
#pragma unroll
    for (int j = 0; j < kFlagsPerThread; j++)
      if (k + j < done && flags[k + j] != 0) set |= 1u << j;
    int upTo = __popc(set);
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFull, upTo, o);
      if (lane >= o) upTo += v;
    }
    if (lane == 31) sWarp[warp] = upTo;
    __syncthreads();
    int at = base + upTo - __popc(set);
    for (int w = 0; w < kFinishThreads / 32; w++) {
      if (w < warp) at += sWarp[w];
      base += sWarp[w];
    }
    for (; set; set &= set - 1) {
      const int m = k + __ffs(set) - 1;
      fp->intraList[tr.mbBase + at++] = (uint32_t)((tr.mbY0 + m / tw) * mbCols + tr.mbX0 + m % tw);
    }
    __syncthreads();
  }
  if (tid == 0) fp->tileStat[tile].intraCount = base;
  if (!fp->inter) return;
  if (tw <= kRowMax) predictVectorsShared(fp, tr, done, sV, tid);
  else if (warp == 0) predictVectors(fp, tile, done, lane);
}

// ---------------------------------------------------------------------------
// Dequantization + inverse DCT of a whole macroblock (warp-cooperative)
// ---------------------------------------------------------------------------
// Every coded block of the macroblock at once (ebiv/quant.go:72-80,
// ebiv/transform.go:129-194): bit k of mask selects luma block k of the
// tx-sized grid, bits 16/17 the Cb/Cr 8x8 blocks.  dense and tmp are
// per-warp scratch of 384 words; on return dense holds the luma residual
// (16x16 raster) in words 0-255 and the Cb and Cr residuals (8x8 raster) in
// 256-319 and 320-383, zero at the positions of unselected blocks.

// The transform is bound by its reads of shared memory and of the cosines, not
// by its products: an output of its own per lane takes two reads a product, so
// a lane makes Q outputs of one column (or row) at once and reads its N levels
// once and the cosines, which lie side by side, four to a load.
template <int N, int Q>
__device__ __forceinline__ void dctColumn(const int32_t* c, const int32_t* in, int32_t* out) {
  int64_t acc[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) acc[q] = 4096;
#pragma unroll 4
  for (int k = 0; k < N; k++) {
    const int64_t d = in[k * N];
#pragma unroll
    for (int q = 0; q < Q; q += 4) {
      const int4 w = __ldg(reinterpret_cast<const int4*>(c + k * N + q));
      acc[q] += w.x * d;
      acc[q + 1] += w.y * d;
      acc[q + 2] += w.z * d;
      acc[q + 3] += w.w * d;
    }
  }
#pragma unroll
  for (int q = 0; q < Q; q++) out[q * N] = (int32_t)(acc[q] >> 13);
}
template <int N, int Q>
__device__ __forceinline__ void dctRow(const int32_t* c, const int32_t* in, int32_t* out) {
  int64_t acc[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) acc[q] = 4096;
#pragma unroll 1
  for (int l = 0; l < N; l += 4) {
    const int4 d4 = *reinterpret_cast<const int4*>(in + l);
    const int64_t d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int q = 0; q < Q; q += 4) {
        const int4 w = __ldg(reinterpret_cast<const int4*>(c + (l + u) * N + q));
        acc[q] += w.x * d[u];
        acc[q + 1] += w.y * d[u];
        acc[q + 2] += w.z * d[u];
        acc[q + 3] += w.w * d[u];
      }
  }
#pragma unroll
  for (int q = 0; q < Q; q += 4)
    *reinterpret_cast<int4*>(out + q) = make_int4((int32_t)(acc[q] >> 13), (int32_t)(acc[q + 1] >> 13),
                                                  (int32_t)(acc[q + 2] >> 13), (int32_t)(acc[q + 3] >> 13));
}
// B blocks of N x N, one behind the other at in, Q outputs a lane; the rows'
// outputs go to a raster of the given pitch, per blocks across.
template <int N, int Q, int B>
__device__ __forceinline__ void dctColumns(const int32_t* in, int32_t* tmp, int lane) {
  constexpr int kParts = N / Q;
  const int32_t* c = gDct[N == 4 ? 0 : (N == 8 ? 1 : 2)];
#pragma unroll 1
  for (int o = lane; o < B * N * kParts; o += 32) {
    const int l = o % N, i0 = o / N % kParts * Q, at = o / (N * kParts) * (N * N);
    dctColumn<N, Q>(c + i0, in + at + l, tmp + at + i0 * N + l);
  }
}
template <int N, int Q, int B>
__device__ __forceinline__ void dctRows(const int32_t* tmp, int32_t* out, int per, int pitch, int lane) {
  constexpr int kParts = N / Q;
  const int32_t* c = gDct[N == 4 ? 0 : (N == 8 ? 1 : 2)];
#pragma unroll 1
  for (int o = lane; o < B * N * kParts; o += 32) {
    const int i = o % N, m0 = o / N % kParts * Q, b = o / (N * kParts);
    dctRow<N, Q>(c + m0, tmp + b * (N * N) + i * N, out + (b / per * N + i) * pitch + b % per * N + m0);
  }
}
__device__ void mbResidual(const uint32_t* coef, int tx, uint32_t mask, int32_t qdc, int32_t qac, int32_t* dense,
                           int32_t* tmp, int lane) {
  const int n = 4 << tx, nn = n * n, per = 4 >> tx, nb = per * per;
#pragma unroll
  for (int i = 0; i < 3; i++) reinterpret_cast<int4*>(dense)[lane + 32 * i] = make_int4(0, 0, 0, 0);
  // Scatter the sparse levels (luma block b at dense[b*nn], Cb at 256, Cr at
  // 320).  Lane b reads block b's count; the entries of all blocks are then
  // fetched as one flattened list, up to four per lane in flight.  The block
  // that owns an entry is found by its rank among the blocks with entries:
  // the number of their first entries up to it.
  const int nEnt = nb + 2;
  int myCount = 0;
  if (lane < nEnt) {
    const bool luma = lane < nb;
    if ((mask >> (luma ? lane : 16 + lane - nb)) & 1)
      myCount = (int)coef[luma ? lane * (nn + 1) : (lane == nb ? kCoefCb : kCoefCr)];
  }
  int incl = myCount;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(kFull, incl, 31);
  const int excl = incl - myCount;
  const unsigned coded = __ballot_sync(kFull, myCount > 0);
  const unsigned below = (1u << lane) - 1u;
  if (myCount > 0) {
    const bool luma = lane < nb;
    const int from = (luma ? lane * (nn + 1) : (lane == nb ? kCoefCb : kCoefCr)) + 1 - excl;  // entry t is at from + t
    tmp[__popc(coded & below)] = from;
    tmp[32 + __popc(coded & below)] = luma ? lane * nn : 256 + (lane - nb) * 64;
  }
  __syncwarp();
  int rank0 = -1;  // the rank of the block that owns the entry before the current 32
  for (int t0 = 0; t0 < total; t0 += 128) {
    uint32_t val[4];
    int dst[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int w0 = t0 + u * 32, t = w0 + lane;
      dst[u] = -1;
      if (w0 < total) {
        const unsigned first = __reduce_or_sync(kFull, myCount > 0 && (unsigned)(excl - w0) < 32u ? 1u << (excl - w0) : 0u);
        if (t < total) {
          const int rank = rank0 + __popc(first & (below << 1 | 1u));
          val[u] = coef[tmp[rank] + t];
          dst[u] = tmp[32 + rank];
        }
        rank0 += __popc(first);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (dst[u] < 0) continue;
      const int pos = (int)(val[u] & 0xFF);
      dense[dst[u] + pos] = wmul((int32_t)val[u] >> 8, pos == 0 ? qdc : qac);
    }
  }
  __syncwarp();
  // Columns: tmp[b][i][l] = sum_k c[k][i] * dense[b][k][l]; rows: out[i][m] =
  // sum_l c[l][m] * tmp[b][i][l], into dense (read only by the column pass,
  // which is complete).  Luma or chroma without a coded block stays zero.
  const bool luma = (mask & 0xFFFFu) != 0, chroma = (mask >> 16) != 0;
  if (luma) {
    if (tx == 0) dctColumns<4, 4, 16>(dense, tmp, lane);
    else if (tx == 1) dctColumns<8, 8, 4>(dense, tmp, lane);
    else dctColumns<16, 8, 1>(dense, tmp, lane);
  }
  if (chroma) dctColumns<8, 4, 2>(dense + 256, tmp + 256, lane);
  __syncwarp();
  if (luma) {
    if (tx == 0) dctRows<4, 4, 16>(tmp, dense, 4, 16, lane);
    else if (tx == 1) dctRows<8, 8, 4>(tmp, dense, 2, 16, lane);
    else dctRows<16, 8, 1>(tmp, dense, 1, 16, lane);
  }
  if (chroma) dctRows<8, 4, 2>(tmp + 256, dense + 256, 1, 8, lane);
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Motion compensation samples (clamped form of ebiv/motioncomp.go:49-97)
// ---------------------------------------------------------------------------
// A macroblock's residual between kInterRecon phase 0 and its consumer
// (phase 1, or the intra stage), stored over its coefficient region.  When
// every value fits in 16 bits (any real stream: a coded sample's residual is
// within a few thousand), values go in pairs — word w < 128: luma samples w
// (low half) and w + 128; word 256 + w, w < 64: chroma samples 256 + w and
// 320 + w — and word kResFormatWord is 1: 768 bytes instead of 1536.
// Otherwise (a hostile stream whose int32-wrapped arithmetic made a value no
// 16-bit number reproduces under the reconstruction's wrapping add) the 384
// words are stored as they are and the format word is 0.  Both formats put
// the values the readers load first at the same words.
constexpr int kResFormatWord = kCoefPerMB - 1;
__device__ __forceinline__ int32_t lo16(uint32_t w) { return (int32_t)(int16_t)(w & 0xFFFFu); }
__device__ __forceinline__ int32_t hi16(uint32_t w) { return (int32_t)(int16_t)(w >> 16); }
__device__ __forceinline__ int resWordLo(int w) { return w < 128 ? w : w + 128; }  // w < 192: the low sample
__device__ __forceinline__ void storeResidual(uint32_t* cg, const int32_t* res, int lane) {
  bool fits = true;
  for (int q = lane; q < 384; q += 32) fits = fits && res[q] >= -32768 && res[q] <= 32767;
  fits = __all_sync(kFull, fits);
  if (fits) {
    for (int w = lane; w < 192; w += 32) {
      const int a = resWordLo(w), b = a + (w < 128 ? 128 : 64);
      cg[w < 128 ? w : w + 128] = (uint32_t)(uint16_t)res[a] | ((uint32_t)res[b] << 16);
    }
  } else {
    for (int q = lane; q < 384; q += 32) cg[q] = (uint32_t)res[q];
  }
  if (lane == 0) cg[kResFormatWord] = fits ? 1u : 0u;
}
__device__ __forceinline__ void loadResidual(const uint32_t* cg, int32_t* res, int lane) {
  if (cg[kResFormatWord]) {
    for (int w = lane; w < 192; w += 32) {
      const uint32_t v = cg[w < 128 ? w : w + 128];
      const int a = resWordLo(w);
      res[a] = lo16(v);
      res[a + (w < 128 ? 128 : 64)] = hi16(v);
    }
  } else {
    for (int q = lane; q < 384; q += 32) res[q] = (int32_t)cg[q];
  }
}

__device__ __forceinline__ int lumaSample(const uint8_t* p, int stride, int w, int h, int px, int py, int fx, int fy) {
  auto g = [&](int x, int y) -> int32_t { return __ldg(p + (size_t)clampC(y, h) * stride + clampC(x, w)); };
  if (fx == 0 && fy == 0) return g(px, py);
  if (fy == 0) {
    const int32_t* t = cTaps[fx];
    return clampByteD((t[0] * g(px - 1, py) + t[1] * g(px, py) + t[2] * g(px + 1, py) + t[3] * g(px + 2, py) + 32) >> 6);
  }
  if (fx == 0) {
    const int32_t* t = cTaps[fy];
    return clampByteD((t[0] * g(px, py - 1) + t[1] * g(px, py) + t[2] * g(px, py + 1) + t[3] * g(px, py + 2) + 32) >> 6);
  }
  const int32_t* tx = cTaps[fx];
  const int32_t* ty = cTaps[fy];
  int32_t v = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int yy = py - 1 + k;
    v += ty[k] * (tx[0] * g(px - 1, yy) + tx[1] * g(px, yy) + tx[2] * g(px + 1, yy) + tx[3] * g(px + 2, yy));
  }
  return clampByteD((v + 2048) >> 12);
}

// Eight samples of a row at once, with the columns sx - 1 to sx + 9 inside the
// plane and the aligned words that hold them inside the row: per line four
// words, from which each sample's four taps are cut and summed by one
// instruction (a sample by itself takes 16 byte loads, clamps and products).
// Whole-sample positions in one direction are its taps {0, 64, 0, 0}, which
// give the same as leaving that direction out.
__device__ __forceinline__ int dotTaps(uint32_t samples, int32_t taps) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(samples), "r"(taps), "r"(0));
  return d;
}
__device__ __forceinline__ void lumaEight(const uint8_t* p, int stride, int h, int sx, int sy, int fx, int fy, int (&out)[8]) {
  const int32_t* t = cTaps[fx];
  const int32_t taps = (t[0] & 0xFF) | (t[1] & 0xFF) << 8 | (t[2] & 0xFF) << 16 | t[3] << 24;
  const int base = (sx - 1) & ~3, sh = ((sx - 1) & 3) * 8;
#pragma unroll
  for (int k = 0; k < 8; k++) out[k] = 2048;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    if (fy == 0 && r != 1) continue;
    const uint32_t* const w = reinterpret_cast<const uint32_t*>(p + (size_t)clampC(sy - 1 + r, h) * stride + base);
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3);
    const uint32_t a[3] = {__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh)};
    const int ty = cTaps[fy][r];
#pragma unroll
    for (int k = 0; k < 8; k++)
      out[k] += ty * dotTaps(k & 3 ? __funnelshift_r(a[k >> 2], a[(k >> 2) + 1], 8 * (k & 3)) : a[k >> 2], taps);
  }
#pragma unroll
  for (int k = 0; k < 8; k++) out[k] = clampByteD(out[k] >> 12);
}

// Two neighbouring chroma samples, which share the column between them.
__device__ __forceinline__ void chromaPair(const uint8_t* p, int stride, int w, int h, int px, int py, int fx, int fy,
                                           int& o0, int& o1) {
  const int x0 = clampC(px, w), x1 = clampC(px + 1, w), x2 = clampC(px + 2, w);
  const uint8_t* const a = p + (size_t)clampC(py, h) * stride;
  const uint8_t* const b = p + (size_t)clampC(py + 1, h) * stride;
  const int a0 = __ldg(a + x0), a1 = __ldg(a + x1);
  if (fx == 0 && fy == 0) {
    o0 = a0;
    o1 = a1;
    return;
  }
  const int a2 = __ldg(a + x2), b0 = __ldg(b + x0), b1 = __ldg(b + x1), b2 = __ldg(b + x2);
  const int gx = 8 - fx, gy = 8 - fy;
  o0 = (gy * (gx * a0 + fx * a1) + fy * (gx * b0 + fx * b1) + 32) >> 6;
  o1 = (gy * (gx * a1 + fx * a2) + fy * (gx * b1 + fx * b2) + 32) >> 6;
}

__device__ __forceinline__ int partIndex(int part, int x, int y) {  // luma coords within the MB
  switch (part) {
    case part16x8: return y >= 8;
    case part8x16: return x >= 8;
    case part8x8: return (y >= 8) * 2 + (x >= 8);
    default: return 0;
  }
}

// ---------------------------------------------------------------------------
// Register copies for the reconstruction kernels.  Their byte stores to the
// planes may alias any other memory as far as the compiler knows, so fields
// read through the descriptor or record pointers would be re-loaded after
// every store; these copies are read once.
// ---------------------------------------------------------------------------
struct ReconView {
  uint8_t* rec[3];
  const uint8_t* ref[3];
  const uint8_t* gold[3];
  int strideY, strideC, padW, padH, padCW, padCH, mbCols;
  int32_t qdc, qac;
  bool words;  // the planes' 4-byte words are aligned
  const MBRec* mbrec;
  uint32_t* coef;
  __device__ __forceinline__ void load(const FrameDesc& f) {
    for (int k = 0; k < 3; k++) {
      rec[k] = f.rec[k];
      ref[k] = f.ref[k];
      gold[k] = f.gold[k];
    }
    strideY = f.strideY;
    strideC = f.strideC;
    words = ((reinterpret_cast<uintptr_t>(rec[0]) | reinterpret_cast<uintptr_t>(rec[1]) |
              reinterpret_cast<uintptr_t>(rec[2]) | (uintptr_t)strideY | (uintptr_t)strideC) & 3) == 0;
    padW = f.padW;
    padH = f.padH;
    padCW = f.padCW;
    padCH = f.padCH;
    mbCols = f.mbCols;
    qdc = f.qdc;
    qac = f.qac;
    mbrec = f.mbrec;
    coef = f.coef;
  }
};

// A macroblock record as three 16-byte words (see MBRec).
struct RecRegs {
  uint4 a, b, c;  // words 0-3, 4-7, 8-11
  __device__ __forceinline__ void load(const MBRec* p) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    a = q[0];
    b = q[1];
    c = q[2];
  }
  __device__ __forceinline__ int mode() const { return (int)(a.x & 0xFF); }
  __device__ __forceinline__ int ref() const { return (int)((a.x >> 8) & 0xFF); }
  __device__ __forceinline__ int part() const { return (int)((a.x >> 16) & 0xFF); }
  __device__ __forceinline__ int cbp() const { return (int)(a.x >> 24); }
  __device__ __forceinline__ int tx() const { return (int)(a.y & 0xFF); }
  __device__ __forceinline__ int cmode() const { return (int)((a.y >> 8) & 0xFF); }
  __device__ __forceinline__ uint32_t mv(int i) const { return i == 0 ? a.z : (i == 1 ? a.w : (i == 2 ? b.x : b.y)); }
  __device__ __forceinline__ int lmode(int k) const {
    const uint32_t w = k < 8 ? (k < 4 ? b.z : b.w) : (k < 12 ? c.x : c.y);
    return (int)((w >> ((k & 3) * 8)) & 0xFF);
  }
  __device__ __forceinline__ uint32_t nzmask() const { return c.z; }
  __device__ __forceinline__ uint32_t wmask() const { return c.w; }
};

// ---------------------------------------------------------------------------
// Stage B1: inter macroblock reconstruction
// ---------------------------------------------------------------------------
constexpr int kInterWarps = 4;

struct InterScratch {
  __align__(16) int32_t res[384];  // levels, then residuals (mbResidual)
  __align__(16) int32_t tmp[384];
};

// Reconstruction kernels are launched with programmatic stream
// serialisation, so a grid may start while the previous kernel of the stream
// runs; this wait (a no-op without a prerequisite grid) holds every thread
// until that kernel's results are complete and visible.
__device__ __forceinline__ void waitPreviousGrid() {
#ifdef __CUDA_ARCH__
  asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// Lets the next kernel of the stream be scheduled now: its CTAs start and
// hold in waitPreviousGrid until this grid is complete, so the launch
// latency overlaps this kernel.
__device__ __forceinline__ void allowNextGrid() {
#ifdef __CUDA_ARCH__
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

// Whether inter macroblock (mbx, mby) of f predicts from pixels of an intra
// macroblock of the previous frame (f.prevRec) — a conservative test over
// the bounding box of its vectors' source blocks, widened for the filter
// taps and chroma rounding.  A previous key frame makes every macroblock
// dependent; a golden-reference macroblock reads an older, complete frame.
__device__ __forceinline__ bool interDepends(const FrameDesc& f, const RecRegs& r, int mode, int part, int mbx,
                                             int mby, int lane) {
  if (!f.prevRec) return false;
  if (f.prevKey) return true;
  if (mode == kRecInter && r.ref() == refGolden) return false;
  const int np = mode == kRecInter ? (part == partWhole ? 1 : (part == part8x8 ? 4 : 2)) : 1;
  int lo = 1 << 30, hi = -(1 << 30), vlo = 1 << 30, vhi = -(1 << 30);
  for (int i = 0; i < np; i++) {
    const uint32_t m = r.mv(i);
    const int dx = (int16_t)(m & 0xFFFFu) >> 2, dy = (int16_t)(m >> 16) >> 2;
    lo = min(lo, dx);
    hi = max(hi, dx);
    vlo = min(vlo, dy);
    vhi = max(vhi, dy);
  }
  // Samples outside the plane are clamped to its edge: clamp each end of the
  // box on its own, so a box wholly outside still names the edge macroblocks.
  const int x0 = min(max(0, mbx * 16 + lo - 4), f.padW - 1), x1 = min(max(0, mbx * 16 + 15 + hi + 4), f.padW - 1);
  const int y0 = min(max(0, mby * 16 + vlo - 4), f.padH - 1), y1 = min(max(0, mby * 16 + 15 + vhi + 4), f.padH - 1);
  const int bx0 = x0 >> 4, bx1 = x1 >> 4, by0 = y0 >> 4, by1 = y1 >> 4;
  const int nx = bx1 - bx0 + 1, n = nx * (by1 - by0 + 1);
  if (n > 16) return true;  // wide spread: wait
  bool waits = false;
  if (lane < n) {  // a lane per macroblock of the box
    const MBRec* q = f.prevRec + (by0 + lane / nx) * f.mbCols + bx0 + lane % nx;
    waits = q->mode == kRecIntra && q->wmask != 0;
  }
  return __any_sync(kFull, waits);
}

// Bound by the latency of a warp's chain of loads (record, the box of source
// macroblocks, counts, levels, reference samples) and by its instructions, not
// by bandwidth: 8160 macroblocks of 1080p move 10 MB, 1.5 us.  So every step of
// the chain is one load by many lanes: the box a lane per macroblock, the
// levels of all blocks as one list, eight samples from four words a line.  A
// sample, an output of the transform and a box's macroblock at a time it took
// 21 us for an inter frame of 1080p and 50 for a key frame's residuals (cold
// caches); now 17 and 26.  Six or eight CTAs to an SM make no difference.
//
// phase 0: the macroblocks that do not depend on the previous frame's intra
// stage (all of them when that stage is complete), and the residuals of the
// intra macroblocks; phase 1: the other inter macroblocks.
__global__ void __launch_bounds__(32 * kInterWarps, 6) kInterRecon(const FrameDesc* frames, int phase) {
  allowNextGrid();
  waitPreviousGrid();
  __shared__ InterScratch sS[kInterWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const FrameDesc& f = frames[blockIdx.y];
  if (f.gate && *f.gate) {
    if (threadIdx.x == 0) atomicExch(f.status, kSkipped);
    return;
  }
  const int idx = blockIdx.x * kInterWarps + warp;
  if (idx >= f.mbCols * f.mbRows) return;
  ReconView v;
  v.load(f);
  RecRegs r;
  r.load(v.mbrec + idx);
  const int mode = r.mode();
  const uint32_t wm = r.wmask();
  if (!wm) return;
  InterScratch& S = sS[warp];
  // An intra macroblock's residual needs no pixels: phase 0 computes it and
  // stores it over the macroblock's coefficient region, where the intra
  // stage reads it.
  const bool intra = mode == kRecIntra;
  if (intra ? phase != 0 : (!f.inter || (mode != kRecSkip && mode != kRecInter))) return;
  const int mbx = idx % v.mbCols, mby = idx / v.mbCols;
  const bool golden = mode == kRecInter && r.ref() == refGolden;
  const uint8_t* const* refp = golden ? v.gold : v.ref;
  const int part = mode == kRecInter ? r.part() : partWhole;
  const int cbp = mode == kRecInter ? r.cbp() : 0;
  bool deferred = false;  // phase 0: left to phase 1, whose residual is computed now
  if (intra) {
  } else if (phase == 0) {
    deferred = interDepends(f, r, mode, part, mbx, mby, lane);
    if (lane == 0 && f.prevRec) f.dep[idx] = deferred ? 1 : 0;
  } else if (!f.prevRec || !f.dep[idx]) {
    return;
  }
  const uint32_t nzm = r.nzmask();
  const int tx = r.tx();

  // Residuals of the coded blocks that are written, all at once.  Phase 0
  // computes those of intra and deferred macroblocks and stores them over
  // the coefficient region (off the critical path); phase 1 reads them back.
  uint32_t resMask = intra ? nzm & wm : 0;
  if (cbp & cbpLuma) resMask |= nzm & wm & 0xFFFFu;
  if (cbp & cbpCb) resMask |= nzm & wm & (1u << 16);
  if (cbp & cbpCr) resMask |= nzm & wm & (1u << 17);
  uint32_t* const cg = v.coef + (size_t)idx * kCoefPerMB;
  if (phase == 1) {
    if (resMask) loadResidual(cg, S.res, lane);
    __syncwarp();
  } else if (resMask) {
    mbResidual(cg, tx, resMask, v.qdc, v.qac, S.res, S.tmp, lane);
  }
  if (intra || deferred) {
    if (resMask) storeResidual(cg, S.res, lane);
    return;
  }

  // Luma: lane -> row lane/2, 8 columns.
  {
    const int row = lane >> 1, c0 = (lane & 1) * 8;
    const uint32_t m = r.mv(partIndex(part, c0, row));
    const int mvx = (int16_t)(m & 0xFFFFu), mvy = (int16_t)(m >> 16);
    const int fx = mvx & 3, fy = mvy & 3;
    const int sx = mbx * 16 + c0 + (mvx >> 2), sy = mby * 16 + row + (mvy >> 2);
    int pred[8];
    if (fx == 0 && fy == 0 && sx >= 0 && sy >= 0 && sy < v.padH && sx + 8 <= v.padW && (sx & ~7) + 16 <= v.strideY) {
      // Whole-pel vector with the row segment inside the plane: the samples
      // need no clamping; two aligned 8-byte loads cover them (rows start
      // 64-byte aligned and the loads stay inside the row's stride).
      const uint8_t* rowp = refp[0] + (size_t)sy * v.strideY;
      const int base = sx & ~7, sh = (sx & 7) * 8;
      uint64_t w = __ldg(reinterpret_cast<const unsigned long long*>(rowp + base));
      if (sh) w = (w >> sh) | ((uint64_t)__ldg(reinterpret_cast<const unsigned long long*>(rowp + base + 8)) << (64 - sh));
#pragma unroll
      for (int k = 0; k < 8; k++) pred[k] = (int)((w >> (8 * k)) & 0xFF);
    } else if (sx >= 1 && sx + 10 <= v.padW && ((sx - 1) & ~3) + 16 <= v.strideY) {
      lumaEight(refp[0], v.strideY, v.padH, sx, sy, fx, fy, pred);
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++) pred[k] = lumaSample(refp[0], v.strideY, v.padW, v.padH, sx + k, sy, fx, fy);
    }
    const int n = 4 << tx, per = 4 >> tx;
    uint8_t* out = v.rec[0] + (size_t)(mby * 16 + row) * v.strideY + mbx * 16 + c0;
    const int blkA = (row / n) * per + c0 / n, blkB = (row / n) * per + (c0 + 7) / n;
    if (((wm >> blkA) & 1) && ((wm >> blkB) & 1)) {
      uint64_t o = 0;  // all eight samples are written: one 8-byte store (out is 8-byte aligned)
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int val = resMask ? clampByteD(wadd(pred[k], S.res[row * 16 + c0 + k])) : pred[k];
        o |= (uint64_t)(uint32_t)val << (8 * k);
      }
      *reinterpret_cast<unsigned long long*>(out) = o;
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int c = c0 + k;
        const int blk = (row / n) * per + c / n;
        if (!((wm >> blk) & 1)) continue;
        const int val = resMask ? clampByteD(wadd(pred[k], S.res[row * 16 + c])) : pred[k];
        out[k] = (uint8_t)val;
      }
    }
  }
  // Chroma: lane -> row lane/4, 2 columns; Cb then Cr.
#pragma unroll
  for (int pl = 0; pl < 2; pl++) {
    const uint32_t bit = 1u << (16 + pl);
    if (!(wm & bit)) continue;
    const int row = lane >> 2, c0 = (lane & 3) * 2;
    const uint32_t m = r.mv(partIndex(part, c0 * 2, row * 2));
    const int mvx = (int16_t)(m & 0xFFFFu), mvy = (int16_t)(m >> 16);
    const int fx = mvx & 7, fy = mvy & 7;
    const int sx = mbx * 8 + c0 + (mvx >> 3), sy = mby * 8 + row + (mvy >> 3);
    int p0, p1;
    chromaPair(refp[1 + pl], v.strideC, v.padCW, v.padCH, sx, sy, fx, fy, p0, p1);
    if (resMask & bit) {
      p0 = clampByteD(wadd(p0, S.res[256 + pl * 64 + row * 8 + c0]));
      p1 = clampByteD(wadd(p1, S.res[256 + pl * 64 + row * 8 + c0 + 1]));
    }
    uint8_t* out = v.rec[1 + pl] + (size_t)(mby * 8 + row) * v.strideC + mbx * 8 + c0;
    if (v.words) {
      *reinterpret_cast<uint16_t*>(out) = (uint16_t)(p0 | p1 << 8);
    } else {
      out[0] = (uint8_t)p0;
      out[1] = (uint8_t)p1;
    }
  }
}

// ---------------------------------------------------------------------------
// Stage B2: intra reconstruction wavefront
// ---------------------------------------------------------------------------

// Per-warp scratch of the intra stage: the samples that the macroblock's
// prediction may read, in shared memory.  Samples go four to a word: rows
// start at x = 0 in column kAreaX, so that words are aligned.
// Luma: areaY row 0 is the row above the macroblock (from four left of it to
// 31 right of its left edge), row 1 + y its row y; colY[k] is the column left
// of x = 4k, top to bottom (colY[0]: of the macroblock's left neighbour).
// Chroma has one block a plane: the row above and the column to its left.
constexpr int kAreaX = 16, kAreaW = 48;
struct __align__(16) IntraScratch {
  int32_t res[384];  // the macroblock's residual (computed by kInterRecon phase 0)
  uint8_t areaY[17 * kAreaW];
  uint8_t colY[5][16];
  uint8_t topC[2][32];
  uint8_t colC[2][16];
};

// The neighbours of one n x n block as predictIntra sees them after
// substituteRefs (ebiv/predict.go:131-219): top[j] is the sample above column
// j, top[-1] the corner, col[r] the one left of row r.  A missing side is
// replaced by the other side's nearest sample, both missing by kDCPred; past
// n - 1 the left column repeats, and the top row does without above-right.
template <int N>
struct IntraRefs {
  const uint8_t* top;
  const uint8_t* col;
  bool above, left, aboveRight;
  __device__ __forceinline__ int t(int j) const {
    return above ? top[(j < N || aboveRight) ? j : N - 1] : (left ? col[0] : kDCPred);
  }
  __device__ __forceinline__ int l(int r) const { return left ? col[min(r, N - 1)] : (above ? top[0] : kDCPred); }
  __device__ __forceinline__ int corner() const {
    return left ? (above ? top[-1] : col[0]) : (above ? top[0] : kDCPred);
  }
  // Samples j to j + 3 (j a multiple of 4, below N).
  __device__ __forceinline__ uint32_t top4(int j) const {
    return above ? *reinterpret_cast<const uint32_t*>(top + j) : 0x01010101u * (uint32_t)(left ? col[0] : kDCPred);
  }
  __device__ __forceinline__ uint32_t left4(int r) const {
    return left ? *reinterpret_cast<const uint32_t*>(col + r) : 0x01010101u * (uint32_t)(above ? top[0] : kDCPred);
  }
};

// Predicts and reconstructs P samples of an N x N block, row r from column c
// on (predictIntra, ebiv/predict.go:131-219), into the bytes of the result;
// res is null or their residual.
template <int N, int P>
__device__ __forceinline__ uint32_t intraSamples(const IntraRefs<N>& f, int mode, int r, int c, const int32_t* res) {
  int v[P];
  int32_t add[P];
#pragma unroll
  for (int i = 0; i < P; i++) add[i] = 0;
  if (res) {
    if (P == 4) {
      const int4 q = *reinterpret_cast<const int4*>(res);
      add[0] = q.x;
      add[P / 4] = q.y;
      add[P / 2] = q.z;
      add[3 * P / 4] = q.w;
    } else {
#pragma unroll
      for (int i = 0; i < P; i++) add[i] = res[i];
    }
  }
  if (mode == modeDC) {
    uint32_t sum = N;
#pragma unroll
    for (int i = 0; i < N; i += 4) sum = __dp4a(f.left4(i), 0x01010101u, __dp4a(f.top4(i), 0x01010101u, sum));
#pragma unroll
    for (int i = 0; i < P; i++) v[i] = (int)(sum / (2 * N));
  } else if (mode == modeV || mode == modeTM) {
    const int d = mode == modeTM ? f.l(r) - f.corner() : 0;
    const uint32_t t = P == 4 ? f.top4(c) : 0u;
#pragma unroll
    for (int i = 0; i < P; i++) v[i] = clampByteD((P == 4 ? (int)((t >> (8 * i)) & 0xFF) : f.t(c + i)) + d);
  } else if (mode == modeH) {
    v[0] = f.l(r);
#pragma unroll
    for (int i = 1; i < P; i++) v[i] = v[0];
  } else {
    // An angle: position (a + 1) * angle / 32 along the main side (the top
    // row of a vertical mode), continued on the other side below 0.
    const bool vertical = mode == modeD45 || mode == modeD27 || mode == modeD23;
    const int angle = mode == modeD45 || mode == modeD135 ? 32 : (mode == modeD27 || mode == modeD117 ? 13 : -13);
    constexpr int kInv = -630;  // of -13
    auto ext = [&](int k) __attribute__((always_inline)) {
      if (k == 0) return f.corner();
      if (k > 2 * N) return 0;
      if (k > 0) return vertical ? f.t(k - 1) : f.l(k - 1);
      const int t = (k * kInv + 128) >> 8;
      return t == 0 ? f.corner() : (vertical ? f.l(t - 1) : f.t(t - 1));
    };
    uint32_t o = 0;
#pragma unroll 1  // for the size of the code (see kIntraRecon)
    for (int i = 0; i < P; i++) {
      const int pos = ((vertical ? r : c + i) + 1) * angle, idx = pos >> 5, fact = pos & 31;
      const int k = (vertical ? c + i : r) + idx;
      const int a = ((32 - fact) * ext(k + 1) + fact * ext(k + 2) + 16) >> 5;
      o |= (uint32_t)clampByteD(wadd(a, res ? res[i] : 0)) << (8 * i);
    }
    return o;
  }
  uint32_t o = 0;
#pragma unroll
  for (int i = 0; i < P; i++) o |= (uint32_t)clampByteD(wadd(v[i], add[i])) << (8 * i);
  return o;
}

// Four samples of a plane: one word when the plane's words are aligned (always
// but for the planes that a caller of ebivgpu_decode_key_noalloc may give).
__device__ __forceinline__ void storeQuad(uint8_t* p, uint32_t o, bool words) {
  if (words) {
    *reinterpret_cast<uint32_t*>(p) = o;
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) p[i] = (uint8_t)(o >> (8 * i));
  }
}
__device__ __forceinline__ uint32_t loadQuad(const uint8_t* p, bool words) {
  if (words) return *reinterpret_cast<const uint32_t*>(p);
  return (uint32_t)p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24;
}

// One N x N luma block at (x, y) of its macroblock, by lanes l of nl: into the
// plane at p (the block's first sample) and where later blocks look for it.
template <int N>
__device__ __forceinline__ void intraLumaBlock(IntraScratch& S, int x, int y, int mode, bool above, bool left,
                                               bool aboveRight, bool hasRes, uint8_t* p, int stride, bool words, int l,
                                               int nl) {
  const IntraRefs<N> f = {S.areaY + y * kAreaW + kAreaX + x, S.colY[x >> 2] + y, above, left, aboveRight};
  // As many lanes as there are: a 4x4 block has a sample for each of its half
  // warp's, an 8x8 one two for each of the warp's, a 16x16 one words.
  constexpr int P = N == 4 ? 1 : (N == 8 ? 2 : 4);
#pragma unroll 1
  for (int q = l; q < N * N / P; q += nl) {
    const int r = q / (N / P), c = P * (q % (N / P));
    const uint32_t o = intraSamples<N, P>(f, mode, r, c, hasRes ? S.res + (y + r) * 16 + x + c : nullptr);
    uint8_t* const to = p + (size_t)r * stride + c;
    if (P == 4) {
      storeQuad(to, o, words);
    } else {
#pragma unroll
      for (int i = 0; i < P; i++) {
        const uint8_t v = (uint8_t)(o >> (8 * i));
        to[i] = v;
        if ((r & 3) == 3) S.areaY[(1 + y + r) * kAreaW + kAreaX + x + c + i] = v;
        if (((c + i) & 3) == 3) S.colY[(x + c + i + 1) >> 2][y + r] = v;
      }
    }
  }
}

// Progress of the intra macroblocks of one tile, shared by the warps of its
// CTA.  luma[m] counts the completed diagonal steps of macroblock m's 4x4
// luma blocks (kLumaDone when the luma is complete, at once for 8x8 and
// 16x16 transforms); chroma[m] is 1 when both chroma blocks are.  Every
// other macroblock of the tile starts complete.  A wait that runs past
// kIntraSpinLimit polls sets abort, which ends every later wait at once;
// the frame is then reported failed.
constexpr int kLumaDone = 10;
constexpr int kIntraSpinLimit = 1 << 20;
struct IntraSync {
  volatile uint8_t* luma;
  volatile uint8_t* chroma;
  volatile int* abort;
  int x0, y0, x1, tw;  // the tile: first column and row, end column, width (macroblocks)
  __device__ __forceinline__ int at(int mbx, int mby) const { return (mby - y0) * tw + (mbx - x0); }
  // Waits until progress word p reaches need (all lanes poll the same word).
  __device__ __forceinline__ void wait(volatile uint8_t* p, int need) const {
    for (int it = 0; *p < need && !*abort; it++) {
      if (it >= kIntraSpinLimit) {
        *abort = 1;
        break;
      }
      __nanosleep(20);
    }
    __threadfence_block();
  }
  // Publishes progress v once every lane's writes so far are visible to the CTA.
  __device__ __forceinline__ void publish(volatile uint8_t* p, int v, int lane) const {
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();  // and with it the other lanes' writes, which the barrier ordered before
      *p = (uint8_t)v;
    }
  }
};

// The luma of an intra macroblock.  With 4x4 transforms the blocks run in
// ten diagonal steps (bx + 2*by); step t needs the left neighbour's blocks
// up to step t+3 (its column 3 at rows by), which the macroblock waits for
// step by step, and the row above complete: the above-left and above
// macroblocks done and the above-right one past step 6 (its block (0,3),
// the only one the top-right block reads).  Other transform sizes wait for
// all four neighbours to be done.
__device__ __forceinline__ void intraLuma(const ReconView& f, IntraScratch& S, const IntraSync& sy, int mbx, int mby, int lane) {
  const int idx = mby * f.mbCols + mbx;
  RecRegs r;
  r.load(f.mbrec + idx);
  if (r.mode() != kRecIntra) return;
  const uint32_t wm = r.wmask();
  if (!wm) return;
  const uint32_t nzm = r.nzmask();
  const int tx = r.tx(), per = 4 >> tx, nb = per * per;
  const int tileLeft = sy.x0 * 16, tileTop = sy.y0 * 16, tileRight = sy.x1 * 16;
  const int mbLeft = mbx * 16, mbTop = mby * 16, mbRight = mbLeft + 16;
  uint8_t* const Y = f.rec[0];
  const int ys = f.strideY;
  const uint32_t resMask = nzm & wm;
  const uint32_t* rg = f.coef + (size_t)idx * kCoefPerMB;
  const bool up = mbTop > tileTop, left = mbLeft > tileLeft, ar = up && mbRight < tileRight;
  volatile uint8_t* const own = sy.luma + sy.at(mbx, mby);
  volatile uint8_t* const leftP = left ? sy.luma + sy.at(mbx - 1, mby) : nullptr;
  // The residual, the row above and, when the left neighbour is complete,
  // the left column are loaded together (one global latency); otherwise the
  // left column follows the left neighbour's steps.
  const bool lumaRes = (resMask & 0xFFFFu) != 0;
  int32_t rv[8];
  if (lumaRes) {
    // Words lane + 32q (q < 4) hold samples in either format; the format
    // word says whether they are pairs or the second half follows.
    uint32_t w4[4];
#pragma unroll
    for (int q = 0; q < 4; q++) w4[q] = rg[lane + 32 * q];
    if (rg[kResFormatWord]) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        rv[q] = lo16(w4[q]);
        rv[q + 4] = hi16(w4[q]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        rv[q] = (int32_t)w4[q];
        rv[q + 4] = (int32_t)rg[lane + 32 * (q + 4)];
      }
    }
  }
  if (up) {
    if (left) sy.wait(sy.luma + sy.at(mbx - 1, mby - 1), kLumaDone);
    sy.wait(sy.luma + sy.at(mbx, mby - 1), kLumaDone);
    if (ar) sy.wait(sy.luma + sy.at(mbx + 1, mby - 1), tx == 0 ? 7 : kLumaDone);
  }
  if (left && tx != 0) sy.wait(leftP, kLumaDone);
  // One decision for the whole warp (lane 0's reading of the flag).
  bool leftNow = false;
  if (left) leftNow = __shfl_sync(kFull, *leftP >= kLumaDone ? 1 : 0, 0) != 0;
  if (leftNow) __threadfence_block();
  // The row above in words: lane 0 the four samples left of the macroblock,
  // lanes 1-4 above it, lanes 5-8 right of it.
  const bool haveA = up && (lane == 0 ? left : lane <= 4 || (lane <= 8 && mbRight < tileRight));
  uint32_t a0 = 0;
  uint8_t lc = 0;
  if (haveA) a0 = loadQuad(Y + (size_t)(mbTop - 1) * ys + mbLeft - 4 + 4 * lane, f.words);
  if (leftNow && lane < 16) lc = Y[(size_t)(mbTop + lane) * ys + mbLeft - 1];
  if (lumaRes)
#pragma unroll
    for (int q = 0; q < 8; q++) S.res[lane + 32 * q] = rv[q];
  if (haveA) *reinterpret_cast<uint32_t*>(S.areaY + kAreaX - 4 + 4 * lane) = a0;
  if (leftNow && lane < 16) S.colY[0][lane] = lc;
  // The corner of blocks below the first row, at the macroblock's left edge:
  // the sample left of and above them, in the area's column left of x = 0.
  if (leftNow && lane < 16 && (lane & 3) == 3) S.areaY[(1 + lane) * kAreaW + kAreaX - 1] = lc;
  auto block = [&](auto size, int k, int l, int nl) __attribute__((always_inline)) {
    constexpr int n = decltype(size)::value;
    constexpr int kPer = 16 / n;
    const int bx = k % kPer * n, by = k / kPer * n;
    const int x0 = mbLeft + bx, y0 = mbTop + by;
    const bool avAR = y0 > tileTop && x0 + 2 * n <= tileRight && (by == 0 || x0 + 2 * n <= mbRight);
    intraLumaBlock<n>(S, bx, by, r.lmode(k), y0 > tileTop, x0 > tileLeft, avAR, (nzm >> k) & 1,
                      Y + (size_t)y0 * ys + x0, ys, f.words, l, nl);
  };
  if (tx == 0) {
    // Blocks beyond the first unwritten one (a prefix in raster order) are
    // skipped; each step is published all the same.
    const int half = lane >> 4;
#pragma unroll 1
    for (int t = 0; t < 10; t++) {
      if (left && !leftNow && !(t & 1) && t <= 6) {  // left column rows 2t..2t+3, for block (0, t/2)
        sy.wait(leftP, t + 4);
        if (lane < 4) {
          const uint8_t v = Y[(size_t)(mbTop + 2 * t + lane) * ys + mbLeft - 1];
          S.colY[0][2 * t + lane] = v;
          if (lane == 3) S.areaY[(4 + 2 * t) * kAreaW + kAreaX - 1] = v;
        }
      }
      __syncwarp();
      int k = -1, seen = 0;
      for (int yy = 0; yy < 4; yy++) {
        const int xx = t - 2 * yy;
        if (xx >= 0 && xx < 4) {
          if (seen == half) k = yy * 4 + xx;
          seen++;
        }
      }
      if (k >= 0 && ((wm >> k) & 1)) block(std::integral_constant<int, 4>(), k, lane & 15, 16);
      sy.publish(own, t + 1, lane);
    }
  } else {
    __syncwarp();  // the left column was loaded with the row above
#pragma unroll 1
    for (int k = 0; k < nb; k++) {
      if (!((wm >> k) & 1)) break;
      if (tx == 1) block(std::integral_constant<int, 8>(), k, lane, 32);
      else block(std::integral_constant<int, 16>(), k, lane, 32);
      __syncwarp();
    }
  }
}

// The chroma of an intra macroblock: waits for the left, above-left and
// above macroblocks' chroma (chroma prediction reads no above-right samples).
__device__ __forceinline__ void intraChroma(const ReconView& f, IntraScratch& S, const IntraSync& sy, int mbx, int mby, int lane) {
  const int idx = mby * f.mbCols + mbx;
  RecRegs r;
  r.load(f.mbrec + idx);
  if (r.mode() != kRecIntra) return;
  const uint32_t wm = r.wmask();
  if (!(wm >> 16)) return;
  const uint32_t nzm = r.nzmask();
  const bool up = mby > sy.y0, left = mbx > sy.x0;
  const int cs = f.strideC;
  const uint32_t* rg = f.coef + (size_t)idx * kCoefPerMB;
  const bool chromaRes = ((nzm & wm) >> 16) != 0;
  int32_t rv[4];
  if (chromaRes) {
    const uint32_t a = rg[256 + lane], b = rg[288 + lane];
    if (rg[kResFormatWord]) {
      rv[0] = lo16(a);
      rv[1] = lo16(b);
      rv[2] = hi16(a);
      rv[3] = hi16(b);
    } else {
      rv[0] = (int32_t)a;
      rv[1] = (int32_t)b;
      rv[2] = (int32_t)rg[320 + lane];
      rv[3] = (int32_t)rg[352 + lane];
    }
  }
  if (up) {
    if (left) sy.wait(sy.chroma + sy.at(mbx - 1, mby - 1), 1);
    sy.wait(sy.chroma + sy.at(mbx, mby - 1), 1);
  }
  if (left) sy.wait(sy.chroma + sy.at(mbx - 1, mby), 1);
  // A half warp per plane: the row above with its corner (words left of and
  // above the block) and the left column, then the block's sixteen words.
  const int pl = lane >> 4, l = lane & 15;
  uint8_t* const P = (pl ? f.rec[2] : f.rec[1]) + (size_t)(mby * 8) * cs + mbx * 8;
  const bool haveT = up && l < 3 && (l > 0 || left), haveL = left && l >= 8;
  uint32_t t = 0;
  uint8_t lc = 0;
  if (haveT) t = loadQuad(P - cs + 4 * l - 4, f.words);
  if (haveL) lc = P[(size_t)(l - 8) * cs - 1];
  if (chromaRes)
#pragma unroll
    for (int q = 0; q < 4; q++) S.res[256 + lane + 32 * q] = rv[q];
  if (haveT) *reinterpret_cast<uint32_t*>(S.topC[pl] + kAreaX - 4 + 4 * l) = t;
  if (haveL) S.colC[pl][l - 8] = lc;
  __syncwarp();
  // Cr is written only after Cb.
  if (pl == 0 ? (wm >> 16) & 1 : (wm >> 16) == 3) {
    const IntraRefs<8> refs = {S.topC[pl] + kAreaX, S.colC[pl], up, left, false};
    const int row = l >> 1, c = 4 * (l & 1);
    storeQuad(P + (size_t)row * cs + c,
              intraSamples<8, 4>(refs, r.cmode(), row, c, (nzm >> (16 + pl)) & 1 ? S.res + 256 + pl * 64 + row * 8 + c : nullptr),
              f.words);
  }
}

// Tiles of up to this many macroblocks keep their progress in shared memory;
// larger ones use the slot's progress bytes in global memory.
constexpr int kIntraFlagMBs = 32768;
// Shared memory for ordering a tile's jobs (key counts, then the ordered list).
constexpr int kIntraSortBytes = 64 * 1024;

// Wavefront key of an intra macroblock at (x, y) of its tile: a 4x4-luma
// macroblock can start 4 diagonal steps after its left neighbour, 7 after
// the above-right one and 11 after the one above (10 steps, then the row
// above is complete), so 4x + 11y orders every job after the jobs it waits
// for and interleaves the rows the way the dependencies allow.
__device__ __forceinline__ int intraKey(int x, int y) { return 4 * x + 11 * y; }

// One CTA of W warps per tile, or two (gridDim.y), one for luma and one for
// both chroma planes, neither of which reads the other's samples: a dataflow
// schedule.  The warps take the tile's intra macroblocks' luma and chroma as
// jobs in wavefront order (intraKey; raster order when the tile's ordering
// does not fit sortInts) and each job waits for exactly the neighbouring
// samples it predicts from (IntraSync).  Either order lists every job after
// the jobs it waits for, so the earliest unfinished job can always proceed.
// The residuals were computed by kInterRecon phase 0.  Dynamic shared memory:
// W IntraScratch, 2 * flagMBs progress bytes (rounded to 16), sortInts words
// for the ordering.
//
// A tile is bound by its warps' work, 550 instructions a job at 11 cycles
// each, more than by the chain of its dependencies (a 40x23 key tile takes 1.6
// times as long with 8 warps as with 16), so few tiles take two CTAs of 16
// warps each; with more tiles than half the SMs, where two CTAs would have 8
// warps each and luma more than half the work, one; with more than the SMs,
// CTAs of fewer warps, several to an SM.  One CTA, and a reference array built
// for every block: 390 us for four such tiles, 294 us for twelve of 30x22,
// 2.54 ms for one of 80x45; two CTAs and the references read in place: 265,
// 225 us and 1.57 ms.  One CTA a tile, 120 tiles of 40x23: 401 us, now 356.
//
// The code is kept small: with the samples of an angle unrolled it leaves the
// SMs' instruction caches, and many SMs fetch it from the L2 (690 us for the
// 120 tiles, 280 us for four).
template <int W>
__global__ void __launch_bounds__(32 * W, 16 / W)
    kIntraRecon(const FrameDesc* frames, const int2* jobs, int njobs, int flagMBs, int sortInts) {
  allowNextGrid();
  extern __shared__ __align__(16) uint8_t sDyn[];
  __shared__ int sNext, sAbort, sWarpTot[W];
  IntraScratch* sS = reinterpret_cast<IntraScratch*>(sDyn);
  const int j = blockIdx.x;
  if (j >= njobs) return;
  // Up to the job loop this kernel reads only what the entropy stage wrote
  // (tile statistics, the intra list), so it runs ahead of the previous
  // kernel's completion; the gate and every pixel are read after the wait.
  const FrameDesc& f = frames[jobs[j].x];
  const int tile = jobs[j].y;
  const int n = f.tileStat[tile].intraCount;
  if (n == 0) {
    waitPreviousGrid();
    if (threadIdx.x == 0 && f.gate && *f.gate) atomicExch(f.status, kSkipped);
    return;
  }
  const TileRange tr = f.tiles[tile];
  const int tw = tr.mbX1 - tr.mbX0, th = tr.mbY1 - tr.mbY0, tmbs = tw * th;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  // The planes of this CTA: each has its own progress, also where two CTAs
  // keep it in the same global memory.
  const bool both = gridDim.y == 1, lumaHere = both || blockIdx.y == 0, chromaHere = both || blockIdx.y == 1;
  uint8_t* flags;
  if (tmbs <= flagMBs) {
    flags = sDyn + sizeof(IntraScratch) * W;
  } else if (f.dep) {
    flags = f.dep + (size_t)f.mbCols * f.mbRows + 2 * (size_t)tr.mbBase;
  } else {
    if (tid == 0) atomicExch(f.status, kErrDevice);
    return;
  }
  IntraSync sy;
  sy.luma = flags;
  sy.chroma = flags + tmbs;
  sy.abort = &sAbort;
  sy.x0 = tr.mbX0;
  sy.y0 = tr.mbY0;
  sy.x1 = tr.mbX1;
  sy.tw = tw;
  const uint32_t* list = f.intraList + tr.mbBase;
  for (int i = tid; i < tmbs; i += blockDim.x) {
    if (lumaHere) sy.luma[i] = kLumaDone;
    if (chromaHere) sy.chroma[i] = 1;
  }
  if (tid == 0) {
    sNext = 0;
    sAbort = 0;
  }
  __syncthreads();
  const int mbCols = f.mbCols;
  for (int i = tid; i < n; i += blockDim.x) {
    const int idx = (int)(list[i] & kIndexMask);
    const int m = sy.at(idx % mbCols, idx / mbCols);
    if (lumaHere) sy.luma[m] = 0;
    if (chromaHere) sy.chroma[m] = 0;
  }
  __syncthreads();
  // Wavefront order: a counting sort of the list by intraKey in shared memory.
  const uint32_t* order = list;
  const int nkeys = intraKey(tw - 1, th - 1) + 1;
  if (nkeys + n <= sortInts) {
    int* cnt = reinterpret_cast<int*>(sDyn + sizeof(IntraScratch) * W + (((size_t)2 * flagMBs + 15) & ~(size_t)15));
    uint32_t* out = reinterpret_cast<uint32_t*>(cnt + nkeys);
    auto keyOf = [&](uint32_t e) {
      const int idx = (int)(e & kIndexMask);
      return intraKey(idx % mbCols - tr.mbX0, idx / mbCols - tr.mbY0);
    };
    for (int i = tid; i < nkeys; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) atomicAdd(&cnt[keyOf(list[i])], 1);
    __syncthreads();
    {  // exclusive scan of cnt: per-thread chunks, then warps, then the CTA
      const int per = (nkeys + (int)blockDim.x - 1) / (int)blockDim.x;
      const int b = min(tid * per, nkeys), e = min(b + per, nkeys);
      int run = 0;
      for (int i = b; i < e; i++) run += cnt[i];
      int incl = run;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) sWarpTot[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        const int t = lane < W ? sWarpTot[lane] : 0;
        int it = t;
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(kFull, it, o);
          if (lane >= o) it += v;
        }
        if (lane < W) sWarpTot[lane] = it - t;
      }
      __syncthreads();
      int acc = sWarpTot[warp] + incl - run;
      for (int i = b; i < e; i++) {
        const int c = cnt[i];
        cnt[i] = acc;
        acc += c;
      }
    }
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) {
      const uint32_t e = list[i];
      out[atomicAdd(&cnt[keyOf(e)], 1)] = e;
    }
    __syncthreads();
    order = out;
  }
  waitPreviousGrid();
  if (f.gate && *f.gate) {
    if (threadIdx.x == 0) atomicExch(f.status, kSkipped);
    return;
  }
  ReconView view;
  view.load(f);
  IntraScratch& S = sS[warp];
  const int jobsHere = both ? 2 * n : n;
  for (;;) {
    int k = 0;
    if (lane == 0) k = atomicAdd(&sNext, 1);
    k = __shfl_sync(kFull, k, 0);
    if (k >= jobsHere) break;
    const int idx = (int)(order[both ? k >> 1 : k] & kIndexMask);
    const int mbx = idx % mbCols, mby = idx / mbCols;
    if (both ? k & 1 : (int)blockIdx.y) {
      intraChroma(view, S, sy, mbx, mby, lane);
      sy.publish(sy.chroma + sy.at(mbx, mby), 1, lane);
    } else {
      intraLuma(view, S, sy, mbx, mby, lane);
      sy.publish(sy.luma + sy.at(mbx, mby), kLumaDone, lane);
    }
    __syncwarp();
  }
  __syncthreads();
  if (tid == 0 && sAbort) atomicExch(f.status, kErrDevice);
}

}  // namespace dev

// ---------------------------------------------------------------------------
// Launch wrappers
// ---------------------------------------------------------------------------
int uploadCodingTables(const int* scan4, const int* scan8, const int* scan16, const int32_t* dct) {
  uint32_t s[3][257];
  uint8_t pos[3][256] = {};
  std::memset(s, 0, sizeof(s));
  const int* scans[3] = {scan4, scan8, scan16};
  for (int k = 0; k < 3; k++)
    for (int i = 0; i < (16 << (2 * k)); i++) {
      const int band = bandOf(i);
      s[k][i] = (uint32_t)scans[k][i] | (uint32_t)band * dev::kGroupBytes << 8;
      pos[k][i] = (uint8_t)scans[k][i];
    }
  if (cudaMemcpyToSymbol(dev::cScanRow, s, sizeof(s)) != cudaSuccess) return kErrDevice;
  if (cudaMemcpyToSymbol(dev::gScan, pos, sizeof(pos)) != cudaSuccess) return kErrDevice;
  if (cudaMemcpyToSymbol(dev::gDct, dct, sizeof(int32_t) * 3 * 256) != cudaSuccess) return kErrDevice;
  return kOK;
}

// next: a zeroed device counter for the persistent grid (sized to the CTAs
// the device holds at once), or null for one CTA per job.
void launchEntropy(const FrameDesc* frames, const int4* jobs, int njobs, int* next, int maxTileMBs, cudaStream_t s) {
  if (njobs <= 0) return;
  constexpr int kTables = (int)sizeof(dev::EntropyTables);
  // Per device, once: the shared-memory limit and the CTAs it holds at once.
  static std::atomic<int> resident[64];
  int dev = 0;
  cudaGetDevice(&dev);
  const bool known = dev >= 0 && dev < 64;
  int held = known ? resident[dev].load(std::memory_order_acquire) : 0;
  if (!held) {
    int perSM = 0, sms = 0;
    cudaFuncSetAttribute(dev::kEntropy, cudaFuncAttributeMaxDynamicSharedMemorySize, kTables);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, dev::kEntropy, 32 * dev::kEntropyWarps, kTables);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    held = std::max(1, perSM * sms);
    if (known) resident[dev].store(held, std::memory_order_release);
  }
  const int grid = next ? std::min(njobs, held) : njobs;
  dev::kEntropy<<<grid, 32 * dev::kEntropyWarps, kTables, s>>>(frames, jobs, njobs, next);
  dev::kParseMB<<<dim3(njobs * kEntropyTilesPerJob, (maxTileMBs + dev::kParseWarps - 1) / dev::kParseWarps),
                  32 * dev::kParseWarps, 0, s>>>(frames, jobs, njobs);
  dev::kTileFinish<<<dim3(njobs, kEntropyTilesPerJob), dev::kFinishThreads, 0, s>>>(frames, jobs, njobs);
}

// The reconstruction launches overlap their start with the previous kernel
// of the stream (programmatic dependent launch; the kernels wait for it).
// A launch that is refused leaves its error for the caller's cudaGetLastError
// (a round's is read when its results are collected).
template <class... A>
static void launchDependent(void (*k)(A...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, args...);
}

void launchInter(const FrameDesc* frames, int nframes, int maxMBs, int phase, cudaStream_t s) {
  if (nframes <= 0 || maxMBs <= 0) return;
  dim3 grid((maxMBs + dev::kInterWarps - 1) / dev::kInterWarps, nframes);
  launchDependent(dev::kInterRecon, grid, dim3(32 * dev::kInterWarps), 0, s, frames, phase);
}

template <int W>
static void allowIntraSmem() {
  cudaFuncSetAttribute(dev::kIntraRecon<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(sizeof(dev::IntraScratch) * W + 2 * (size_t)dev::kIntraFlagMBs + dev::kIntraSortBytes));
}

template <int W>
static void launchIntraW(const FrameDesc* frames, const int2* jobs, int njobs, int ctas, int flagMBs, int sortInts,
                         cudaStream_t s) {
  constexpr size_t kScratch = sizeof(dev::IntraScratch) * W;
  const size_t smem = kScratch + (((size_t)2 * flagMBs + 15) & ~(size_t)15) + 4 * (size_t)sortInts;
  launchDependent(dev::kIntraRecon<W>, dim3(njobs, ctas), dim3(32 * W), smem, s, frames, jobs, njobs, flagMBs, sortInts);
}

// maxTileMBs: the largest tile of the launch's frames, in macroblocks;
// maxTileKeys: the largest wavefront key range of its tiles (4*(w-1) +
// 11*(h-1) + 1 for a tile of w x h macroblocks).  warps: the warps per CTA
// (4, 8 or 16; anything else picks by the tile count: 16 up to one CTA per
// SM, 8 up to two, else 4).  Whatever their warps, a tile has two CTAs, one for
// luma and one for chroma, while the tiles are at most half the SMs
// (kIntraRecon says why), else one for both.
void launchIntra(const FrameDesc* frames, const int2* jobs, int njobs, int maxTileMBs, int maxTileKeys, int warps,
                 cudaStream_t s) {
  if (njobs <= 0) return;
  // Per device, once: the shared-memory limits of all three variants, and then
  // the SM count, whose presence says that the limits are raised (engines of
  // several threads may come here first together; each then raises them).
  static std::atomic<int> sms[64];
  int d = 0;
  cudaGetDevice(&d);
  const bool known = d >= 0 && d < 64;
  int nsm = known ? sms[d].load(std::memory_order_acquire) : 0;
  if (!nsm) {
    allowIntraSmem<16>();
    allowIntraSmem<8>();
    allowIntraSmem<4>();
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, d);
    nsm = std::max(1, nsm);
    if (known) sms[d].store(nsm, std::memory_order_release);
  }
  const int flagMBs = std::max(1, std::min(maxTileMBs, dev::kIntraFlagMBs));
  int sortInts = std::max(0, maxTileMBs) + std::max(0, maxTileKeys);
  if (4 * (size_t)sortInts > (size_t)dev::kIntraSortBytes) sortInts = 0;  // raster order
  const int ctas = 2 * njobs <= nsm ? 2 : 1;  // per tile
  if (warps != 4 && warps != 8 && warps != 16) warps = njobs <= nsm ? 16 : (njobs <= 2 * nsm ? 8 : 4);
  if (warps == 16)
    launchIntraW<16>(frames, jobs, njobs, ctas, flagMBs, sortInts, s);
  else if (warps == 8)
    launchIntraW<8>(frames, jobs, njobs, ctas, flagMBs, sortInts, s);
  else
    launchIntraW<4>(frames, jobs, njobs, ctas, flagMBs, sortInts, s);
}

}  // namespace ebiv
