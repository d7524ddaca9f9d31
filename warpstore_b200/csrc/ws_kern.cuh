// Scan kernel bodies, templated over a row evaluator `Ev`.  The library instantiates them with the
// on-device interpreter (InterpEv, ws_interp.cuh); every query plan instantiates them again with its
// own generated evaluator, compiled by NVRTC for sm_100a (ws_codegen.cpp).  No host headers.
//
// Evaluator contract (all row indices are within the current batch):
//   static constexpr int NK, NA;            loop bounds (>= nk(), na())
//   static constexpr bool COMPACT;          shared tables hold compact accumulators (else accumulator rows)
//   static constexpr int DENSE_V, FLUSH_ROWS, *_MIN_BLOCKS;   see the kernels
//   Ev(const Launch&);  void bind(const Launch&, int batch);  bool fastOk;
//   int nk(), na(), rowWords(), kind(a), woff(a); bool keyInt(k);
//   void load(i64 r0, bool fast, int nv);   rows r0 .. r0+3 (nv valid) into registers
//   bool where(i); i64 ikey(k, i); double dkey(k, i); bool ival(a, i, i64&); double dval(a, i)
//   void prep(i, bool live); void finish()
// Evaluators with HOT = true (columns of known storage) keep the fetched rows packed and decode a row where it
// is used; they evaluate only rows that passed (prep), and give sumMag(i), the magnitude word of row i's SUM
// arguments (see sumMagnitude), and for the GROUP BY keys of KEY32 (a bit per key) ikey32(k, i).
//
// Work decomposition: a batch (segment / write buffer) is cut into tiles of kTile rows; a CTA of
// kThreads threads takes one tile per iteration, each thread 4 consecutive rows (128-bit loads of
// 4-byte columns, 2 x 128-bit of 8-byte columns).  Grids are persistent (a multiple of the SM count);
// CTAs stride over the tiles of all batches of the launch.
#pragma once
#include "ws_dev.cuh"

namespace ws {

constexpr int kThreads = 256;
constexpr int kTile = kThreads * 4;
constexpr u64 kEmpty = ~0ull;
constexpr int kMaxRowWords = 1 + 2 * WS_MAX_AGGS;

WS_DI u64 mix64(u64 x) {  // splitmix64 finalizer (Steele, Lea, Flood 2014)
  x ^= x >> 30;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 27;
  x *= 0x94d049bb133111ebull;
  x ^= x >> 31;
  return x;
}

// The 4 loaded rows of a thread, one after another: filter the row, evaluate its common
// subexpressions (prep), hand it to f when it passes.  Evaluating and consuming each row before the
// next keeps one row's temporaries live at a time (fewer registers, more resident warps).
template <class Ev, class F>
WS_DI void rowGroup(Ev& ev, unsigned live, int b, i64 r0, F&& f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool ok = ((live >> i) & 1u) && ev.where(i);
    if constexpr (Ev::HOT) {
      if (ok) {
        ev.prep(i, true);
        f(i, b, r0 + i);
      }
    } else {
      ev.prep(i, ok);
      if (ok) f(i, b, r0 + i);
    }
  }
}

// The batch holding tile t of the launch (tileStart[b] <= t < tileStart[b + 1]; empty batches skipped).
WS_DI int batchOfTile(const Launch& L, i64 t) {
  int lo = 0, hi = L.nb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(L.tileStart + mid) <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Walks the tiles this CTA owns: the contiguous range [T c / G, T (c + 1) / G) of the launch's T tiles
// (c = ctaIndex, G = ctaCount), batch by batch.  A CTA crosses one or two batches, so the batch's
// size, bitmap and column views (and an encoded column's header) are read once or twice per CTA
// rather than once per batch of the launch.  tile(t, b, r0, n, del) is called by every thread of the
// CTA for each tile t of batch b (r0 = the thread's first row in the batch, n = the batch's rows,
// del = its deleted bitmap); it returns true to end the walk (the same value in every thread).
// V > 1: a CTA of V * kThreads threads walks as V CTAs of kThreads would (V ranges, one per group of kThreads
// threads); its body then has no CTA-wide barrier in the walk.
template <int V = 1, class Ev, class F>
WS_DI void forEachOwnedTile(const Launch& L, Ev& ev, F&& tile) {
  const i64 T = L.ntiles, G = (i64)ctaCount(L) * V, c = (i64)ctaIndex(L) * V + (V > 1 ? threadIdx.x / kThreads : 0);
  const int tid = V > 1 ? threadIdx.x % kThreads : threadIdx.x;
  i64 t = T * c / G;
  const i64 tEnd = T * (c + 1) / G;
  if (t >= tEnd) return;
  for (int b = batchOfTile(L, t); t < tEnd && b < L.nb; ++b) {
    const i64 bs = __ldg(L.tileStart + b), bend = __ldg(L.tileStart + b + 1), be = bend < tEnd ? bend : tEnd;
    if (t >= be) continue;  // an empty batch
    ev.bind(L, b);
    const i64 n = __ldg(L.n + b);
    const uint32_t* del = L.del[b];
    for (; t < be; ++t)
      if (tile(t, b, (t - bs) * kTile + tid * 4, n, del)) return;
  }
}

// Loads the thread's 4 rows from r0 and visits the live ones (not deleted, passing the filter).
template <class Ev, class F>
WS_DI void visitRows(Ev& ev, int b, i64 r0, i64 n, const uint32_t* del, F&& f) {
  const i64 left = n - r0;
  if (left <= 0) return;
  const int nv = left >= 4 ? 4 : (int)left;
  ev.load(r0, ev.fastOk && nv == 4, nv);
  unsigned live = (1u << nv) - 1;
  if (del) live &= ~(__ldg(del + (r0 >> 5)) >> (r0 & 31)) & 0xfu;
  rowGroup(ev, live, b, r0, f);
}

// Visits every live row of the tiles this CTA owns.  f(i, batch, row) is called with i = the row's
// position (0..3) in the evaluator's 4-row group.  tileEnd() is called by every thread of the CTA
// after each of the CTA's tiles (a CTA-uniform point); it returns the same value in every thread,
// true to end the visit there.
template <class Ev, class F, class E>
WS_DI void forEachRowTiles(const Launch& L, Ev& ev, F&& f, E&& tileEnd) {
  forEachOwnedTile(L, ev, [&](i64, int b, i64 r0, i64 n, const uint32_t* del) {
    visitRows(ev, b, r0, n, del, f);
    return tileEnd();
  });
  ev.finish();
}

template <int V = 1, class Ev, class F>
WS_DI void forEachRow(const Launch& L, Ev& ev, F&& f) {
  forEachOwnedTile<V>(L, ev, [&](i64, int b, i64 r0, i64 n, const uint32_t* del) {
    visitRows(ev, b, r0, n, del, f);
    return false;
  });
  ev.finish();
}

// Same visit, with each tile's column chunks brought into shared memory by bulk asynchronous copies
// (TMA engine), warp-specialized: the CTA has kThreads consumer threads plus one producer warp (the
// last).  A ring of S stages of Ev::STAGE_BYTES has two mbarriers per stage: `full` (the producer's
// arrive.expect_tx; the copies complete its transaction count) and `empty` (one arrival per consumer
// warp once it has read the stage).  The producer refills a stage as soon as every consumer warp has
// released it, so consumers never wait on a CTA-wide barrier.  Tiles that cannot be copied in bulk (a
// batch's ragged last tile, a column not 16-byte aligned) are marked "direct": their full barrier gets
// a plain arrive and the consumers read global memory as forEachRow does.  Every wait is bounded
// (2^L.waitLog2 cycles); one that runs out sets err[2] and ends that warp's loop.  Before the producer
// warp leaves, it waits (bounded, ~2 s) until the copies of the stages it issued last have landed, so
// no bulk copy is still writing into the CTA's shared memory when the CTA ends.
constexpr int kStagedThreads = kThreads + 32;

template <class Ev, class F>
WS_DI void forEachRowStaged(const Launch& L, Ev& ev, unsigned char* stages, int S, F&& f) {
  __shared__ __align__(8) u64 full[8], empty[8];
  __shared__ int smode[8];
  __shared__ typename Ev::Stage pst;  // the producer's view of its current batch
  constexpr int kConsumerWarps = kThreads / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbarInit(smemAddr(&full[s]), 1);
      mbarInit(smemAddr(&empty[s]), kConsumerWarps);
    }
    fenceMbarInit();
    fenceProxyAsync();
  }
  __syncthreads();
  // this CTA's tiles: the contiguous range [tFirst, tFirst + K) (as forEachOwnedTile)
  const i64 tFirst = L.ntiles * (i64)ctaIndex(L) / ctaCount(L);
  const i64 K = L.ntiles * ((i64)ctaIndex(L) + 1) / ctaCount(L) - tFirst;
  if (warp == kConsumerWarps) {  // ---- producer warp (one elected lane)
    if (lane == 0) {
      int pb = K > 0 ? batchOfTile(L, tFirst) : 0, pbatch = -1;
      i64 issued = 0;
      for (i64 k = 0; k < K; ++k) {
        const int s = (int)(k % S);
        if (k >= S && !mbarWait(smemAddr(&empty[s]), (unsigned)(((k / S) - 1) & 1), L.waitLog2)) {
          L.err[2] = 1;
          break;
        }
        issued = k + 1;
        const i64 t = tFirst + k;
        while (t >= __ldg(L.tileStart + pb + 1)) ++pb;
        if (pb != pbatch) {
          Ev::stageBind(L, pb, pst);
          pbatch = pb;
        }
        const i64 tr0 = (t - __ldg(L.tileStart + pb)) * kTile;
        const bool bulk = pst.ok && tr0 + kTile <= __ldg(L.n + pb);
        smode[s] = bulk;
        const unsigned bar = smemAddr(&full[s]);
        if (bulk) {
          fenceProxyAsync();  // the stage was last read through the generic proxy
          mbarArriveTx(bar, pst.bytes);
          Ev::stageIssue(pst, tr0, smemAddr(stages + (size_t)s * Ev::STAGE_BYTES), bar);
        } else {
          mbarArrive(bar);
        }
      }
      // drain: the last phase issued on each stage completes when its copies have landed (earlier
      // phases completed before their stage was reissued)
      for (i64 k = issued > S ? issued - S : 0; k < issued; ++k)
        if (!mbarWait(smemAddr(&full[(int)(k % S)]), (unsigned)((k / S) & 1))) L.err[2] = 1;
    }
    __syncwarp();
    return;
  }
  // ---- consumer warps
  int b = K > 0 ? batchOfTile(L, tFirst) : 0, bound = -1;
  for (i64 k = 0; k < K; ++k) {
    const i64 t = tFirst + k;
    const int s = (int)(k % S);
    if (!__all_sync(0xffffffffu, mbarWait(smemAddr(&full[s]), (unsigned)((k / S) & 1), L.waitLog2))) {
      if (lane == 0) L.err[2] = 1;
      break;
    }
    while (t >= __ldg(L.tileStart + b + 1)) ++b;
    if (b != bound) {
      ev.bind(L, b);
      bound = b;
    }
    const i64 n = __ldg(L.n + b);
    const i64 r0 = (t - __ldg(L.tileStart + b)) * kTile + tid * 4;
    const i64 left = n - r0;
    if (left > 0) {
      const int nv = left >= 4 ? 4 : (int)left;
      if (smode[s]) ev.loadStage(stages + (size_t)s * Ev::STAGE_BYTES, tid * 4);
      else ev.load(r0, ev.fastOk && nv == 4, nv);
      unsigned live = (1u << nv) - 1;
      const uint32_t* del = L.del[b];
      if (del) live &= ~(__ldg(del + (r0 >> 5)) >> (r0 & 31)) & 0xfu;
      rowGroup(ev, live, b, r0, f);
    }
    __syncwarp();
    if (lane == 0) mbarArrive(smemAddr(&empty[s]));  // this warp is done with the stage
  }
  ev.finish();
}

// Visits rows, staged through shared memory when the evaluator supports it and stages were given.
template <class Ev, class F>
WS_DI void scanRows(const Launch& L, Ev& ev, F&& f) {
  if constexpr (Ev::STAGED) {
    if (L.stages >= 2 && blockDim.x == kStagedThreads) {
      extern __shared__ __align__(16) u64 wsSmem[];
      forEachRowStaged(L, ev, (unsigned char*)wsSmem, L.stages, f);
      return;
    }
  }
  forEachRow(L, ev, f);
}

// ------------------------------------------------------------------ register rows
// Per-thread accumulators of the no-key and dense kernels: one word per slot (fwoff).  An integer SUM
// adds into an int64 word; when an addition overflows it (signed), the word keeps the wrapped value
// and +-1 goes to the high word of the CTA's shared int128 spill counter of its (group, slot), so the
// exact sum is word + 2^64 * spill at the end.
template <class Ev>
WS_DI void fastIdentity(const Ev& ev, u64* w) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.fwoff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: case SK_ISUM: case SK_DSUM: w[o] = 0; break;
      case SK_IMIN: w[o] = (u64)0x7fffffffffffffffll; break;
      case SK_IMAX: w[o] = (u64)0x8000000000000000ll; break;
      case SK_DMIN: w[o] = (u64)dord(__longlong_as_double(0x7ff0000000000000ll)); break;
      case SK_DMAX: w[o] = (u64)dord(__longlong_as_double((i64)0xfff0000000000000ull)); break;
      default: break;
    }
  }
}
// The register-row contribution of row i (NULL arguments: the slot's identity).
template <class Ev>
WS_DI void fastOfInput(const Ev& ev, int i, u64* x) {
  fastIdentity(ev, x);
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.fwoff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: x[o] = 1; break;
      case SK_ISUM: case SK_IMIN: case SK_IMAX: {
        i64 v;
        if (ev.ival(a, i, v)) x[o] = (u64)v;
        break;
      }
      case SK_DSUM: {
        const double v = ev.dval(a, i);
        if (v == v) x[o] = (u64)__double_as_longlong(v);
        break;
      }
      case SK_DMIN: case SK_DMAX: {
        const double v = ev.dval(a, i);
        if (v == v) x[o] = (u64)dord(v);
        break;
      }
      default: break;
    }
  }
}
// *w += x for an int64 SUM word, carrying a signed overflow into the spill's high word.
WS_DI void addCarry(u64* w, u64 x, u64* spillHi) {
  const u64 old = *w, r = old + x;
  const unsigned ho = (unsigned)(old >> 32), hx = (unsigned)(x >> 32), hr = (unsigned)(r >> 32);
  if ((int)((ho ^ hr) & (hx ^ hr)) < 0) atomicAdd(spillHi, (int)hx < 0 ? ~0ull : 1ull);  // signed overflow
  *w = r;
}
// Exact integer sums without a test per addition.  A thread adds at most R rows into any one of its
// integer SUM words.  While every argument x has |x| <= 2^(63 - k), with 2^k >= R, no partial sum of
// those additions leaves the int64 range, so the words need no overflow test.  The host sets
// L.sumShift = 31 - k for each launch (-1 when no k applies).  sumMagnitude ORs the high words of the
// row's SUM arguments' magnitudes (x >= 0: x >> 32; x < 0: ~x >> 32 = (|x| - 1) >> 32); the bound holds
// while (magnitude >> sumShift) == 0.  A thread that meets a row breaking it switches to tested
// additions (signed overflow carried into the int128 spill) for the rest of the launch, so words that
// take unbounded values are always tested from their first such value on.
template <class Ev>
WS_DI unsigned sumMagnitude(const Ev& ev, const u64* x, int i) {
  if constexpr (Ev::HOT) return ev.sumMag(i);
  unsigned m = 0;
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    if (ev.kind(a) == SK_ISUM) {
      const unsigned hi = (unsigned)(x[ev.fwoff(a)] >> 32);
      m |= hi ^ (unsigned)((int)hi >> 31);
    }
  }
  return m;
}
WS_DI bool sumsNeedTests(const Launch& L, unsigned magnitude) {
  return L.sumShift < 0 || (magnitude >> L.sumShift) != 0;
}

// w += x (register rows); spill = this group's [slot][2] int128 counters
template <class Ev>
WS_DI void fastCombine(const Ev& ev, u64* w, const u64* x, u64* spill) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.fwoff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: w[o] += x[o]; break;
      case SK_ISUM: addCarry(&w[o], x[o], spill + 2 * a + 1); break;
      case SK_IMIN: case SK_DMIN: if ((i64)x[o] < (i64)w[o]) w[o] = x[o]; break;
      case SK_IMAX: case SK_DMAX: if ((i64)x[o] > (i64)w[o]) w[o] = x[o]; break;
      case SK_DSUM:
        w[o] = (u64)__double_as_longlong(__longlong_as_double((i64)w[o]) + __longlong_as_double((i64)x[o]));
        break;
      default: break;
    }
  }
}
// register row -> accumulator row (integer sums widened to int128)
template <class Ev>
WS_DI void fastExpand(const Ev& ev, const u64* f, u64* w) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.woff(a), fo = ev.fwoff(a);
    if (ev.kind(a) == SK_ISUM) w[o] = f[fo], w[o + 1] = (u64)((i64)f[fo] >> 63);
    else if (ev.kind(a) != SK_NONE) w[o] = f[fo];
  }
}

// ------------------------------------------------------------------ row words
// A group's accumulator row: word 0 = key word, then each slot's words at woff(a) (slot kinds in
// SlotKind).  DMIN / DMAX words hold dord(value) so that integer min / max orders them.
template <class Ev>
WS_DI void rowIdentity(const Ev& ev, u64* w) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.woff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: w[o] = 0; break;
      case SK_ISUM: w[o] = 0, w[o + 1] = 0; break;
      case SK_IMIN: w[o] = (u64)0x7fffffffffffffffll; break;
      case SK_IMAX: w[o] = (u64)0x8000000000000000ll; break;
      case SK_DSUM: w[o] = 0; break;
      case SK_DMIN: w[o] = (u64)dord(__longlong_as_double(0x7ff0000000000000ll)); break;
      case SK_DMAX: w[o] = (u64)dord(__longlong_as_double((i64)0xfff0000000000000ull)); break;
      default: break;
    }
  }
}
// Adds row `i` of the current 4-row group into accumulator words w (registers).
template <class Ev>
WS_DI void rowAccumulate(const Ev& ev, int i, u64* w) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.woff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: w[o] += 1; break;
      case SK_ISUM: {
        i64 v;
        if (ev.ival(a, i, v)) add128(w[o], *(i64*)&w[o + 1], v);
        break;
      }
      case SK_IMIN: {
        i64 v;
        if (ev.ival(a, i, v) && v < (i64)w[o]) w[o] = (u64)v;
        break;
      }
      case SK_IMAX: {
        i64 v;
        if (ev.ival(a, i, v) && v > (i64)w[o]) w[o] = (u64)v;
        break;
      }
      case SK_DSUM: {
        const double v = ev.dval(a, i);
        if (v == v) w[o] = (u64)__double_as_longlong(__longlong_as_double((i64)w[o]) + v);
        break;
      }
      case SK_DMIN: {
        const double v = ev.dval(a, i);
        if (v == v && dord(v) < (i64)w[o]) w[o] = (u64)dord(v);
        break;
      }
      case SK_DMAX: {
        const double v = ev.dval(a, i);
        if (v == v && dord(v) > (i64)w[o]) w[o] = (u64)dord(v);
        break;
      }
      default: break;
    }
  }
}
// w += x (both accumulator rows, same layout)
template <class Ev>
WS_DI void rowCombine(const Ev& ev, u64* w, const u64* x) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.woff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: w[o] += x[o]; break;
      case SK_ISUM: add128w(w[o], *(i64*)&w[o + 1], x[o], (i64)x[o + 1]); break;
      case SK_IMIN: case SK_DMIN: if ((i64)x[o] < (i64)w[o]) w[o] = x[o]; break;
      case SK_IMAX: case SK_DMAX: if ((i64)x[o] > (i64)w[o]) w[o] = x[o]; break;
      case SK_DSUM:
        w[o] = (u64)__double_as_longlong(__longlong_as_double((i64)w[o]) + __longlong_as_double((i64)x[o]));
        break;
      default: break;
    }
  }
}
// Atomic w += x into a row in shared or global memory (generic addressing).
template <class Ev>
WS_DI void rowAtomicCombine(const Ev& ev, u64* w, const u64* x) {
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) {
    if (a >= ev.na()) break;
    const int o = ev.woff(a);
    switch (ev.kind(a)) {
      case SK_COUNT: if (x[o]) atomicAdd(w + o, x[o]); break;
      case SK_ISUM: if (x[o] || x[o + 1]) atomicAdd128(w + o, (i64*)(w + o + 1), x[o], (i64)x[o + 1]); break;
      case SK_IMIN: case SK_DMIN: if ((i64)x[o] < (i64)*(volatile u64*)(w + o)) atomicMin((i64*)(w + o), (i64)x[o]); break;
      case SK_IMAX: case SK_DMAX: if ((i64)x[o] > (i64)*(volatile u64*)(w + o)) atomicMax((i64*)(w + o), (i64)x[o]); break;
      case SK_DSUM: {
        const double v = __longlong_as_double((i64)x[o]);
        if (v != 0.0) atomicAdd((double*)(w + o), v);
        break;
      }
      default: break;
    }
  }
}
// The accumulator row of a single input row (count 1, each argument once; NULL arguments neutral).
template <class Ev>
WS_DI void rowOfInput(const Ev& ev, int i, u64* w) {
  rowIdentity(ev, w);
  rowAccumulate(ev, i, w);
}

// Warp + block reduction of one accumulator row per thread into `out` (thread 0's view).
template <class Ev, int RW>
WS_DI void blockReduceRow(const Ev& ev, u64 (&w)[RW], u64* sred /* [kStagedThreads/32][RW] */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rw = ev.rowWords();
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    u64 x[RW];
#pragma unroll
    for (int j = 0; j < RW; ++j) x[j] = j < rw ? __shfl_down_sync(0xffffffffu, w[j], off) : 0;
    rowCombine(ev, w, x);
  }
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < RW; ++j)
      if (j < rw) sred[warp * RW + j] = w[j];
  __syncthreads();
  if (warp == 0) {
    if (lane < (int)(blockDim.x >> 5)) {
#pragma unroll
      for (int j = 0; j < RW; ++j)
        if (j < rw) w[j] = sred[lane * RW + j];
    } else {
      rowIdentity(ev, w);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      u64 x[RW];
#pragma unroll
      for (int j = 0; j < RW; ++j) x[j] = j < rw ? __shfl_down_sync(0xffffffffu, w[j], off) : 0;
      rowCombine(ev, w, x);
    }
  }
  __syncthreads();
}

// (lo, hi) += (l, h) for one slot of kind k.
WS_DI void slotIdentity(int k, u64& lo, u64& hi) {
  hi = 0;
  lo = k == SK_IMIN ? (u64)0x7fffffffffffffffll : k == SK_IMAX ? (u64)0x8000000000000000ll
       : k == SK_DMIN ? (u64)dord(__longlong_as_double(0x7ff0000000000000ll))
       : k == SK_DMAX ? (u64)dord(__longlong_as_double((i64)0xfff0000000000000ull)) : 0ull;
}
WS_DI void slotCombine(int k, u64& lo, u64& hi, u64 l, u64 h) {
  switch (k) {
    case SK_COUNT: lo += l; break;
    case SK_ISUM: add128w(lo, *(i64*)&hi, l, (i64)h); break;
    case SK_IMIN: case SK_DMIN: if ((i64)l < (i64)lo) lo = l; break;
    case SK_IMAX: case SK_DMAX: if ((i64)l > (i64)lo) lo = l; break;
    case SK_DSUM: lo = (u64)__double_as_longlong(__longlong_as_double((i64)lo) + __longlong_as_double((i64)l)); break;
    default: break;
  }
}
// Reduces every (row, slot) of nrows rows over N contributors, one pair per warp at a time: lane l folds
// contributors l, l + 32, ... in order, then a fixed shuffle tree combines the lanes (deterministic), and lane 0
// calls put(row, slot, lo, hi).  get(row, slot, contributor, lo, hi) reads a value.  A pair moves its one or two
// words only and needs no barrier, where whole rows went through every shuffle group by group.  A lane reads
// kPairLoads values before it combines them: a combination branches on the slot's kind, so a load behind it would
// wait for the one before (1M rows, COUNT and two SUMs into 4 groups: 31.9 us that way, 23.5 us so; without GROUP BY
// 14.0 and 10.7 us).
constexpr int kPairLoads = 8;
template <class Ev, class Get, class Put>
WS_DI void reducePairs(const Ev& ev, int nrows, int N, Get&& get, Put&& put) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, na = ev.na();
  for (int p = warp; p < nrows * na; p += nw) {
    const int r = p / na, a = p % na, k = ev.kind(a);
    if (k == SK_NONE) continue;
    u64 lo, hi;
    slotIdentity(k, lo, hi);
    for (int c0 = lane; c0 < N; c0 += 32 * kPairLoads) {
      u64 l[kPairLoads], h[kPairLoads];
#pragma unroll
      for (int j = 0; j < kPairLoads; ++j)
        if (c0 + 32 * j < N) get(r, a, c0 + 32 * j, l[j], h[j]);
#pragma unroll
      for (int j = 0; j < kPairLoads; ++j)
        if (c0 + 32 * j < N) slotCombine(k, lo, hi, l[j], h[j]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const u64 l = __shfl_down_sync(0xffffffffu, lo, off), h = __shfl_down_sync(0xffffffffu, hi, off);
      slotCombine(k, lo, hi, l, h);
    }
    if (lane == 0) put(r, a, lo, hi);
  }
}

// After every CTA wrote its partial rows part[cta][nrows][rw]: the last CTA to finish reduces them
// into rows[nrows][rw] (word 0 of each row = its key word, left as is; rows accumulate across launches (scan
// windows): combined into them), deterministically.
template <class Ev>
WS_DI void lastCtaReduce(const Launch& L, const Ev& ev, int nrows) {
  __shared__ bool amLast;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) amLast = atomicAdd(L.ticket, 1u) == ctaCount(L) - 1;
  __syncthreads();
  if (!amLast) return;
  __threadfence();
  const int rw = ev.rowWords();
  reducePairs(
      ev, nrows, (int)ctaCount(L),
      [&](int r, int a, int c, u64& lo, u64& hi) {
        const u64* p = L.part + ((size_t)c * nrows + r) * rw + ev.woff(a);
        lo = __ldcg(p);
        hi = ev.kind(a) == SK_ISUM ? __ldcg(p + 1) : 0ull;
      },
      [&](int r, int a, u64 lo, u64 hi) {
        u64* out = L.rows + (size_t)r * rw + ev.woff(a);
        const bool two = ev.kind(a) == SK_ISUM;
        u64 l = out[0], h = two ? out[1] : 0ull;
        slotCombine(ev.kind(a), l, h, lo, hi);
        out[0] = l;
        if (two) out[1] = h;
      });
}

// ------------------------------------------------------------------ no GROUP BY
template <class Ev, bool kStaged>
__device__ void aggNoKeys(const Launch& L) {
  constexpr int RW = Ev::RW, FW = Ev::FRW;
  __shared__ u64 sred[(kStagedThreads / 32) * RW];
  __shared__ u64 spill[2 * Ev::NA];
  Ev ev(L);
  for (int j = threadIdx.x; j < 2 * Ev::NA; j += blockDim.x) spill[j] = 0;
  __syncthreads();
  u64 f[FW];
  fastIdentity(ev, f);
  bool tested = false;  // sums take tested additions (sticky, see sumMagnitude)
  // A HOT evaluator knows most rows' magnitudes from its narrow evaluation, so the bounded form pays; for the
  // others a tested addition costs about what the magnitude test does, so every addition is tested.
  auto row = [&](int i, int, i64) {
    u64 x[FW];
    fastOfInput(ev, i, x);
    if constexpr (Ev::HOT) {
      tested |= sumsNeedTests(L, ev.sumMag(i));
      if (!tested) {
#pragma unroll
        for (int a = 0; a < Ev::NA; ++a) {
          const int o = ev.fwoff(a);
          switch (ev.kind(a)) {
            case SK_COUNT: case SK_ISUM: f[o] += x[o]; break;
            case SK_IMIN: case SK_DMIN: if ((i64)x[o] < (i64)f[o]) f[o] = x[o]; break;
            case SK_IMAX: case SK_DMAX: if ((i64)x[o] > (i64)f[o]) f[o] = x[o]; break;
            case SK_DSUM: f[o] = (u64)__double_as_longlong(__longlong_as_double((i64)f[o]) + __longlong_as_double((i64)x[o])); break;
            default: break;
          }
        }
        return;
      }
    }
    fastCombine(ev, f, x, spill);
  };
  if constexpr (kStaged) scanRows(L, ev, row);
  else forEachRow(L, ev, row);
  u64 w[RW];
  rowIdentity(ev, w);
  fastExpand(ev, f, w);
  __syncthreads();
  blockReduceRow(ev, w, sred);
  const int rw = ev.rowWords();
  if (threadIdx.x == 0) {
    for (int a = 0; a < ev.na(); ++a)
      if (ev.kind(a) == SK_ISUM) add128w(w[ev.woff(a)], *(i64*)&w[ev.woff(a) + 1], spill[2 * a], (i64)spill[2 * a + 1]);
    for (int j = 1; j < rw; ++j) L.part[(size_t)ctaIndex(L) * rw + j] = w[j];
  }
  lastCtaReduce(L, ev, 1);
}

// ------------------------------------------------------------------ dense GROUP BY
template <class Ev>
WS_DI bool denseIndex(const Launch& L, const Ev& ev, int i, i64& g) {
  // ranges and G are below 2^26 (the dense limit), so the index arithmetic fits 32 bits
  unsigned gg = 0;
  if constexpr (Ev::HOT && Ev::KEY32 != 0) {
    // int32 keys with |kmin| <= 2^30: key - kmin lies in [-3 * 2^30, 3 * 2^30), so a negative difference's low
    // word is at least 2^30 and only differences in the range (< 2^26) are below it
    if (L.kmin32) {
#pragma unroll
      for (int k = 0; k < Ev::NK; ++k) {
        if (k >= ev.nk()) break;
        unsigned d;
        if ((Ev::KEY32 >> k) & 1) {
          d = (unsigned)ev.ikey32(k, i) - (unsigned)(int)L.kmin[k];
        } else {
          const i64 dd = ev.ikey(k, i) - L.kmin[k];
          d = (u64)dd >> 32 ? 0xffffffffu : (unsigned)dd;
        }
        if (d >= (unsigned)L.range[k]) return false;
        gg += d * (unsigned)L.stride[k];
      }
      g = gg;
      return gg < (unsigned)L.G;
    }
  }
#pragma unroll
  for (int k = 0; k < Ev::NK; ++k) {
    if (k >= ev.nk()) break;
    const i64 d = ev.ikey(k, i) - L.kmin[k];
    if ((u64)d >= (u64)L.range[k]) return false;
    gg += (unsigned)d * (unsigned)L.stride[k];
  }
  g = gg;
  return gg < (unsigned)L.G;
}

// Few groups, register rows in shared memory: every thread owns G private rows laid out
// [group][word][thread] (a warp's accesses are consecutive words: no bank conflicts), so adding a row
// is one read-modify-write per word at a computed address: no atomics, no per-group predication.
// Dynamic shared memory: [stages (staged scans)][private rows G * FRW * blockDim][spill G * NA * 2].
// Each (group, word) is then reduced over the CTA's threads in a fixed order; partial rows per CTA,
// the last CTA reduces them.
template <class Ev, bool kStaged>
__device__ void aggDensePriv(const Launch& L) {
  constexpr int FW = Ev::FRW, T = kThreads;
  extern __shared__ __align__(16) u64 wsSmem[];
  Ev ev(L);
  const int G = (int)L.G, tid = threadIdx.x;
  const bool owner = tid < T;  // the producer warp of a staged launch owns no rows
  const int fw = ev.fastWords();
  u64* priv = wsSmem + (size_t)(L.stages > 1 ? L.stages : 0) * (Ev::STAGE_BYTES / 8);
  u64* spill = priv + (size_t)G * fw * T;
  {
    u64 id[FW];
    fastIdentity(ev, id);
    if (owner)
      for (int g = 0; g < G; ++g)
        for (int j = 0; j < fw; ++j) priv[((size_t)g * fw + j) * T + tid] = id[j];
    for (int j = tid; j < G * 2 * Ev::NA; j += blockDim.x) spill[j] = 0;
  }
  __syncthreads();
  bool tested = false;  // this thread's sums take tested additions (sticky, see sumMagnitude)
  auto row = [&](int i, int, i64) {
    i64 gi;
    if (!denseIndex(L, ev, i, gi)) {
      L.err[0] = 1;
      return;
    }
    u64 x[FW];
    fastOfInput(ev, i, x);
    tested |= sumsNeedTests(L, sumMagnitude(ev, x, i));
    u64* p = priv + ((unsigned)gi * (unsigned)fw * T + tid);
    if (!tested) {  // no atomics on this path: the slots' read-modify-writes overlap
#pragma unroll
      for (int a = 0; a < Ev::NA; ++a) {
        if (a >= ev.na()) break;
        const int o = ev.fwoff(a);
        u64* q = p + (size_t)o * T;
        switch (ev.kind(a)) {
          case SK_COUNT: case SK_ISUM: *q += x[o]; break;
          case SK_IMIN: case SK_DMIN: if ((i64)x[o] < (i64)*q) *q = x[o]; break;
          case SK_IMAX: case SK_DMAX: if ((i64)x[o] > (i64)*q) *q = x[o]; break;
          case SK_DSUM: *q = (u64)__double_as_longlong(__longlong_as_double((i64)*q) + __longlong_as_double((i64)x[o])); break;
          default: break;
        }
      }
      return;
    }
    u64* sp = spill + (unsigned)gi * (2u * Ev::NA);
#pragma unroll
    for (int a = 0; a < Ev::NA; ++a) {
      if (a >= ev.na()) break;
      const int o = ev.fwoff(a);
      u64* q = p + (size_t)o * T;
      switch (ev.kind(a)) {
        case SK_COUNT: *q += x[o]; break;
        case SK_ISUM: addCarry(q, x[o], sp + 2 * a + 1); break;
        case SK_IMIN: case SK_DMIN: if ((i64)x[o] < (i64)*q) *q = x[o]; break;
        case SK_IMAX: case SK_DMAX: if ((i64)x[o] > (i64)*q) *q = x[o]; break;
        case SK_DSUM: *q = (u64)__double_as_longlong(__longlong_as_double((i64)*q) + __longlong_as_double((i64)x[o])); break;
        default: break;
      }
    }
  };
  // the direct-load entry carries no staged path (its register budget allows more resident CTAs)
  if constexpr (kStaged) scanRows(L, ev, row);
  else forEachRow(L, ev, row);
  __syncthreads();
  const int rw = ev.rowWords();
  reducePairs(
      ev, G, T,
      [&](int g, int a, int c, u64& lo, u64& hi) {
        lo = priv[((size_t)g * fw + ev.fwoff(a)) * T + c];
        hi = ev.kind(a) == SK_ISUM ? (u64)((i64)lo >> 63) : 0ull;
      },
      [&](int g, int a, u64 lo, u64 hi) {
        const u64* sp = spill + ((size_t)g * Ev::NA + a) * 2;
        u64* out = L.part + ((size_t)ctaIndex(L) * G + g) * rw + ev.woff(a);
        if (ev.kind(a) == SK_ISUM) {
          add128w(lo, *(i64*)&hi, sp[0], (i64)sp[1]);
          out[1] = hi;
        }
        out[0] = lo;
      });
  lastCtaReduce(L, ev, G);
}

// ------------------------------------------------------------------ compact accumulators
// A group's accumulators in a CTA's shared-memory table: a 64-bit word per slot (COUNT: none) and 32-bit words in arrays
// of their own (COUNT: its count; integer SUM: the bits above the word's 64), updated by 32-bit shared atomics where a
// 64-bit one would be a compare-and-swap loop:
//   COUNT   one 32-bit addition (a CTA visits fewer than 2^32 rows);
//   integer SUM   a 96-bit number in three words: the low word added with its old value returned, the middle word and
//           the carry only when their sum is not zero, i.e. rarely for small arguments, the top word only when the
//           middle addition's carry does not cancel the argument's sign.  2^32 rows of any int64 fit 96 bits, so the
//           sum is exact for every argument (COUNT and two SUMs into 16 groups, 8M rows: 75 us, arguments of 2^51 78 us;
//           those took 3730 us when words of 64 bits sent them to the global table);
//   MIN / MAX   a read, and an atomic only when the row improves on it;
//   DOUBLE SUM   a 64-bit atomic.
// A table of E entries holds each slot's words together (word o64 of entry e at t64[o64 * E + e]): the lanes of a warp
// update one slot of random entries at a time, which then spread over all banks (words entry by entry, four to an
// entry, met in 4 bank pairs, 98 shared-memory wavefronts per 32 rows of five aggregates: 168 us where this takes 118).
// Against accumulator rows of 64-bit and 128-bit words: 40 instead of 56 bytes for COUNT, SUM, MIN, MAX and a DOUBLE
// SUM, so the table takes more groups or leaves room for more warps.
//
// The interpreter (COMPACT = false) keeps whole accumulator rows there, entry by entry: its slots' kinds and offsets are
// not constants, and the branches above cost it more than the atomics (1500 groups, 4M rows: 0.87 ms with rows, 5 to
// 13 ms with compact words, depending on the unrolling).
//
// t64 / t32: the table's words, E entries; e: an entry; x: a row's accumulator words (rowOfInput).
template <class Ev>
WS_DI void compactWords(const Ev& ev, bool tops, int& n64, int& n32) {
  n64 = n32 = 0;
  if constexpr (!Ev::COMPACT) {
    n64 = ev.rowWords();
  } else {
#pragma unroll
    for (int a = 0; a < Ev::NA; ++a) {
      const int k = ev.kind(a);
      n32 += k == SK_COUNT || (k == SK_ISUM && tops);
      n64 += k != SK_COUNT && k != SK_NONE;
    }
  }
}
template <class Ev>
WS_DI unsigned compactTop0(const Ev& ev) {  // the top words' arrays start behind the counts'
  unsigned n = 0;
#pragma unroll
  for (int a = 0; a < Ev::NA; ++a) n += ev.kind(a) == SK_COUNT;
  return n;
}
template <class Ev>
WS_DI void compactIdentity(const Ev& ev, bool tops, u64* t64, unsigned* t32, unsigned e, unsigned E) {
  if constexpr (!Ev::COMPACT) {
    rowIdentity(ev, t64 + (size_t)e * ev.rowWords());
  } else {
    unsigned o64 = e, o32 = e, oTop = e + compactTop0(ev) * E;
#pragma unroll
    for (int a = 0; a < Ev::NA; ++a) {
      const int k = ev.kind(a);
      if (k == SK_NONE) continue;
      if (k == SK_COUNT) {
        t32[o32] = 0, o32 += E;
      } else {
        u64 hi;
        slotIdentity(k, t64[o64], hi);
        o64 += E;
        if (k == SK_ISUM) {
          if (tops) t32[oTop] = 0;
          oTop += E;
        }
      }
    }
  }
}
// A row (words x) may be added to compact words without top words: the sums of all the CTA's rows (2^8 threads of at
// most 2^(31 - sumShift) rows each) stay in the int64 range.
template <class Ev>
WS_DI bool compactOk(const Launch& L, const Ev& ev, const u64* x, int i) {
  if constexpr (!Ev::COMPACT) return true;
  unsigned m = 0;
  if constexpr (Ev::HOT) {
    m = ev.sumMag(i);
  } else {
#pragma unroll
    for (int a = 0; a < Ev::NA; ++a)
      if (ev.kind(a) == SK_ISUM) m |= magHigh((i64)x[ev.woff(a)]);
  }
  return L.sumShift >= 8 && (m >> (L.sumShift - 8)) == 0;
}
template <class Ev>
WS_DI void compactAdd(const Ev& ev, bool tops, const u64* x, u64* t64, unsigned* t32, unsigned e, unsigned E) {
  if constexpr (!Ev::COMPACT) {
    rowAtomicCombine(ev, t64 + (size_t)e * ev.rowWords(), x);
  } else {
    unsigned o64 = e, o32 = e, oTop = e + compactTop0(ev) * E;
#pragma unroll
    for (int a = 0; a < Ev::NA; ++a) {
      const int k = ev.kind(a);
      if (k == SK_NONE) continue;
      const u64 v = x[ev.woff(a)];
      if (k == SK_COUNT) {
        atomicAdd(t32 + o32, 1u);
        o32 += E;
        continue;
      }
      u64* p = t64 + o64;
      o64 += E;
      switch (k) {
        case SK_ISUM: {
          const unsigned lo = (unsigned)v;
          unsigned h = (unsigned)(v >> 32);
          if (lo) h += atomicAdd((unsigned*)p, lo) + lo < lo;  // the carry of the low word
          if (h) {  // 0: nothing to add, or -1 and a carry, which leave the upper words as they are
            const unsigned mid = atomicAdd((unsigned*)p + 1, h) + h;
            if (tops) {
              const int top = ((int)(v >> 32) >> 31) + (int)(mid < h);
              if (top) atomicAdd(t32 + oTop, (unsigned)top);
            }
          }
          oTop += E;
          break;
        }
        case SK_IMIN: case SK_DMIN: if ((i64)v < *(volatile i64*)p) atomicMin((i64*)p, (i64)v); break;
        case SK_IMAX: case SK_DMAX: if ((i64)v > *(volatile i64*)p) atomicMax((i64*)p, (i64)v); break;
        case SK_DSUM: {
          const double d = __longlong_as_double((i64)v);
          if (d != 0.0) atomicAdd((double*)p, d);
          break;
        }
        default: break;
      }
    }
  }
}
// w (an accumulator row) += entry e
template <class Ev>
WS_DI void compactInto(const Ev& ev, bool tops, u64* w, const u64* t64, const unsigned* t32, unsigned e, unsigned E) {
  if constexpr (!Ev::COMPACT) {
    rowCombine(ev, w, t64 + (size_t)e * ev.rowWords());
  } else {
    unsigned o64 = e, o32 = e, oTop = e + compactTop0(ev) * E;
#pragma unroll
    for (int a = 0; a < Ev::NA; ++a) {
      const int k = ev.kind(a), o = ev.woff(a);
      if (k == SK_NONE) continue;
      if (k == SK_COUNT) {
        w[o] += t32[o32], o32 += E;
      } else {
        const u64 v = t64[o64];
        o64 += E;
        u64 one = 0;
        slotCombine(k, w[o], k == SK_ISUM ? w[o + 1] : one, v,
                    (u64)(k == SK_ISUM && tops ? (i64)(int)t32[oTop] : (i64)v >> 63));
        if (k == SK_ISUM) oTop += E;
      }
    }
  }
}

// Medium G: the CTA's groups live in shared memory as compact accumulators, L.copies of each (a power of two; a
// lane uses copy lane % copies, which spreads the lanes of a warp that meet in one of few groups); at the end
// each non-empty group is merged into the global rows with global atomics.  One CTA of Ev::DENSE_V * kThreads
// threads shares a table, so that an SM holds the warps of several CTAs but merges one or two tables: 16.8M
// rows into 1500 groups with five aggregates 215 -> 118 us (accumulator rows of 56 B and CTAs of 256 threads left 16
// warps per SM), 12M into 5000 groups 377 -> 83 us (those rows did not fit, every row went to L2 atomics).  What bounds
// it now is the shared-memory pipe (88 % busy): the atomics of random entries.
template <class Ev, bool tops>
__device__ void aggDenseShared(const Launch& L) {
  extern __shared__ __align__(16) u64 wsSmem[];
  Ev ev(L);
  const int rw = ev.rowWords(), G = (int)L.G, C = L.copies, E = G * C;
  int n64, n32;
  compactWords(ev, tops, n64, n32);
  u64* t64 = wsSmem;
  unsigned* t32 = (unsigned*)(t64 + (size_t)E * n64);
  for (int e = threadIdx.x; e < E; e += blockDim.x) compactIdentity(ev, tops, t64, t32, e, E);
  __syncthreads();
  const int copy = threadIdx.x & (C - 1);
  forEachRow<Ev::DENSE_V>(L, ev, [&](int i, int, i64) {
    i64 gi;
    if (!denseIndex(L, ev, i, gi)) {
      L.err[0] = 1;
      return;
    }
    u64 x[Ev::RW];
    rowOfInput(ev, i, x);
    if (tops || compactOk(L, ev, x, i)) compactAdd(ev, tops, x, t64, t32, (int)gi * C + copy, E);
    else rowAtomicCombine(ev, L.rows + gi * rw, x);
  });
  __syncthreads();
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    u64 w[Ev::RW];
    rowIdentity(ev, w);
    for (int c = 0; c < C; ++c) compactInto(ev, tops, w, t64, t32, g * C + c, E);
    if (w[ev.woff(0)] == 0) continue;  // slot 0 is COUNT(*): no rows of this group in this CTA
    rowAtomicCombine(ev, L.rows + (i64)g * rw, w);
  }
}

// Large G: rows go straight to the global rows with atomics.
template <class Ev>
__device__ void aggDenseGlobal(const Launch& L) {
  Ev ev(L);
  const int rw = ev.rowWords();
  forEachRow(L, ev, [&](int i, int, i64) {
    i64 gi;
    if (!denseIndex(L, ev, i, gi)) {
      L.err[0] = 1;
      return;
    }
    u64 x[Ev::RW];
    rowOfInput(ev, i, x);
    rowAtomicCombine(ev, L.rows + gi * rw, x);
  });
}

// ------------------------------------------------------------------ hash GROUP BY
// Key word of a row: a single integer key is its own key word, a single double key its canonical
// bits (both exact); several keys are folded into a 64-bit hash that identifies the group, and their
// values are stored beside the table.
template <class Ev>
WS_DI u64 keyWord(const Ev& ev, int i, double* kv) {
  if (ev.nk() == 1) {
    const u64 w = ev.keyInt(0) ? (u64)ev.ikey(0, i) : (u64)dkeyBits(ev.dkey(0, i));
    kv[0] = __longlong_as_double((i64)w);
    return w;
  }
  u64 h = 0x9e3779b97f4a7c15ull;
#pragma unroll
  for (int k = 0; k < Ev::NK; ++k) {
    if (k >= ev.nk()) break;
    const u64 b = ev.keyInt(k) ? (u64)ev.ikey(k, i) : (u64)dkeyBits(ev.dkey(k, i));
    kv[k] = __longlong_as_double((i64)b);
    h = mix64(h ^ b) + (u64)k;
  }
  return h == kEmpty ? (h ^ 1) : h;
}

// The key word in key word kw's first slot of the global table, as last seen (globalInsert's starting point).
template <class Ev>
WS_DI u64 globalPeek(const Launch& L, const Ev& ev, u64 kw) {
  return *(volatile u64*)(L.table + (mix64(kw) & L.mask) * ev.rowWords());
}
// Inserts accumulator row x under key word kw into the global table (linear probing, bounded); first: globalPeek.
template <class Ev>
WS_DI void globalInsert(const Launch& L, const Ev& ev, u64 kw, const double* kv, const u64* x, u64 first) {
  const int rw = ev.rowWords();
  // The probe loop only finds the row: the lanes of a warp find theirs after different numbers of steps, and add
  // together behind it.  Every kProbeRound steps they meet, so that a lane that raised the overflow flag has stored it before
  // the others probe on (else the warp may run its longest probe, of up to probeLimit steps, first), and those stop
  // there once the table has overflowed.
  constexpr int kProbeRound = 64;
  u64* hit = nullptr;
  if (kw == kEmpty) {  // the EMPTY key word itself has a dedicated row after the table (a single key: it is the key)
    hit = L.table + (L.mask + 1) * rw;
    if (atomicCAS(hit, 0ull, 1ull) == 0ull && ev.nk() > 1)
      for (int k = 0; k < ev.nk(); ++k) L.tkeys[(L.mask + 1) * ev.nk() + k] = kv[k];
  }
  const unsigned lanes = __activemask();
  u64 s = mix64(kw) & L.mask;
  for (int p0 = 0;; p0 += kProbeRound) {
    const int end = hit ? p0 : min(p0 + kProbeRound, L.probeLimit);
#pragma unroll 1
    for (int p = p0; p < end; ++p) {
      u64* row = L.table + s * rw;
      u64 prev = p ? *(volatile u64*)row : first;
      if (prev == kEmpty) {
        prev = atomicCAS(row, kEmpty, kw);
        if (prev == kEmpty) {
          if (ev.nk() > 1)
            for (int k = 0; k < ev.nk(); ++k) L.tkeys[s * ev.nk() + k] = kv[k];
          const u64 c = atomicAdd(L.count, 1ull) + 1;
          if (c * 10 > (L.mask + 1) * 7) *(volatile int*)(L.err + 1) = 1;  // fuller than 70%: the caller retries bigger
          prev = kw;
        }
      }
      if (prev == kw) {
        hit = row;
        break;
      }
      s = (s + 1) & L.mask;
    }
    __syncwarp(lanes);
    const bool more = !hit && end < L.probeLimit && !*(volatile int*)(L.err + 1);
    if (!__any_sync(lanes, more)) break;
  }
  if (hit) rowAtomicCombine(ev, hit, x);
  else *(volatile int*)(L.err + 1) = 1;  // no free slot within the probe limit
}

// A list of n rows into the global table, Ev::FLUSH_ROWS per thread at a time: key(j) is row j's key word (kEmpty:
// no first probe), insert(j, key word, first) inserts it.  A thread stops once the table has overflowed (the run's
// result is discarded then); the flag is read beside the first probes, so it adds no wait.
template <class Ev, class Key, class Insert>
WS_DI void insertAll(const Launch& L, const Ev& ev, int n, Key&& key, Insert&& insert) {
  for (int j0 = threadIdx.x; j0 < n; j0 += blockDim.x * Ev::FLUSH_ROWS) {
    u64 kw[Ev::FLUSH_ROWS], first[Ev::FLUSH_ROWS];
    const int overflowed = *(volatile int*)(L.err + 1);
#pragma unroll
    for (int r = 0; r < Ev::FLUSH_ROWS; ++r) {
      const int j = j0 + r * (int)blockDim.x;
      kw[r] = j < n ? key(j) : kEmpty;
      first[r] = kw[r] != kEmpty ? globalPeek(L, ev, kw[r]) : 0ull;
    }
    if (overflowed) return;
#pragma unroll 1
    for (int j = j0, r = 0; r < Ev::FLUSH_ROWS && j < n; ++r, j += blockDim.x) {
      insert(j, kw[0], first[0]);
#pragma unroll
      for (int q = 0; q + 1 < Ev::FLUSH_ROWS; ++q) kw[q] = kw[q + 1], first[q] = first[q + 1];
    }
  }
}

// Rows are pre-aggregated in a per-CTA shared-memory table (smemSlots key words with compact accumulators,
// bounded probing), which absorbs hot keys.  A row that finds no slot there is appended to a per-CTA shared buffer (one
// shared atomic per warp); after a tile that appended any, the whole CTA inserts the buffered rows into the
// global table together, Ev::FLUSH_ROWS rows per thread at a time whose first probes are all in flight before the first
// is waited for, so the global probes of the cold keys run with all lanes active and overlap.  (A row finding the
// buffer full goes to the global table directly.)  Every tile ends with a flush, and the shared table is merged into
// the global table when the CTA finishes.
// A tile without such rows costs one CTA barrier, which also votes on the flush: a thread knows whether it appended
// itself, so nobody reads the shared count while others append to it.  (Reading the
// overflow flag from global memory and three barriers after every tile, with accumulator rows of 64-bit atomics:
// 1M rows into 16 groups 33.0 -> 24.8 us, 100M Zipf rows into 3.8M groups 4.56 -> 3.26 ms.  The latter is bound by the
// global table: about one random DRAM sector and three L2 operations per row that is not caught on chip.)
// The first kHotKeys keys of a CTA also have L.copies (1: none; up to kHotCopies, as memory allows) copies of their
// accumulators, a lane's copy by its number: with few groups most lanes of a warp meet in a few slots, and their shared
// atomics on one address run one after another (eight queries of up to 2.5M rows into 100 groups: 172 -> 149 us).  A key's
// copies are used by the rows that see its number; the rows before that went to its slot, and both are merged.
// Sizes of the table, the copies and the buffer: hashTable (ws_shape.h).
// Shared memory: [S] key words | [n64][E] accumulators, E = S + kHotKeys * copies | multi-key [S][nk] key values | [B][rw]
// buffer | multi-key [B][nk] key values | [n32][E] 32-bit words | [S] key numbers (bytes, 255: none).
constexpr int kHotKeys = 16, kHotCopies = 8;
template <class Ev>
__device__ void aggHash(const Launch& L) {
  extern __shared__ __align__(16) u64 wsSmem[];
  __shared__ int spillN, stopFlag, keysN;
  Ev ev(L);
  const int rw = ev.rowWords(), nk = ev.nk();
  const int S = L.smemSlots, B = L.spillRows;
  const bool multi = nk > 1;
  int n64, n32;
  compactWords(ev, true, n64, n32);
  u64* tkey = wsSmem;
  u64* t64 = tkey + S;
  const int copies = L.copies, E = S + (copies > 1 ? kHotKeys * copies : 0);
  double* skv = (double*)(t64 + (size_t)E * n64);
  u64* buf = (u64*)skv + (multi ? (size_t)S * nk : 0);
  double* bkv = (double*)(buf + (size_t)B * rw);
  unsigned* t32 = (unsigned*)(bkv + (multi ? (size_t)B * nk : 0));
  unsigned char* number = (unsigned char*)(t32 + (size_t)E * n32);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    if (e < S) tkey[e] = kEmpty, number[e] = 255;
    compactIdentity(ev, true, t64, t32, e, E);
  }
  if (threadIdx.x == 0) spillN = 0, keysN = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  bool appended = false;  // this thread sent a row to the buffer since the last flush
  // Interpreter: tiles that go past the shared table.  Its slot loops run for the rows that the table took and again for
  // the others; where over a quarter of a tile's rows found no slot, the next kSkipTiles tiles only run the second loop
  // (8M rows, COUNT and eight SUMs into 500 groups: 44 ms with every tile through the table, 19 ms so).
  constexpr int kSkipTiles = 16;
  int skip = 0;
  auto rowFn = [&](int i, int, i64) {
    double kv[Ev::NK];
    const u64 kw = keyWord(ev, i, kv);
    u64 x[Ev::RW];
    rowOfInput(ev, i, x);
    if (kw != kEmpty && S > 0 && (Ev::COMPACT || skip == 0)) {
      unsigned s = (unsigned)(mix64(kw) & (u64)(S - 1));
      bool hit = false;
#pragma unroll 1
      for (int p = 0; p < 8; ++p) {
        u64 prev = *(volatile u64*)(tkey + s);
        if (prev == kEmpty) {
          prev = atomicCAS(tkey + s, kEmpty, kw);
          if (prev == kEmpty) {
            if (multi)
              for (int k = 0; k < nk; ++k) skv[(size_t)s * nk + k] = kv[k];
            const int num = copies > 1 && *(volatile int*)&keysN < kHotKeys ? atomicAdd(&keysN, 1) : kHotKeys;
            if (num < kHotKeys) *(volatile unsigned char*)(number + s) = (unsigned char)num;
            prev = kw;
          }
        }
        if (prev == kw) {
          hit = true;
          break;
        }
        s = (s + 1) & (S - 1);
      }
      if (hit) {  // behind the probes, where the lanes that found a slot are together again
        const unsigned num = *(volatile unsigned char*)(number + s);
        const unsigned e = num < kHotKeys ? S + num * copies + (lane & (copies - 1)) : s;
        compactAdd(ev, true, x, t64, t32, e, E);
        return;
      }
    }
    // bound for the global table: reserve a buffer entry (one shared atomic per warp)
    const unsigned m = __activemask();
    const int leader = __ffs(m) - 1, rank = __popc(m & ((1u << lane) - 1));
    int base = 0;
    if (lane == leader) base = atomicAdd(&spillN, __popc(m));
    base = __shfl_sync(m, base, leader);
    const int at = base + rank;
    appended = true;
    if (at < B) {
      u64* e = buf + (size_t)at * rw;
      for (int w = 1; w < rw; ++w) e[w] = x[w];
      e[0] = kw;
      if (multi)
        for (int k = 0; k < nk; ++k) bkv[(size_t)at * nk + k] = kv[k];
    } else if (!*(volatile int*)(L.err + 1)) {
      globalInsert(L, ev, kw, kv, x, globalPeek(L, ev, kw));
    }
  };
  // Inserts the buffered rows; returns true (in every thread) once the global table has overflowed: the run's result is
  // discarded then (the caller reruns with a bigger table), so the CTA stops.
  auto flush = [&]() -> bool {
    if (!__syncthreads_or(appended)) return false;
    // every thread is past its appends and none appends before the last barrier below
    const int missed = spillN, n = min(missed, B);
    if constexpr (!Ev::COMPACT) skip = skip > 0 ? skip - 1 : missed > kTile / 4 ? kSkipTiles : 0;
    if (threadIdx.x == 0) stopFlag = *(volatile int*)(L.err + 1);
    __syncthreads();
    if (threadIdx.x == 0) spillN = 0;
    appended = false;
    if (stopFlag) return true;
    insertAll(
        L, ev, n, [&](int j) { return buf[(size_t)j * rw]; },
        [&](int j, u64 kw, u64 first) {
          const u64* e = buf + (size_t)j * rw;
          double kv[WS_MAX_KEYS];
          if (multi)
            for (int k = 0; k < nk; ++k) kv[k] = bkv[(size_t)j * nk + k];
          globalInsert(L, ev, kw, kv, e, first);
        });
    __syncthreads();  // the buffer is refilled by the next tile
    return false;
  };
  forEachRowTiles(L, ev, rowFn, flush);
  __syncthreads();  // every tile ended with a flush: only the shared table is left (an overflowed run merges nothing)
  insertAll(
      L, ev, S, [&](int s) { return tkey[s]; },
      [&](int s, u64 kw, u64 first) {
        if (kw == kEmpty) return;
        double kv[WS_MAX_KEYS];
        if (multi)
          for (int k = 0; k < nk; ++k) kv[k] = skv[(size_t)s * nk + k];
        u64 w[Ev::RW];
        rowIdentity(ev, w);
        compactInto(ev, true, w, t64, t32, s, E);
        if (number[s] < kHotKeys)
          for (int c = 0; c < copies; ++c) compactInto(ev, true, w, t64, t32, S + number[s] * copies + c, E);
        globalInsert(L, ev, kw, kv, w, first);
      });
}

// ------------------------------------------------------------------ selection
// One pass over the predicate's columns: a bit per row in selMask (32 words per tile, row r of the tile at bit r % 32 of
// word r / 32) and the selected rows per tile.  The indices are written from the mask (kSelectWrite,
// ws_select_join.cu) after a scan of the tile counts.
template <class Ev>
__device__ void selectMask(const Launch& L) {
  __shared__ int cnt[2];
  Ev ev(L);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  int turn = 0;
  forEachOwnedTile(L, ev, [&](i64 t, int, i64 r0, i64 n, const uint32_t* del) {
    unsigned sel = 0;
    if (r0 < n) {
      const int nv = n - r0 >= 4 ? 4 : (int)(n - r0);
      ev.load(r0, ev.fastOk && nv == 4, nv);
      unsigned live = (1u << nv) - 1;
      if (del) live &= ~(__ldg(del + (r0 >> 5)) >> (r0 & 31)) & 0xfu;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (((live >> i) & 1u) && ev.where(i)) sel |= 1u << i;
    }
    unsigned word = sel << (4 * (lane & 7));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, o);
    if ((lane & 7) == 0) L.selMask[t * (kTile / 32) + threadIdx.x / 8] = word;
    const int c = __reduce_add_sync(0xffffffffu, __popc(sel));
    if (lane == 0 && c) atomicAdd(&cnt[turn], c);
    __syncthreads();
    // cnt[turn] is next added to two tiles on, after the next barrier, which thread 0 reaches behind this
    if (threadIdx.x == 0) L.tileCount[t] = cnt[turn], cnt[turn] = 0;
    turn ^= 1;
    return false;
  });
  ev.finish();
}

}  // namespace ws

// Kernel entry points (extern "C" names so generated modules can be looked up by name).  The Launch
// descriptor is a __grid_constant__ parameter: the evaluator keeps a reference to it without forcing a
// per-thread copy.
#define WS_K_ENTRY_B(PREFIX, NAME, BODY, THREADS, MINB)                                                      \
  extern "C" __global__ void __launch_bounds__(THREADS, MINB) PREFIX##_##NAME(const __grid_constant__ ws::Launch L) { \
    BODY(L);                                                                                                 \
  }
#define WS_K_ENTRY(PREFIX, NAME, BODY) WS_K_ENTRY_B(PREFIX, NAME, BODY, ws::kStagedThreads, 1)
// The same body serving several queries in one launch: each CTA finds its query (binary search of the
// CTA ranges) and runs the body on a shared-memory copy of that query's descriptor with its CTA range.
#define WS_K_MULTI_B(PREFIX, NAME, BODY, THREADS, MINB)                                                       \
  extern "C" __global__ void __launch_bounds__(THREADS, MINB) PREFIX##_multi_##NAME(const __grid_constant__ ws::MultiLaunch M) { \
    __shared__ __align__(16) ws::Launch Lq;                                                                 \
    int lo = 0, hi = M.nq - 1;                                                                               \
    while (lo < hi) {                                                                                        \
      const int mid = (lo + hi + 1) >> 1;                                                                    \
      if (M.ctaStart[mid] <= (int)blockIdx.x) lo = mid;                                                      \
      else hi = mid - 1;                                                                                     \
    }                                                                                                        \
    const unsigned long long* src = (const unsigned long long*)(M.q + lo);                                  \
    for (int w = threadIdx.x; w < (int)(sizeof(ws::Launch) / 8); w += blockDim.x) ((unsigned long long*)&Lq)[w] = src[w]; \
    __syncthreads();                                                                                         \
    if (threadIdx.x == 0) Lq.ctaBase = M.ctaStart[lo], Lq.ctaGrid = M.ctaStart[lo + 1] - M.ctaStart[lo];    \
    __syncthreads();                                                                                         \
    BODY(Lq);                                                                                                \
  }
#define WS_K_MULTI_NOKEYS(EV, PREFIX) \
  WS_K_MULTI_B(PREFIX, nokeys, (ws::aggNoKeys<EV, false>), ws::kThreads, EV::NOKEYS_MIN_BLOCKS)
#define WS_K_MULTI_DENSE_PRIV(EV, PREFIX) \
  WS_K_MULTI_B(PREFIX, dense_priv, (ws::aggDensePriv<EV, false>), ws::kThreads, EV::PRIV_MIN_BLOCKS)
// The hash scan launches kThreads.  For generated plans EV::HASH_MULTI_MIN_BLOCKS resident CTAs (three, two of wide
// plans: hashMinBlocks) bound the registers: reading the launch descriptor from shared memory takes more of them than
// the single-query scan does, and unbounded it ran two CTAs per SM and 20 % longer; bounded to 80 registers five
// aggregates need no spills, seven SUMs 48 bytes.
#define WS_K_MULTI_HASH(EV, PREFIX) \
  WS_K_MULTI_B(PREFIX, hash, ws::aggHash<EV>, ws::kThreads, EV::HASH_MULTI_MIN_BLOCKS)
// Direct loads: EV::NOKEYS_MIN_BLOCKS resident CTAs of kThreads; the staged entry keeps the producer warp.
#define WS_K_NOKEYS(EV, PREFIX) \
  WS_K_ENTRY_B(PREFIX, nokeys, (ws::aggNoKeys<EV, false>), ws::kThreads, EV::NOKEYS_MIN_BLOCKS)
#define WS_K_NOKEYS_STAGED(EV, PREFIX) WS_K_ENTRY(PREFIX, nokeys_staged, (ws::aggNoKeys<EV, true>))
#define WS_K_DENSE_SHARED(EV, PREFIX) \
  WS_K_ENTRY_B(PREFIX, dense_shared, (ws::aggDenseShared<EV, false>), (ws::kThreads * EV::DENSE_V), 1)
#define WS_K_DENSE_TOPS(EV, PREFIX) \
  WS_K_ENTRY_B(PREFIX, dense_tops, (ws::aggDenseShared<EV, true>), (ws::kThreads * EV::DENSE_V), 1)
#define WS_K_DENSE_GLOBAL(EV, PREFIX) WS_K_ENTRY(PREFIX, dense_global, ws::aggDenseGlobal<EV>)
// The direct-load private-row kernel asks for EV::PRIV_MIN_BLOCKS resident CTAs of kThreads (a
// register budget); the staged one keeps the producer warp.
#define WS_K_DENSE_PRIV(EV, PREFIX)                                                                      \
  WS_K_ENTRY_B(PREFIX, dense_priv, (ws::aggDensePriv<EV, false>), ws::kThreads, EV::PRIV_MIN_BLOCKS)
#define WS_K_DENSE_PRIV_STAGED(EV, PREFIX) WS_K_ENTRY(PREFIX, dense_priv_staged, (ws::aggDensePriv<EV, true>))
#define WS_K_HASH(EV, PREFIX) WS_K_ENTRY_B(PREFIX, hash, ws::aggHash<EV>, ws::kThreads, EV::HASH_MIN_BLOCKS)
#define WS_K_SELECT(EV, PREFIX) WS_K_ENTRY_B(PREFIX, select, ws::selectMask<EV>, ws::kThreads, EV::SELECT_MIN_BLOCKS)
