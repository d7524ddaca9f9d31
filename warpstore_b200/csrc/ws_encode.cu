// Segment encoding on the GPU (the flush path of the engine's storage: src/storage.cu:1138-1192 encodes
// segment columns on the host): integer columns to the bit-packed (enc 7) or run-length (enc 8)
// formats that the scan kernels decode (formats: ws_dev.cuh), and any column to the engine's own
// formats by the engine's rule (ws_encode_column_engine: frame of reference, dictionary, decimal).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "ws_internal.h"

namespace ws {
namespace {

int gridFor(int64_t n, int block = 256, int perSm = 8) {
  int64_t g = (n + block - 1) / block;
  const int64_t cap = (int64_t)smCount() * perSm;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}
#define WS_LAUNCH(kernel, grid, block, smem, ...)               \
  do {                                                          \
    kernel<<<(grid), (block), (smem), stream()>>>(__VA_ARGS__); \
    WS_CK(cudaGetLastError());                                  \
    countLaunch();                                              \
  } while (0)
#define WS_GRID_STRIDE(j, n) \
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < (n); j += (int64_t)gridDim.x * blockDim.x)

__device__ __forceinline__ long long rawAt(const void* src, int i32, int64_t i) {
  return i32 ? (long long)((const int*)src)[i] : ((const long long*)src)[i];
}

// Order-preserving unsigned image of an int64 (and its inverse): statistics words that are only ever
// lowered, so that one memset of 0xff sets all their identities.
WS_DI u64 ordU(long long v) { return (u64)v ^ 0x8000000000000000ull; }
inline long long unordU(u64 u) { return (long long)(u ^ 0x8000000000000000ull); }

// The CTA's minimum of m (u64) into *out with one atomic per CTA, skipped when *out is already as low.  The
// statistics kernels were bound by same-address atomics of every warp: 2^20 rows of kMinMax took 14.3 us
// (up to 9472 warps x 2 atomics), kDecimalStats 91.5 us (x 10); with one set per CTA 5.7 and 11.3 us.
WS_DI void ctaAtomicMin(u64 m, u64* red, unsigned long long* out) {
#pragma unroll
  for (int o = 16; o; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
  __syncthreads();  // red is reused from call to call
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = min(m, red[w]);
    if (m < *(volatile unsigned long long*)out) atomicMin(out, m);
  }
}

// st (all bytes 0xff before): st[0] = ordU(min) of the non-NULL values, st[1] = ~ordU(max)
__global__ void kMinMax(const void* src, int i32, long long nul, int64_t n, unsigned long long* st) {
  __shared__ u64 red[32];
  u64 mn = ~0ull, mx = ~0ull;
  WS_GRID_STRIDE(i, n) {
    const long long v = rawAt(src, i32, i);
    if (v != nul) mn = min(mn, ordU(v)), mx = min(mx, ~ordU(v));
  }
  ctaAtomicMin(mn, red, st);
  ctaAtomicMin(mx, red, st + 1);
}

// Segment header (16 bytes) and the 16 pad bytes after the payload, written by the encoding kernels' first CTA
struct SegFrame {
  uint8_t* seg;          // segment column
  long long h0;          // header words
  u64 h1;
  int64_t payload;       // bytes between the header and the pad
};
WS_DI void writeFrame(const SegFrame& f) {
  if (blockIdx.x != 0) return;
  if (threadIdx.x == 0) ((long long*)f.seg)[0] = f.h0, ((u64*)f.seg)[1] = f.h1;
  if (threadIdx.x < 16) f.seg[WS_ENC_HEADER + f.payload + threadIdx.x] = 0;
}

// bit-packed words: word w holds bits [32w, 32w + 32) of the code stream
__global__ void kPack(const void* src, int i32, long long nul, int64_t n, long long base, int b, int64_t nwords,
                      unsigned* words, SegFrame f) {
  writeFrame(f);
  const unsigned nulc = b == 32 ? 0xffffffffu : ((1u << b) - 1u);
  WS_GRID_STRIDE(w, nwords) {
    const u64 lo = (u64)w * 32, hi = lo + 32;  // bit range of this word
    unsigned out = 0;
    for (u64 row = lo / (u64)b; row < (u64)n && row * (u64)b < hi; ++row) {
      const long long v = rawAt(src, i32, (int64_t)row);
      const unsigned code = v == nul ? nulc : (unsigned)(v - base);
      const u64 start = row * (u64)b;
      if (start >= lo) out |= code << (start - lo);
      else out |= code >> (lo - start);
    }
    words[w] = out;
  }
}

// run starts: row i starts a run when it is row 0 or differs from row i - 1
__global__ void kRunCount(const void* src, int i32, int64_t n, int64_t* counts) {
  __shared__ int wsum[8];
  const int64_t i0 = (int64_t)blockIdx.x * 1024 + threadIdx.x * 4;
  int c = 0;
  for (int k = 0; k < 4; ++k) {
    const int64_t i = i0 + k;
    c += i < n && (i == 0 || rawAt(src, i32, i) != rawAt(src, i32, i - 1));
  }
  for (int o = 16; o; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < 8; ++w) t += wsum[w];
    counts[blockIdx.x] = t;
  }
}
__global__ void kScanChunks(int64_t* counts, int64_t n) {  // exclusive scan in place, total in counts[n]
  __shared__ int64_t part[1024];
  const int t = threadIdx.x, T = blockDim.x;
  const int64_t per = (n + T - 1) / T;
  const int64_t lo = min((int64_t)t * per, n), hi = min(lo + per, n);
  int64_t s = 0;
  for (int64_t i = lo; i < hi; ++i) s += counts[i];
  part[t] = s;
  __syncthreads();
  for (int off = 1; off < T; off <<= 1) {
    const int64_t v = t >= off ? part[t - off] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int64_t run = t ? part[t - 1] : 0;
  for (int64_t i = lo; i < hi; ++i) {
    const int64_t c = counts[i];
    counts[i] = run;
    run += c;
  }
  if (t == T - 1) counts[n] = part[T - 1];
}
// run k: starts[k] = its first row, vals[k] = its value (in order)
__global__ void kRunWrite(const void* src, int i32, int64_t n, const int64_t* offs, int* starts, long long* vals) {
  __shared__ int wsum[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * 1024 + threadIdx.x * 4;
  bool f[4];
  int c = 0;
  for (int k = 0; k < 4; ++k) {
    const int64_t i = i0 + k;
    f[k] = i < n && (i == 0 || rawAt(src, i32, i) != rawAt(src, i32, i - 1));
    c += f[k];
  }
  int incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += wsum[w];
  int64_t at = offs[blockIdx.x] + before + incl - c;
  for (int k = 0; k < 4; ++k)
    if (f[k]) starts[at] = (int)(i0 + k), vals[at] = rawAt(src, i32, i0 + k), ++at;
}
__global__ void kRunEnds(const int* starts, int64_t runs, int64_t n, int* ends, SegFrame f) {
  writeFrame(f);
  if ((runs & 1) && blockIdx.x == 0 && threadIdx.x == 0) ends[runs] = 0;  // the run ends are padded to 8 bytes
  WS_GRID_STRIDE(k, runs) ends[k] = k + 1 < runs ? starts[k + 1] : (int)n;
}

// ---- the engine's formats (src/storage.cu:1093-1192).  enc 1/2/3: integer offsets from the minimum as
// uint8 / uint16 / uint32 (all-ones = NULL); enc 4: a dictionary of at most 255 distinct doubles (bit
// patterns, in order of first occurrence) and uint8 codes; enc 5/6: doubles that are exact decimals,
// llround(x * 10^s) - minimum as uint16 / uint32 (all-ones = NaN).  Header: int64 base (the minimum),
// double 10^s (enc 5/6); enc 4's 256 dictionary entries follow the header.
__global__ void kEncodeFor(const void* src, int i32, long long nul, int64_t n, long long mn, int w, SegFrame f) {
  writeFrame(f);
  uint8_t* d = f.seg + WS_ENC_HEADER;
  WS_GRID_STRIDE(i, n) {
    const long long v = rawAt(src, i32, i);
    const u64 code = v == nul ? ~0ull : (u64)v - (u64)mn;
    if (w == 1) d[i] = (uint8_t)code;
    else if (w == 2) ((uint16_t*)d)[i] = (uint16_t)code;
    else ((uint32_t*)d)[i] = (uint32_t)code;
  }
}

// Distinct bit patterns of a double column, up to 255 of them: a 4096-slot open-addressing set
// (key 0 = empty; the pattern 0, +0.0, has its own flag) with each pattern's first row (atomicMin).
// Once more than 255 patterns were claimed, *over is set and the threads stop inserting.
//
// Each CTA collects its rows' patterns in a shared-memory set first and merges that set (at most 255
// entries) into the global one at its end: a column worth a dictionary has few patterns, so inserting
// every row into the global set meant a million atomics on a few addresses (a column of 2^20 rows with 11
// patterns and one with millions: 26.9 ms for the two; through the shared sets 0.015 ms).  A row whose pattern is known costs two shared loads.  A CTA that
// sees more than 255 patterns raises *over and ends: at most 255 + blockDim.x patterns are inserted before
// every thread of the CTA has noticed, below the 1024 slots.
constexpr int kDictSlots = 4096, kDictLocal = 1024, kDictThreads = 256;
constexpr long long kFirstNone = 0x7f7f7f7f7f7f7f7fll;  // "no row yet" (the first-row arrays' memset value)
constexpr int kFirstNone32 = 0x7fffffff;
__global__ void __launch_bounds__(kDictThreads) kDictInsert(const double* x, int64_t n, u64* keys, long long* first,
                                                            long long* zeroFirst, int* count, int* over) {
  __shared__ u64 lkey[kDictLocal];
  __shared__ int lfirst[kDictLocal];
  __shared__ int lzero, lcount;
  for (int s = threadIdx.x; s < kDictLocal; s += blockDim.x) lkey[s] = 0, lfirst[s] = kFirstNone32;
  if (threadIdx.x == 0) lzero = kFirstNone32, lcount = 0;
  __syncthreads();
  bool stop = false;
  WS_GRID_STRIDE(i, n) {
    if (*(volatile int*)&lcount > 255) {
      stop = true;
      break;
    }
    const u64 b = (u64)__double_as_longlong(x[i]);
    const int r = (int)i;
    if (b == 0) {
      if (r < *(volatile int*)&lzero && atomicMin(&lzero, r) == kFirstNone32) atomicAdd(&lcount, 1);
      continue;
    }
    unsigned s = (unsigned)(mix64(b) & (kDictLocal - 1));
    for (int p = 0; p < kDictLocal; ++p) {
      u64 prev = *(volatile u64*)(lkey + s);
      if (prev == 0) {
        prev = atomicCAS((unsigned long long*)(lkey + s), 0ull, b);
        if (prev == 0) atomicAdd(&lcount, 1);
      }
      if (prev == 0 || prev == b) {
        if (r < *(volatile int*)(lfirst + s)) atomicMin(lfirst + s, r);
        break;
      }
      s = (s + 1) & (kDictLocal - 1);
    }
  }
  if (__syncthreads_or(stop || lcount > 255)) {
    if (threadIdx.x == 0) *over = 1;
    return;
  }
  if (threadIdx.x == 0 && lzero != kFirstNone32 && *(volatile long long*)zeroFirst > lzero &&
      atomicMin(zeroFirst, (long long)lzero) == kFirstNone && atomicAdd(count, 1) >= 255)
    *over = 1;
  for (int e = threadIdx.x; e < kDictLocal; e += blockDim.x) {
    const u64 b = lkey[e];
    if (b == 0 || *(volatile int*)over) continue;
    unsigned s = (unsigned)(mix64(b) & (kDictSlots - 1));
    for (int p = 0; p < kDictSlots; ++p) {
      u64 prev = *(volatile u64*)(keys + s);
      if (prev == 0ull) {
        prev = atomicCAS((unsigned long long*)(keys + s), 0ull, b);
        if (prev == 0ull && atomicAdd(count, 1) >= 255) *over = 1;
      }
      if (prev == 0ull || prev == b) {
        if (*(volatile long long*)(first + s) > lfirst[e]) atomicMin(first + s, (long long)lfirst[e]);
        break;
      }
      s = (s + 1) & (kDictSlots - 1);
    }
  }
}
// The set's patterns ranked by first row: dictionary entries in order of first occurrence (zeros past the
// last), each slot's code, the code of +0.0 in code[kDictSlots], and the segment's frame.  One CTA.
__global__ void __launch_bounds__(1024) kDictRank(const u64* keys, const long long* first, uint8_t* code, SegFrame f) {
  __shared__ long long ef[256];
  __shared__ int es[256], cnt;
  writeFrame(f);
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  for (int s = threadIdx.x; s <= kDictSlots; s += blockDim.x) {  // slot kDictSlots stands for +0.0
    if (s < kDictSlots ? keys[s] == 0 : first[s] == kFirstNone) continue;
    const int at = atomicAdd(&cnt, 1);
    if (at < 256) ef[at] = first[s], es[at] = s;
  }
  __syncthreads();
  const int n = min(cnt, 256);
  double* dict = (double*)(f.seg + WS_ENC_HEADER);
  for (int e = threadIdx.x; e < 256; e += blockDim.x) {
    if (e >= n) {
      dict[e] = 0.0;
      continue;
    }
    int rank = 0;
    for (int o = 0; o < n; ++o) rank += ef[o] < ef[e];  // first rows are distinct
    code[es[e]] = (uint8_t)rank;
    dict[rank] = es[e] == kDictSlots ? 0.0 : __longlong_as_double((long long)keys[es[e]]);
  }
}
// codes of the set's patterns (code[slot]; code[kDictSlots] for +0.0) -> uint8 codes of the rows
__global__ void kDictEncode(const double* x, int64_t n, const u64* keys, const uint8_t* code, uint8_t* d) {
  WS_GRID_STRIDE(i, n) {
    const u64 b = (u64)__double_as_longlong(x[i]);
    uint8_t c;
    if (b == 0) {
      c = code[kDictSlots];
    } else {
      unsigned s = (unsigned)(mix64(b) & (kDictSlots - 1));
      for (int p = 0; p < kDictSlots && keys[s] != b; ++p) s = (s + 1) & (kDictSlots - 1);
      c = code[s];
    }
    d[i] = c;
  }
}

// Decimal doubles: for each scale s = 0..4 (p = 10^s), whether every non-NaN x has |x p| < 4e15 and
// llround(x p) / p == x, and the min / max of llround(x p), in words that are 0xff.. before: st[3s] = 0 when
// not exact, st[3s+1] = ordU(min), st[3s+2] = ~ordU(max) (kept for exact scales).
__global__ void kDecimalStats(const double* x, int64_t n, unsigned long long* st) {
  __shared__ u64 red[32];
  int bad[5] = {0, 0, 0, 0, 0};
  long long mn[5], mx[5];
  double p = 1.0;
#pragma unroll
  for (int s = 0; s < 5; ++s) mn[s] = LLONG_MAX, mx[s] = LLONG_MIN;
  WS_GRID_STRIDE(i, n) {
    const double v = x[i];
    if (v != v) continue;
    p = 1.0;
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      const double y = v * p;
      if (bad[s]) {
      } else if (!(fabs(y) < 4e15)) {
        bad[s] = 1;
      } else {
        const long long k = llround(y);
        if ((double)k / p != v) bad[s] = 1;
        mn[s] = min(mn[s], k), mx[s] = max(mx[s], k);
      }
      p *= 10.0;
    }
  }
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    if (__syncthreads_or(bad[s])) {
      if (threadIdx.x == 0) st[3 * s] = 0;
      continue;
    }
    ctaAtomicMin(mn[s] <= mx[s] ? ordU(mn[s]) : ~0ull, red, st + 3 * s + 1);
    ctaAtomicMin(mn[s] <= mx[s] ? ~ordU(mx[s]) : ~0ull, red, st + 3 * s + 2);
  }
}
__global__ void kDecimalEncode(const double* x, int64_t n, double p, long long mn, int w, SegFrame f) {
  writeFrame(f);
  uint8_t* d = f.seg + WS_ENC_HEADER;
  WS_GRID_STRIDE(i, n) {
    const double v = x[i];
    const u64 code = v != v ? ~0ull : (u64)(llround(v * p) - mn);
    if (w == 2) ((uint16_t*)d)[i] = (uint16_t)code;
    else ((uint32_t*)d)[i] = (uint32_t)code;
  }
}

}  // namespace
}  // namespace ws

using namespace ws;

extern "C" {

int ws_encode_column(const void* src, int t, int64_t n, int enc, void** out, int64_t* bytes, int* enc_used) {
  return guardedCall([&] {
    *out = nullptr;
    *bytes = 0;
    if (!(t == WS_T_I32 || t == WS_T_I64 || t == WS_T_I32N || t == WS_T_I64N))
      throw Error("encode: integer columns only", WS_ERR_ARG);
    if (enc != 0 && enc != 7 && enc != 8) throw Error("encode: enc must be 0 (choose), 7 or 8", WS_ERR_ARG);
    if (n < 0 || n > INT32_MAX) throw Error("encode: segment row count out of range", WS_ERR_ARG);
    const int i32 = t == WS_T_I32 || t == WS_T_I32N;
    const long long nul = i32 ? (long long)WS_NULL_I32 : (long long)WS_NULL_I64;
    // statistics: min / max and the run count
    DBuf<unsigned long long> st(2);
    WS_CK(cudaMemsetAsync(st.p, 0xff, 8 * 2, stream()));
    if (n) WS_LAUNCH(kMinMax, gridFor(n, 256, 4), 256, 0, src, i32, nul, n, st.p);
    const int64_t nchunks = std::max<int64_t>((n + 1023) / 1024, 1);
    DBuf<int64_t> counts(nchunks + 1);
    if (n) {
      WS_LAUNCH(kRunCount, (unsigned)nchunks, 256, 0, src, i32, n, counts.p);
      WS_LAUNCH(kScanChunks, 1, 1024, 0, counts.p, nchunks);
    } else {
      WS_CK(cudaMemsetAsync(counts.p, 0, 8 * (nchunks + 1), stream()));
    }
    unsigned long long hs[2];
    int64_t runs = 0;
    WS_CK(cudaMemcpyAsync(hs, st.p, sizeof hs, cudaMemcpyDeviceToHost, stream()));
    WS_CK(cudaMemcpyAsync(&runs, counts.p + nchunks, 8, cudaMemcpyDeviceToHost, stream()));
    sync();
    const long long vmin = unordU(hs[0]), vmax = unordU(~hs[1]);
    const bool anyValue = vmin <= vmax;
    const long long base = anyValue ? vmin : 0;
    const unsigned long long range = anyValue ? (unsigned long long)vmax - (unsigned long long)vmin : 0;
    int b = 1;  // codes 0 .. range, the all-ones code reserved for NULL
    while (b < 64 && (range + 1) >> b) ++b;
    const int64_t nwords = (n * (int64_t)b + 31) / 32;
    const int64_t packBytes = b <= 32 ? WS_ENC_HEADER + 4 * nwords + 16 : INT64_MAX;
    const int64_t rleBytes = WS_ENC_HEADER + ((runs * 4 + 7) & ~7ll) + 8 * runs + 16;
    int use = enc;
    if (use == 0) use = rleBytes < packBytes ? 8 : 7;
    if (use == 7 && b > 32) throw Error("encode: value range too wide to bit-pack (more than 32 bits)", WS_ERR_RANGE);
    const int64_t total = use == 7 ? packBytes : rleBytes;
    DBuf<uint8_t> buf(total);
    const SegFrame frame{buf.p, use == 7 ? base : (long long)runs, use == 7 ? (u64)b : 0,
                         total - WS_ENC_HEADER - 16};
    if (use == 7) {
      WS_LAUNCH(kPack, gridFor(nwords), 256, 0, src, i32, nul, n, base, b, nwords, (unsigned*)(buf.p + 16), frame);
    } else {
      DBuf<int> starts(std::max<int64_t>(runs, 1));
      int* ends = (int*)(buf.p + WS_ENC_HEADER);
      long long* vals = (long long*)(buf.p + WS_ENC_HEADER + ((runs * 4 + 7) & ~7ll));
      if (runs) WS_LAUNCH(kRunWrite, (unsigned)nchunks, 256, 0, src, i32, n, counts.p, starts.p, vals);
      WS_LAUNCH(kRunEnds, gridFor(runs), 256, 0, starts.p, runs, n, ends, frame);
    }
    *out = buf.release();
    *bytes = total;
    if (enc_used) *enc_used = use;
  });
}

int ws_encode_column_engine(const void* src, int ptype, int64_t n, void** out, int64_t* bytes, int* enc_used) {
  return guardedCall([&] {
    *out = nullptr;
    *bytes = 0;
    *enc_used = 0;
    if (ptype != WS_PT_I32 && ptype != WS_PT_I64 && ptype != WS_PT_F64)
      throw Error("encode: ptype must be I32, I64 or F64", WS_ERR_ARG);
    if (n < 0 || n > INT32_MAX) throw Error("encode: segment row count out of range", WS_ERR_ARG);
    if (n < 1024) return;  // the engine keeps short columns raw
    auto finish = [&](DBuf<uint8_t>& buf, int64_t total, int e) {
      *out = buf.release();
      *bytes = total;
      *enc_used = e;
    };
    if (ptype != WS_PT_F64) {  // frame of reference
      const int i32 = ptype == WS_PT_I32;
      const long long nul = i32 ? (long long)WS_NULL_I32 : (long long)WS_NULL_I64;
      DBuf<unsigned long long> st(2);
      WS_CK(cudaMemsetAsync(st.p, 0xff, 8 * 2, stream()));
      WS_LAUNCH(kMinMax, gridFor(n, 256, 4), 256, 0, src, i32, nul, n, st.p);
      unsigned long long hs[2];
      d2hSync(hs, st.p, sizeof hs);
      long long mn = unordU(hs[0]), mx = unordU(~hs[1]);
      if (mn > mx) mn = mx = 0;  // every value NULL
      const unsigned long long range = (unsigned long long)mx - (unsigned long long)mn;
      const int e = range < 0xFFull ? 1 : range < 0xFFFFull ? 2 : (!i32 && range < 0xFFFFFFFFull) ? 3 : 0;
      if (!e) return;
      const int w = e == 1 ? 1 : e == 2 ? 2 : 4;
      const int64_t total = WS_ENC_HEADER + n * w + 16;
      DBuf<uint8_t> buf(total);
      WS_LAUNCH(kEncodeFor, gridFor(n), 256, 0, src, i32, nul, n, mn, w, SegFrame{buf.p, mn, 0, n * w});
      finish(buf, total, e);
      return;
    }
    const double* x = (const double*)src;
    // dictionary of at most 255 distinct bit patterns, in order of first occurrence
    {
      DBuf<u64> keys(kDictSlots);
      DBuf<long long> first(kDictSlots + 1);
      DBuf<int> ctl(2);  // [0] count, [1] over
      WS_CK(cudaMemsetAsync(keys.p, 0, 8 * kDictSlots, stream()));
      WS_CK(cudaMemsetAsync(first.p, 0x7f, 8 * (kDictSlots + 1), stream()));  // kFirstNone
      WS_CK(cudaMemsetAsync(ctl.p, 0, 8, stream()));
      WS_LAUNCH(kDictInsert, gridFor(n, kDictThreads, 2), kDictThreads, 0, x, n, keys.p, first.p, first.p + kDictSlots,
                ctl.p, ctl.p + 1);
      int hc[2];
      d2hSync(hc, ctl.p, 8);
      if (!hc[1] && hc[0] <= 255) {
        const int64_t payload = 256 * 8 + n, total = WS_ENC_HEADER + payload + 16;
        DBuf<uint8_t> buf(total);
        DBuf<uint8_t> code(kDictSlots + 1);
        WS_LAUNCH(kDictRank, 1, 1024, 0, keys.p, first.p, code.p, SegFrame{buf.p, 0, 0, payload});
        WS_LAUNCH(kDictEncode, gridFor(n), 256, 0, x, n, keys.p, code.p, buf.p + WS_ENC_HEADER + 256 * 8);
        finish(buf, total, 4);
        return;
      }
    }
    // decimal doubles: the first scale s at which every value is an exact decimal decides
    DBuf<unsigned long long> st(15);
    WS_CK(cudaMemsetAsync(st.p, 0xff, 8 * 15, stream()));
    WS_LAUNCH(kDecimalStats, gridFor(n, 256, 4), 256, 0, x, n, st.p);
    unsigned long long hs[15];
    d2hSync(hs, st.p, sizeof hs);
    double p = 1.0;
    for (int sc = 0; sc < 5; ++sc, p *= 10.0) {
      if (hs[3 * sc] == 0) continue;  // not every value is exact at this scale
      long long mn = unordU(hs[3 * sc + 1]), mx = unordU(~hs[3 * sc + 2]);
      if (mn > mx) mn = mx = 0;
      const unsigned long long range = (unsigned long long)(mx - mn);
      const int e = range < 0xFFFFull ? 5 : range < 0xFFFFFFFFull ? 6 : 0;
      if (!e) return;
      const int w = e == 5 ? 2 : 4;
      const int64_t total = WS_ENC_HEADER + n * w + 16;
      DBuf<uint8_t> buf(total);
      u64 pbits;
      memcpy(&pbits, &p, 8);
      WS_LAUNCH(kDecimalEncode, gridFor(n), 256, 0, x, n, p, mn, w, SegFrame{buf.p, mn, pbits, n * w});
      finish(buf, total, e);
      return;
    }
  });
}

}  // extern "C"
