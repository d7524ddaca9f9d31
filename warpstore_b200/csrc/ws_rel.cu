// Relational helpers around the scan / join operators: join-filter key bitmaps and deleted bits,
// dictionary code remaps, NULL-aware and encoded gathers, expression evaluation at row indices
// (projection and post-aggregation keys), and the stable multi-key sort permutation of ORDER BY
// (reference: src/gpu.cu:149-163, :802-888, :1011-1087, :1323-1367).
#include <climits>
#include <cmath>
#include <cstring>

#include "ws_internal.h"
#include "ws_interp.cuh"

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

// ---------------------------------------------------------------- bitmaps, codes, gathers
// Join-key values are read like the join's keys: I32 widened, I64 as stored, F64 truncated; the
// NULL sentinels / NaN never set a bit.
__device__ __forceinline__ bool keyOf(const ws_col_view& c, int64_t r, long long& k) {
  if (c.t == 0 || c.t == 3) {
    const int v = ((const int*)c.p)[r];
    k = v;
    return v != WS_NULL_I32;
  }
  if (c.t == 1 || c.t == 4) {
    k = ((const long long*)c.p)[r];
    return k != WS_NULL_I64;
  }
  const double d = ((const double*)c.p)[r];
  k = (long long)d;
  return d == d;
}

__global__ void kKeyBitmap(ws_col_view key, int64_t n, long long lo, int64_t nbits, uint32_t* bits) {
  WS_GRID_STRIDE(i, n) {
    long long k;
    if (!keyOf(key, i, k)) continue;
    const u64 v = (u64)k - (u64)lo;
    if (v < (u64)nbits) atomicOr(bits + (v >> 5), 1u << (v & 31));
  }
}
__global__ void kSetBits(uint32_t* bits, const int32_t* idx, int64_t m) {
  WS_GRID_STRIDE(j, m) atomicOr(bits + (idx[j] >> 5), 1u << (idx[j] & 31));
}
__global__ void kRemapCodes(const int32_t* in, int64_t n, const int32_t* map, int64_t mapN, int32_t* out) {
  WS_GRID_STRIDE(j, n) {
    const int32_t c = in[j];
    out[j] = c == WS_NULL_I32 ? WS_NULL_I32 : (c >= 0 && c < mapN) ? __ldg(map + c) : -2;
  }
}
__global__ void kBitsToDouble(const double* src, int64_t n, double* dst) {
  WS_GRID_STRIDE(j, n) dst[j] = (double)__double_as_longlong(src[j]);
}
template <class T>
__global__ void kGatherNull(const T* src, const int32_t* idx, int64_t m, T* dst, T nul) {
  WS_GRID_STRIDE(j, m) dst[j] = idx[j] < 0 ? nul : src[idx[j]];
}
// fixed-size elements of `words` 32-bit words; index -1 gives a NULL element (NaN floats when nulls,
// else zeros)
__global__ void kGatherWords(const uint32_t* src, int words, const int32_t* idx, int64_t m, uint32_t* dst, int nulls) {
  WS_GRID_STRIDE(j, m * words) {
    const int64_t r = j / words, w = j % words;
    const int32_t i = idx[r];
    dst[j] = i < 0 ? (nulls ? 0x7fc00000u : 0u) : src[(int64_t)i * words + w];
  }
}
// encoded segment column -> raw values (NULL sentinels kept as stored for integers)
__global__ void kGatherEnc(ws_col_view v, int ptype, const int32_t* idx, int64_t m, void* dst) {
  WS_GRID_STRIDE(j, m) {
    const i64 r = idx[j];
    if (ptype == WS_PT_F64) ((double*)dst)[j] = colDblAt(v, r);
    else if (ptype == WS_PT_I32) ((int32_t*)dst)[j] = (int32_t)colIntAt(v, r);
    else ((int64_t*)dst)[j] = colIntAt(v, r);
  }
}

// ---------------------------------------------------------------- evaluation at rows
struct EvalSpec {
  const TInstr* code;
  int start, len;
  int isInt;                // the program's result type
  int single;               // the program is one integer OP_COL (read exactly)
  int col;
  int simple;               // raw columns, literals and arithmetic within a stack of kSimpleDepth (kEvalSimple)
};

// Programs of raw numeric columns, literals, + - * / and negation (most ORDER BY and projection expressions), four rows
// per thread: the stack is kSimpleDepth registers per row that shift on a push, so no word goes through local
// memory and each instruction is decoded once for four rows.  The operators are the interpreter loop's.  4,000,037 rows, one
// column and price * (100 - discount) / 100.0: 120 -> 60 us for the two.
constexpr int kSimpleDepth = 4, kSimpleRows = 4;
template <bool kIntOut>
__global__ void __launch_bounds__(256) kEvalSimple(const __grid_constant__ EvalSpec s, const ws_col_view* cv,
                                                   const __grid_constant__ EnvK env, const int32_t* idx, int64_t m,
                                                   void* out) {
  for (int64_t j0 = blockIdx.x * (int64_t)(256 * kSimpleRows) + threadIdx.x; j0 < m;
       j0 += (int64_t)gridDim.x * 256 * kSimpleRows) {
    int64_t row[kSimpleRows];
    Word st[kSimpleDepth][kSimpleRows];
#pragma unroll
    for (int r = 0; r < kSimpleRows; ++r) {  // past the end: the last row again
      const int64_t j = min(j0 + r * 256, m - 1);
      row[r] = idx ? idx[j] : j;
#pragma unroll
      for (int d = 0; d < kSimpleDepth; ++d) st[d][r].i = 0;
    }
    for (int pc = s.start; pc < s.start + s.len; ++pc) {
      const TInstr in = s.code[pc];
      if (in.op == WS_OP_COL || in.op == WS_OP_CONST) {
#pragma unroll
        for (int d = kSimpleDepth - 1; d > 0; --d)
#pragma unroll
          for (int r = 0; r < kSimpleRows; ++r) st[d][r] = st[d - 1][r];
        if (in.op == WS_OP_CONST) {
#pragma unroll
          for (int r = 0; r < kSimpleRows; ++r) st[0][r].d = env.consts[in.arg];
          continue;
        }
        const void* p = cv[in.arg].p;
        const int t = cv[in.arg].t;
        i64 v[kSimpleRows];
        if (t == 0 || t == 3) {
#pragma unroll
          for (int r = 0; r < kSimpleRows; ++r) v[r] = __ldg((const int*)p + row[r]);
        } else {
#pragma unroll
          for (int r = 0; r < kSimpleRows; ++r) v[r] = __ldg((const i64*)p + row[r]);
        }
#pragma unroll
        for (int r = 0; r < kSimpleRows; ++r) {
          if (t == 3) st[0][r].d = nullIfI32(v[r]);
          else if (t == 4) st[0][r].d = nullIfI64(v[r]);
          else st[0][r].i = v[r];  // integers, or a double's bits
        }
        continue;
      }
#pragma unroll
      for (int r = 0; r < kSimpleRows; ++r) {
        Word o;
        if (in.op == WS_OP_NEG) {
          if (in.rInt) o.i = (i64)(0ull - (u64)st[0][r].i);
          else o.d = -st[0][r].d;
          st[0][r] = o;
          continue;
        }
        const Word a = st[1][r], b = st[0][r];
        if (in.op == WS_OP_DIV) {
          o.d = divz(asD(a, in.aInt), asD(b, in.bInt));
        } else if (in.rInt) {
          o.i = in.op == WS_OP_ADD ? iaddc(a.i, b.i, env.ovf) : in.op == WS_OP_SUB ? isubc(a.i, b.i, env.ovf)
                                                                : imulc(a.i, b.i, env.ovf);
        } else {
          const double x = asD(a, in.aInt), y = asD(b, in.bInt);
          o.d = in.op == WS_OP_ADD ? x + y : in.op == WS_OP_SUB ? x - y : x * y;
        }
        st[0][r] = o;
      }
      if (in.op != WS_OP_NEG) {
#pragma unroll
        for (int d = 1; d < kSimpleDepth - 1; ++d)
#pragma unroll
          for (int r = 0; r < kSimpleRows; ++r) st[d][r] = st[d + 1][r];
      }
    }
#pragma unroll
    for (int r = 0; r < kSimpleRows; ++r) {
      const int64_t j = j0 + r * 256;
      if (j >= m) continue;
      const Word w = st[0][r];
      if constexpr (kIntOut) ((i64*)out)[j] = s.isInt ? w.i : w.d != w.d ? (i64)WS_NULL_I64 : llround(w.d);
      else ((double*)out)[j] = s.isInt ? (double)w.i : w.d;
    }
  }
}

// out[j] = the program at row idx[j] (or j): doubles (NULL = NaN) ...
__global__ void kEvalAt(const __grid_constant__ EvalSpec s, const ws_col_view* cv, const __grid_constant__ EnvK env,
                        const int32_t* idx, int64_t m, double* out) {
  WS_GRID_STRIDE(j, m) {
    const Word w = vmRun(s.code, s.start, s.len, cv, idx ? idx[j] : j, env);
    out[j] = s.isInt ? (double)w.i : w.d;
  }
}
// ... or int64 (NULL = the BIGINT NULL sentinel): exact for integer programs, else the double rounded
__global__ void kEvalAtInt(const __grid_constant__ EvalSpec s, const ws_col_view* cv, const __grid_constant__ EnvK env,
                           const int32_t* idx, int64_t m, int64_t* out) {
  WS_GRID_STRIDE(j, m) {
    const i64 r = idx ? idx[j] : j;
    if (s.single) {
      const ws_col_view& c = cv[s.col];
      const i64 v = colIntAt(c, r);
      out[j] = (c.t == 0 || c.t == 3) && v == (i64)WS_NULL_I32 ? (i64)WS_NULL_I64 : v;
      continue;
    }
    const Word w = vmRun(s.code, s.start, s.len, cv, r, env);
    if (s.isInt) out[j] = w.i;
    else out[j] = w.d != w.d ? (i64)WS_NULL_I64 : llround(w.d);
  }
}

// ---------------------------------------------------------------- sort permutation
// Stable LSD radix sort of (packed key, int32 row) pairs by 8-bit digits.
//
// The sort keys are packed first: every double key becomes its order key (64 bits), of which only the bits
// between the lowest and the highest one that differ among the rows are kept (kKeyBits finds them); the
// fields of the keys, least significant key lowest, form one composite of at most 64 bits (more keys: several
// composites, sorted one after another, least significant first).  Dates, counts and cents vary in a few
// bits, so an ORDER BY of two keys is one sort of 4 to 6 digits rather than two of 16.
//
// A pass is three launches over tiles of kRTile items: digit counts per tile, a scan of each digit's counts
// over the tiles, and the scatter, in which a CTA ranks its items by digit (warp matches, in item order: the
// sort is stable), puts them in order in shared memory and writes each digit's run contiguously.  Bound by
// the pairs' traffic (12 B read, 12 B written an item and pass for composites over 32 bits, and 8 B for the
// counts), which for a few million items stays in L2.  No CTA waits for another, so a pass of few tiles costs
// three short launches instead of a chain of look-backs.  4,000,037 rows by two keys: 2.07 ms with 4-bit
// digits and one uncoalesced store per item, 0.33 ms with this form.
constexpr int kRThreads = 256, kRItems = 16, kRTile = kRThreads * kRItems, kRBuckets = 256, kRWarps = kRThreads / 32;
constexpr int kRMinBlocks = 2;  // 3 (with spills) measured the same
constexpr int kRKeys = 8;  // sort keys per launch of the key kernels

// double sort key -> unsigned order key: NULL (NaN) sorts first as -inf, -0 as 0; descending inverts
__device__ __forceinline__ u64 orderKey(double v, bool desc) {
  if (v != v) v = -__longlong_as_double(0x7ff0000000000000ll);
  if (v == 0.0) v = 0.0;
  u64 b = (u64)__double_as_longlong(v);
  b = (b >> 63) ? ~b : (b | 0x8000000000000000ull);
  return desc ? ~b : b;
}
struct SortKeys {
  const double* key[kRKeys];
  int desc[kRKeys];
  int n;
};
// bits[2k], bits[2k + 1] (0xff.. before): the AND of key k's order keys and of their complements
__global__ void kKeyBits(const __grid_constant__ SortKeys s, int64_t m, unsigned long long* bits) {
  __shared__ u64 red[2 * kRWarps];
  const double* key = s.key[blockIdx.y];
  const bool desc = s.desc[blockIdx.y] != 0;
  u64 a = ~0ull, z = ~0ull;
  WS_GRID_STRIDE(j, m) {
    const u64 k = orderKey(key[j], desc);
    a &= k, z &= ~k;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) a &= __shfl_xor_sync(0xffffffffu, a, o), z &= __shfl_xor_sync(0xffffffffu, z, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a, red[kRWarps + (threadIdx.x >> 5)] = z;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kRWarps; ++w) a &= red[w], z &= red[kRWarps + w];
    atomicAnd(bits + 2 * blockIdx.y, a);
    atomicAnd(bits + 2 * blockIdx.y + 1, z);
  }
}
struct PackSpec {
  SortKeys s;
  int lo[kRKeys], width[kRKeys], off[kRKeys];  // the key's varying bits and their place in the composite
};
// out[j] = composite of row perm[j] (row j without perm)
template <class K>
__global__ void kPackKeys(const __grid_constant__ PackSpec p, const int32_t* perm, int64_t m, K* out) {
  WS_GRID_STRIDE(j, m) {
    const int64_t r = perm ? perm[j] : j;
    u64 c = 0;
    for (int k = 0; k < p.s.n; ++k) {
      const u64 f = orderKey(p.s.key[k][r], p.s.desc[k] != 0) >> p.lo[k];
      c |= (p.width[k] < 64 ? f & ((1ull << p.width[k]) - 1) : f) << p.off[k];
    }
    out[j] = (K)c;
  }
}
__global__ void kIota(int32_t* p, int64_t m) {
  WS_GRID_STRIDE(j, m) p[j] = (int32_t)j;
}
// counts[v * ntiles + tile]: items of the tile with digit value v; total[v] += the same
// (shared atomics; a warp match per item, which serialises over the distinct digits, took 26 us instead of
// 13 us for 4,000,037 items)
template <class K>
__global__ void __launch_bounds__(kRThreads) kTileCount(const K* keys, int64_t m, int shift, int64_t ntiles,
                                                        unsigned* counts, unsigned* total) {
  __shared__ unsigned h[kRBuckets];
  const int t = threadIdx.x, lane = t & 31;
  h[t] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRTile;
  const int valid = (int)min((int64_t)kRTile, m - base);
#pragma unroll
  for (int i = 0; i < kRItems; ++i) {
    const int at = i * kRThreads + t;
    const int d = at < valid ? (int)(keys[base + at] >> shift) & (kRBuckets - 1) : -1;
    if (__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {  // nearly sorted or constant digits
      if (lane == 0 && d >= 0) atomicAdd(&h[d], 32u);
    } else if (d >= 0) {
      atomicAdd(&h[d], 1u);
    }
  }
  __syncthreads();
  const unsigned c = h[t];
  counts[(int64_t)t * ntiles + blockIdx.x] = c;
  if (c) atomicAdd(total + t, c);
}
// counts[v * ntiles ..] of digit value v = blockIdx.x -> first output position of each tile's items
__global__ void __launch_bounds__(kRThreads) kTileScan(unsigned* counts, int64_t ntiles, const unsigned* total) {
  __shared__ unsigned wsum[kRWarps], below;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned b = t < (int)blockIdx.x ? total[t] : 0;  // items of smaller digits
#pragma unroll
  for (int o = 16; o; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  if (lane == 0) wsum[warp] = b;
  __syncthreads();
  if (t == 0) {
    below = 0;
    for (int w = 0; w < kRWarps; ++w) below += wsum[w];
  }
  __syncthreads();
  unsigned run = below;
  unsigned* c = counts + (int64_t)blockIdx.x * ntiles;
  for (int64_t i0 = 0; i0 < ntiles; i0 += kRThreads) {
    const int64_t i = i0 + t;
    const unsigned v = i < ntiles ? c[i] : 0;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kRWarps; ++w) {
      if (w < warp) before += wsum[w];
      all += wsum[w];
    }
    if (i < ntiles) c[i] = run + before + incl - v;
    run += all;
    __syncthreads();
  }
}
// The lanes whose digit equals this lane's: one ballot per bit, independent from item to item (a warp match
// serialises over the distinct digits: the scatter took 42 us instead of 30 us for 4,000,037 items).
__device__ __forceinline__ unsigned sameDigit(int d) {
  unsigned same = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned v = __ballot_sync(0xffffffffu, (d >> b) & 1);
    same &= (d >> b) & 1 ? v : ~v;
  }
  return same;
}

// Stable scatter of one tile.  vals null: an item's row is its index; keysOut null (the last pass): only the
// rows are written.
template <class K>
__global__ void __launch_bounds__(kRThreads, kRMinBlocks) kTileScatter(const K* keys, const int32_t* vals, int64_t m, int shift,
                                                             int64_t ntiles, const unsigned* offs, K* keysOut,
                                                             int32_t* valsOut) {
  __shared__ K ex[kRTile];                  // the tile in digit order (keys, then rows)
  __shared__ int whist[kRWarps][kRBuckets];  // per warp: items of each digit, then the first position of its items
  __shared__ unsigned gbase[kRBuckets];     // output position of the tile's item at position p, digit d: gbase[d] + p
  __shared__ int wsum[kRWarps];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned lower = (1u << lane) - 1u;
  const int64_t base = (int64_t)blockIdx.x * kRTile;
  const int valid = (int)min((int64_t)kRTile, m - base);
  const int w0 = warp * (kRTile / kRWarps) + lane;  // a warp owns consecutive items, 32 at a time
  K k[kRItems];
#pragma unroll
  for (int i = 0; i < kRItems; ++i)  // items past the end have every bit set: they rank behind all others
    k[i] = w0 + i * 32 < valid ? keys[base + w0 + i * 32] : ~(K)0;
#pragma unroll
  for (int w = 0; w < kRWarps; ++w) whist[w][t] = 0;
  __syncthreads();
  int pos[kRItems];
#pragma unroll
  for (int i = 0; i < kRItems; ++i) {
    const int d = (int)(k[i] >> shift) & (kRBuckets - 1);
    const unsigned same = sameDigit(d);
    const int leader = __ffs(same) - 1;
    int old = 0;
    if (lane == leader) {
      old = whist[warp][d];
      whist[warp][d] = old + __popc(same);
    }
    pos[i] = __shfl_sync(0xffffffffu, old, leader) + __popc(same & lower);
    __syncwarp();
  }
  __syncthreads();
  {  // thread t: digit t's first position in the tile, then each warp's
    int run = 0, c[kRWarps];
#pragma unroll
    for (int w = 0; w < kRWarps; ++w) c[w] = run, run += whist[w][t];
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int start = incl - run;
    for (int w = 0; w < warp; ++w) start += wsum[w];
#pragma unroll
    for (int w = 0; w < kRWarps; ++w) whist[w][t] = start + c[w];
    gbase[t] = offs[(int64_t)t * ntiles + blockIdx.x] - (unsigned)start;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRItems; ++i) {
    pos[i] += whist[warp][(int)(k[i] >> shift) & (kRBuckets - 1)];
    ex[pos[i]] = k[i];
  }
  __syncthreads();
  unsigned dst[kRItems];
#pragma unroll
  for (int i = 0; i < kRItems; ++i) {
    const int p = i * kRThreads + t;
    const K key = ex[p];
    dst[i] = gbase[(int)(key >> shift) & (kRBuckets - 1)] + (unsigned)p;
    if (p < valid && keysOut) keysOut[dst[i]] = key;
  }
  __syncthreads();
  int* exv = (int*)ex;
#pragma unroll
  for (int i = 0; i < kRItems; ++i) {
    const int at = w0 + i * 32;
    exv[pos[i]] = at < valid ? (vals ? vals[base + at] : (int)(base + at)) : 0;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRItems; ++i) {
    const int p = i * kRThreads + t;
    if (p < valid) valsOut[dst[i]] = exv[p];
  }
}
__global__ void kMapRank(double* keys, const int32_t* rank, int64_t m) {
  WS_GRID_STRIDE(j, m) keys[j] = keys[j] != keys[j] ? -1.0 : (double)__ldg(rank + (int64_t)keys[j]);
}

// ---------------------------------------------------------------- distinct values, bitmaps, temp columns
// bit (v - base) of every non-NULL value v in [base, base + span) of an exact int64 array
__global__ void kDistinctBits(const i64* v, int64_t m, i64 base, i64 span, uint32_t* bits) {
  WS_GRID_STRIDE(j, m) {
    const i64 x = v[j];
    if (x == (i64)WS_NULL_I64) continue;
    const u64 k = (u64)x - (u64)base;
    if ((i64)k < 0 || (i64)k >= span || x < base) continue;
    const uint32_t bit = 1u << (k & 31);
    if (!(__ldg(bits + (k >> 5)) & bit)) atomicOr(bits + (k >> 5), bit);
  }
}
// bit (v - base) of the non-NULL values of an INT (out 0) / BIGINT (out 1) column; *nul: any NULL
__global__ void kBitsFromColumn(const void* col, int out, int64_t n, i64 base, i64 nbits, uint32_t* bits, int* nul) {
  int sawNull = 0;
  WS_GRID_STRIDE(i, n) {
    i64 v;
    if (out == 1) {
      v = ((const i64*)col)[i];
      if (v == (i64)WS_NULL_I64) {
        sawNull = 1;
        continue;
      }
    } else {
      const int x = ((const int*)col)[i];
      if (x == WS_NULL_I32) {
        sawNull = 1;
        continue;
      }
      v = x;
    }
    const i64 k = v - base;
    if (k >= 0 && k < nbits) atomicOr(bits + (k >> 5), 1u << (k & 31));
  }
  if (__any_sync(0xffffffffu, sawNull) && (threadIdx.x & 31) == 0) atomicOr(nul, 1);
}
// One temp-table column from compacted groups (column-major keys / accs); min / max of an integer
// output over the non-NULL groups (mnmx[0] / [1]).
__global__ void kTempColumn(const double* keys, const double* accs, int64_t g, const __grid_constant__ ws_temp_col_spec s,
                            void* out, long long* mnmx) {
  long long mn = LLONG_MAX, mx = LLONG_MIN;
  WS_GRID_STRIDE(r, g) {
    auto A = [&](int j) { return accs[(int64_t)j * g + r]; };
    auto bits = [](double d) { return (i64)__double_as_longlong(d); };
    bool nul = s.src == 1 && s.cnt >= 0 && A(s.cnt) == 0;
    bool isInt = false;
    i64 iv = 0;
    double dv = 0;
    if (s.src == 0) {
      const double k = keys[(int64_t)s.idx * g + r];
      if (s.key_int) {
        iv = bits(k);
        isInt = true;
        nul = iv == (i64)WS_NULL_I64 || iv == (i64)WS_NULL_I32;
      } else {
        dv = k;
        nul = k != k;
      }
    } else if (!nul) {
      switch (s.kind) {
        case 1: iv = bits(A(s.idx)); isInt = true; break;
        case 2: iv = (i64)((u64)bits(A(s.hi)) * 4294967296ull + (u64)bits(A(s.idx))); isInt = true; break;
        case 3: iv = (i64)A(s.idx); isInt = true; break;
        case 4: {
          const double sum = s.sum_bits ? (s.hi >= 0 ? (double)bits(A(s.hi)) * 4294967296.0 + (double)bits(A(s.idx))
                                                     : (double)bits(A(s.idx)))
                                        : A(s.idx);
          dv = sum / s.div / A(s.cnt);
          break;
        }
        default:
          dv = A(s.idx) / s.div;
          nul = dv != dv;
      }
    }
    if (s.mul != 1 && !nul) {
      dv = (isInt ? (double)iv : dv) * s.mul;
      isInt = false;
    }
    if (s.out == 2) {
      ((double*)out)[r] = nul ? __longlong_as_double(0x7ff8000000000000ll) : isInt ? (double)iv : dv;
      continue;
    }
    const long long v = nul ? 0 : isInt ? iv : llround(dv);
    if (!nul) mn = v < mn ? v : mn, mx = v > mx ? v : mx;
    if (s.out == 1) ((i64*)out)[r] = nul ? (i64)WS_NULL_I64 : v;
    else ((int32_t*)out)[r] = nul ? WS_NULL_I32 : (int32_t)v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const long long a = __shfl_xor_sync(0xffffffffu, mn, o), b = __shfl_xor_sync(0xffffffffu, mx, o);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
  if ((threadIdx.x & 31) == 0 && mn <= mx) {
    atomicMin(&mnmx[0], mn);
    atomicMax(&mnmx[1], mx);
  }
}
// host column of ptype -> double sort keys
__global__ void kToDouble(const void* src, int ptype, int64_t n, double* out) {
  WS_GRID_STRIDE(i, n) {
    out[i] = ptype == WS_PT_I32 ? (double)((const int*)src)[i]
             : ptype == WS_PT_I64 ? (double)((const i64*)src)[i] : ((const double*)src)[i];
  }
}

// The engine evaluates gpuDistinctInts' program exactly only when it is built of integer columns,
// integer literals, + - * and negation within a 16-deep stack (src/gpu.cu:826-865); any other program
// yields no values.
bool exactIntProgram(const ws_expr_env& env, ws_prog p) {
  int sp = 0;
  for (int i = 0; i < p.len; ++i) {
    const ws_instr in = env.code[p.start + i];
    switch (in.op) {
      case WS_OP_COL: {
        const int t = env.cols[in.arg].t;
        if (t == 2 || t == 5 || t == 6 || sp >= 16) return false;
        ++sp;
        break;
      }
      case WS_OP_CONST:
        if (!in.isInt || sp >= 16) return false;
        ++sp;
        break;
      case WS_OP_ADD: case WS_OP_SUB: case WS_OP_MUL:
        if (sp < 2) return false;
        --sp;
        break;
      case WS_OP_NEG:
        if (sp < 1) return false;
        break;
      default: return false;
    }
  }
  return sp == 1;
}

// Sorts perm (null: the rows in their own order) by the composite p of `total` bits, stably.
template <class K>
void sortComposite(const PackSpec& p, int total, int64_t m, DBuf<int32_t>& perm) {
  const int64_t ntiles = (m + kRTile - 1) / kRTile;
  const int passes = (total + 7) / 8;
  DBuf<K> k1(m), k2(passes > 1 ? m : 0);
  DBuf<int32_t> perm2(m);
  DBuf<unsigned> counts(kRBuckets * ntiles), totals((int64_t)kRBuckets * passes);
  WS_CK(cudaMemsetAsync(totals.p, 0, sizeof(unsigned) * kRBuckets * passes, stream()));
  WS_LAUNCH(kPackKeys<K>, gridFor(m), 256, 0, p, perm.p, m, k1.p);
  for (int d = 0; d < passes; ++d) {
    WS_LAUNCH(kTileCount<K>, (unsigned)ntiles, kRThreads, 0, k1.p, m, 8 * d, ntiles, counts.p, totals.p + kRBuckets * d);
    WS_LAUNCH(kTileScan, kRBuckets, kRThreads, 0, counts.p, ntiles, totals.p + kRBuckets * d);
    if (!perm2.p) perm2 = DBuf<int32_t>(m);
    WS_LAUNCH(kTileScatter<K>, (unsigned)ntiles, kRThreads, 0, k1.p, perm.p, m, 8 * d, ntiles, counts.p,
              d + 1 < passes ? k2.p : nullptr, perm2.p);
    std::swap(k1, k2);
    std::swap(perm, perm2);
  }
}

double kNullF64() {  // the engine's NULL double: the canonical quiet NaN
  const uint64_t b = 0x7ff8000000000000ull;
  double d;
  memcpy(&d, &b, 8);
  return d;
}

EvalSpec evalSpec(const ws_expr_env& env, int ncols, ws_prog prog, DBuf<uint8_t>& progBuf) {
  if (ncols < 0 || ncols > WS_MAX_COLS) throw Error("bad column count", WS_ERR_ARG);
  ws_agg_plan plan;
  memset(&plan, 0, sizeof plan);
  plan.hasWhere = 1;
  plan.where = prog;
  plan.naggs = 1;  // the hidden COUNT(*) slot only (no program): the layout needs one slot
  plan.ops[0] = WS_AGG_COUNT;
  TProgs* tp = new TProgs;
  try {
    buildTProgs(env, ncols, plan, true, *tp);
  } catch (...) {
    delete tp;
    throw;
  }
  EvalSpec s{};
  s.start = tp->where[0];
  s.len = tp->where[1];
  s.isInt = typeProg(env, prog, ncols).isInt() ? 1 : 0;
  const ws_instr& in0 = env.code[prog.start];
  s.single = prog.len == 1 && in0.op == WS_OP_COL && env.cols[in0.arg].t != 2 ? 1 : 0;
  s.col = in0.arg;
  s.simple = 1;
  for (int pc = s.start, depth = 0; pc < s.start + s.len && s.simple; ++pc) {
    const TInstr& in = tp->code[pc];
    switch (in.op) {
      case WS_OP_COL:
        s.simple = in.arg < ncols && env.cols[in.arg].t <= 4 && env.cols[in.arg].enc == 0 && ++depth <= kSimpleDepth;
        break;
      case WS_OP_CONST: s.simple = ++depth <= kSimpleDepth; break;
      case WS_OP_ADD: case WS_OP_SUB: case WS_OP_MUL: case WS_OP_DIV: s.simple = --depth >= 1; break;
      case WS_OP_NEG: s.simple = depth >= 1; break;
      default: s.simple = 0;
    }
  }
  const size_t bytes = sizeof(TInstr) * (size_t)std::max(s.start + s.len, 1);
  progBuf = DBuf<uint8_t>((int64_t)bytes);
  uint8_t* st = pinnedStage(bytes);
  memcpy(st, tp->code, bytes);
  delete tp;
  h2dAsync(progBuf.p, st, bytes);
  stageCopied();
  s.code = (const TInstr*)progBuf.p;
  return s;
}

const ws_col_view* uploadCols(const ws_expr_env& env, int ncols, DBuf<uint8_t>& buf) {
  if (ncols < 0 || ncols > WS_MAX_COLS) throw Error("bad column count", WS_ERR_ARG);
  const size_t bytes = sizeof(ws_col_view) * (size_t)std::max(ncols, 1);
  buf = DBuf<uint8_t>((int64_t)bytes);
  uint8_t* st = pinnedStage(bytes);
  memcpy(st, env.cols, sizeof(ws_col_view) * (size_t)ncols);
  h2dAsync(buf.p, st, bytes);
  stageCopied();
  return (const ws_col_view*)buf.p;
}

}  // namespace
}  // namespace ws

using namespace ws;

extern "C" {

int ws_key_bitmap(ws_col_view key, int64_t n, int64_t lo, int64_t nbits, uint32_t* bits) {
  return guardedCall([&] {
    if (nbits < 0) throw Error("negative bitmap size", WS_ERR_ARG);
    WS_CK(cudaMemsetAsync(bits, 0, (size_t)((nbits + 31) / 32) * 4, stream()));
    if (n > 0 && nbits > 0) WS_LAUNCH(kKeyBitmap, gridFor(n), 256, 0, key, n, (long long)lo, nbits, bits);
  });
}

int ws_set_bits(uint32_t* bits, const int32_t* idx, int64_t m) {
  return guardedCall([&] {
    if (m > 0) WS_LAUNCH(kSetBits, gridFor(m), 256, 0, bits, idx, m);
  });
}

int ws_remap_codes(const int32_t* in, int64_t n, const int32_t* map, int64_t map_n, int32_t* out) {
  return guardedCall([&] {
    if (n > 0) WS_LAUNCH(kRemapCodes, gridFor(n), 256, 0, in, n, map, map_n, out);
  });
}

int ws_bits_to_double(const double* src, int64_t n, double* dst) {
  return guardedCall([&] {
    if (n > 0) WS_LAUNCH(kBitsToDouble, gridFor(n), 256, 0, src, n, dst);
  });
}

int ws_gather_null(const void* src, int ptype, const int32_t* idx, int64_t m, void* dst) {
  return guardedCall([&] {
    if (m <= 0) return;
    if (ptype == WS_PT_I32)
      WS_LAUNCH(kGatherNull<int32_t>, gridFor(m), 256, 0, (const int32_t*)src, idx, m, (int32_t*)dst, (int32_t)WS_NULL_I32);
    else if (ptype == WS_PT_I64)
      WS_LAUNCH(kGatherNull<long long>, gridFor(m), 256, 0, (const long long*)src, idx, m, (long long*)dst,
                (long long)WS_NULL_I64);
    else if (ptype == WS_PT_F64)
      WS_LAUNCH(kGatherNull<double>, gridFor(m), 256, 0, (const double*)src, idx, m, (double*)dst, kNullF64());
    else
      throw Error("gather: unsupported physical type", WS_ERR_ARG);
  });
}

int ws_gather_bytes(const void* src, int esize, const int32_t* idx, int64_t m, void* dst, int nulls) {
  return guardedCall([&] {
    if (esize <= 0 || esize % 4) throw Error("gather: element size must be a multiple of 4 bytes", WS_ERR_ARG);
    if (m > 0) WS_LAUNCH(kGatherWords, gridFor(m * (esize / 4)), 256, 0, (const uint32_t*)src, esize / 4, idx, m,
                         (uint32_t*)dst, nulls);
  });
}

int ws_gather_enc(ws_col_view v, int ptype, const int32_t* idx, int64_t m, void* dst) {
  return guardedCall([&] {
    if (m <= 0) return;
    ws_col_view w = v;
    w.t = ptype == WS_PT_I32 ? 3 : ptype == WS_PT_I64 ? 4 : 2;  // NULL sentinels kept as stored
    WS_LAUNCH(kGatherEnc, gridFor(m), 256, 0, w, ptype, idx, m, dst);
  });
}

int ws_eval_at(const ws_expr_env* env, int ncols, ws_prog prog, const int32_t* idx, int64_t m, double* out) {
  return guardedCall([&] {
    if (m <= 0) return;
    DBuf<uint8_t> pb, cb;
    const EvalSpec s = evalSpec(*env, ncols, prog, pb);
    const ws_col_view* cv = uploadCols(*env, ncols, cb);
    if (s.simple)
      WS_LAUNCH(kEvalSimple<false>, gridFor(m, 256 * kSimpleRows), 256, 0, s, cv, envK(*env), idx, m, (void*)out);
    else
      WS_LAUNCH(kEvalAt, gridFor(m), 256, 0, s, cv, envK(*env), idx, m, out);
  });
}

int ws_eval_at_int(const ws_expr_env* env, int ncols, ws_prog prog, const int32_t* idx, int64_t m, int64_t* out) {
  return guardedCall([&] {
    if (m <= 0) return;
    DBuf<uint8_t> pb, cb;
    const EvalSpec s = evalSpec(*env, ncols, prog, pb);
    const ws_col_view* cv = uploadCols(*env, ncols, cb);
    if (s.simple && !s.single)
      WS_LAUNCH(kEvalSimple<true>, gridFor(m, 256 * kSimpleRows), 256, 0, s, cv, envK(*env), idx, m, (void*)out);
    else
      WS_LAUNCH(kEvalAtInt, gridFor(m), 256, 0, s, cv, envK(*env), idx, m, out);
  });
}

int ws_sort_perm(const double* const* keys, const int* desc, int nkeys, int64_t m, int32_t** out_perm) {
  return guardedCall([&] {
    *out_perm = nullptr;
    if (m < 0 || m > INT32_MAX) throw Error("sort: row count out of range", WS_ERR_ARG);
    DBuf<int32_t> perm;  // empty: the rows in their own order
    if (m > 0 && nkeys > 0) {
      // the bits of each key that differ among the rows
      DBuf<unsigned long long> bits(2 * (int64_t)nkeys);
      WS_CK(cudaMemsetAsync(bits.p, 0xff, 16 * (size_t)nkeys, stream()));
      for (int k0 = 0; k0 < nkeys; k0 += kRKeys) {
        SortKeys s{};
        s.n = std::min(kRKeys, nkeys - k0);
        for (int k = 0; k < s.n; ++k) s.key[k] = keys[k0 + k], s.desc[k] = desc[k0 + k];
        WS_LAUNCH(kKeyBits, dim3(gridFor(m, 256, 4), s.n), kRThreads, 0, s, m, bits.p + 2 * k0);
      }
      std::vector<unsigned long long> h(2 * (size_t)nkeys);
      d2hSync(h.data(), bits.p, 8 * h.size());
      for (int key = nkeys - 1; key >= 0;) {  // composites, least significant keys first
        PackSpec p{};
        int total = 0;
        for (; key >= 0 && p.s.n < kRKeys; --key) {
          const u64 vary = ~(h[2 * (size_t)key] | h[2 * (size_t)key + 1]);
          if (!vary) continue;  // every row has the same value
          const int lo = __builtin_ctzll(vary), width = 64 - __builtin_clzll(vary) - lo;
          if (total + width > 64) break;
          p.s.key[p.s.n] = keys[key], p.s.desc[p.s.n] = desc[key];
          p.lo[p.s.n] = lo, p.width[p.s.n] = width, p.off[p.s.n] = total;
          ++p.s.n;
          total += width;
        }
        if (!total) continue;
        if (total <= 32) sortComposite<uint32_t>(p, total, m, perm);
        else sortComposite<u64>(p, total, m, perm);
      }
    }
    if (!perm.p) {
      perm = DBuf<int32_t>(std::max<int64_t>(m, 1));
      if (m) WS_LAUNCH(kIota, gridFor(m), 256, 0, perm.p, m);
    }
    *out_perm = perm.release();
  });
}

int ws_distinct_ints(const ws_expr_env* env, int ncols, ws_prog prog, const int32_t* idx, int64_t m, int64_t base,
                     int64_t span, int64_t* out, int64_t max_out, int64_t* count) {
  return guardedCall([&] {
    *count = 0;
    if (m <= 0 || span <= 0) return;
    if (prog.start < 0 || prog.len <= 0 || prog.start + prog.len > WS_MAX_CODE)
      throw Error("ws_distinct_ints: program outside the code array", WS_ERR_ARG);
    if (!exactIntProgram(*env, prog)) return;
    if (span > ((int64_t)1 << 40)) throw Error("ws_distinct_ints: span too large for a bitmap", WS_ERR_ARG);
    DBuf<uint8_t> pb, cb;
    const EvalSpec s = evalSpec(*env, ncols, prog, pb);
    const ws_col_view* cv = uploadCols(*env, ncols, cb);
    DBuf<i64> vals(m);
    WS_LAUNCH(kEvalAtInt, gridFor(m), 256, 0, s, cv, envK(*env), idx, m, (int64_t*)vals.p);
    const int64_t words = (span + 31) / 32;
    DBuf<uint32_t> bits(words);
    WS_CK(cudaMemsetAsync(bits.p, 0, (size_t)words * 4, stream()));
    WS_LAUNCH(kDistinctBits, gridFor(m), 256, 0, vals.p, m, base, span, bits.p);
    std::vector<uint32_t> h((size_t)words);
    d2hLarge(h.data(), bits.p, (size_t)words * 4);
    int64_t c = 0;
    for (int64_t w = 0; w < words; ++w)
      for (uint32_t b = h[(size_t)w]; b; b &= b - 1) {
        if (c < max_out && out) out[c] = base + w * 32 + __builtin_ctz(b);
        ++c;
      }
    *count = c;
    if (c > max_out) throw Error("ws_distinct_ints: more distinct values than out holds", WS_ERR_SIZE);
  });
}

int ws_bits_from_column(const void* col, int out, int64_t n, int64_t base, int64_t nbits, uint32_t** bits,
                        int* saw_null) {
  return guardedCall([&] {
    ensureInit();
    *bits = nullptr;
    *saw_null = 0;
    if (nbits < 0 || n < 0 || (out != 0 && out != 1)) throw Error("ws_bits_from_column: bad arguments", WS_ERR_ARG);
    const size_t bytes = std::max<size_t>(4, (size_t)((nbits + 31) / 32) * 4);
    uint32_t* b = nullptr;
    WS_CK(cudaMalloc(&b, bytes));
    try {
      WS_CK(cudaMemsetAsync(b, 0, bytes, stream()));
      DBuf<int> nul(1);
      WS_CK(cudaMemsetAsync(nul.p, 0, 4, stream()));
      if (n > 0) WS_LAUNCH(kBitsFromColumn, gridFor(n), 256, 0, col, out, n, base, nbits, b, nul.p);
      int h = 0;
      d2hSync(&h, nul.p, 4);
      *saw_null = h != 0;
    } catch (...) {
      cudaStreamSynchronize(stream());
      cudaFree(b);
      throw;
    }
    *bits = b;
  });
}

int ws_temp_column(const double* keys, int nk, const double* accs, int na, int64_t g, const ws_temp_col_spec* s,
                   void** col, double* mn, double* mx) {
  return guardedCall([&] {
    ensureInit();
    *col = nullptr;
    if (g < 0 || s->out > 2 || (s->src == 0 && (s->idx < 0 || s->idx >= nk)) ||
        (s->src == 1 && (s->idx < 0 || s->idx >= na || s->hi >= na || s->cnt >= na)))
      throw Error("ws_temp_column: spec outside the groups' keys / slots", WS_ERR_ARG);
    const size_t w = s->out == 0 ? 4 : 8;
    void* o = nullptr;
    WS_CK(cudaMalloc(&o, std::max<size_t>(1, (size_t)g * w)));
    long long h[2] = {LLONG_MAX, LLONG_MIN};
    try {
      DBuf<long long> mm(2);
      uint8_t* st = pinnedStage(sizeof h);
      memcpy(st, h, sizeof h);
      h2dAsync(mm.p, st, sizeof h);
      stageCopied();
      if (g > 0) WS_LAUNCH(kTempColumn, gridFor(g), 256, 0, keys, accs, g, *s, o, mm.p);
      d2hSync(h, mm.p, sizeof h);
    } catch (...) {
      cudaStreamSynchronize(stream());
      cudaFree(o);
      throw;
    }
    *mn = s->out == 2 || h[0] > h[1] ? -INFINITY : (double)h[0];
    *mx = s->out == 2 || h[0] > h[1] ? INFINITY : (double)h[1];
    *col = o;
  });
}

int ws_sort_perm_host(const void* host_col, int ptype, int64_t n, int32_t* perm) {
  return guardedCall([&] {
    if (n <= 0) return;
    if (ptype != WS_PT_I32 && ptype != WS_PT_I64 && ptype != WS_PT_F64)
      throw Error("ws_sort_perm_host: ptype must be I32, I64 or F64", WS_ERR_ARG);
    const size_t esz = ptype == WS_PT_I32 ? 4 : 8;
    DBuf<uint8_t> raw((int64_t)(n * esz));
    WS_CK(cudaMemcpyAsync(raw.p, host_col, (size_t)n * esz, cudaMemcpyHostToDevice, stream()));
    DBuf<double> k(n);
    WS_LAUNCH(kToDouble, gridFor(n), 256, 0, raw.p, ptype, n, k.p);
    const double* keys[1] = {k.p};
    const int desc[1] = {0};
    int32_t* p = nullptr;
    const int rc = ws_sort_perm(keys, desc, 1, n, &p);
    if (rc != WS_OK) throw Error(ws_last_error(), rc);
    DBuf<int32_t> pp;
    pp.p = p, pp.n = n;
    d2hLarge(perm, p, (size_t)n * 4);
  });
}

int ws_map_rank(double* keys, const int32_t* rank, int64_t m) {
  return guardedCall([&] {
    if (m > 0) WS_LAUNCH(kMapRank, gridFor(m), 256, 0, keys, rank, m);
  });
}

}  // extern "C"
