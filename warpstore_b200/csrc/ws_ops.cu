// Operators of libwarpstore_b200: aggregation (GpuAggregator), selection, gathers and hash joins
// (reference: src/gpu.cu:393-800, :1089-1316).  Scan kernels come from ws_kern.cuh, instantiated here
// with the interpreter and per plan by the code generator; the helper kernels below are plain CUDA.
#include <cstring>

#include "ws_internal.h"
#include "ws_shape.h"

namespace ws {

// Interpreter instantiations of every scan kernel (prefix wsi), one translation unit per group.
void interpSyms_agg(const void** s);
void interpSyms_priv(const void** s);
void interpSyms_hash(const void** s);
void interpSyms_select(const void** s);

const KernelSet& interpKernels() {
  static KernelSet ks = [] {
    KernelSet k;
    const void* syms[K_COUNT_] = {};
    interpSyms_agg(syms);
    interpSyms_priv(syms);
    interpSyms_hash(syms);
    interpSyms_select(syms);
    for (int i = 0; i < K_COUNT_; ++i) {
      cudaFunction_t f;
      if (!syms[i]) continue;  // staged kernels: compiled plans only
      WS_CK(cudaGetFuncBySymbol(&f, syms[i]));
      k.fn[i] = (CUfunction)f;
    }
    k.interp = true;
    return k;
  }();
  return ks;
}

namespace {

int gridFor(int64_t n, int block = 256, int perSm = 8) {
  int64_t g = (n + block - 1) / block;
  const int64_t cap = (int64_t)smCount() * perSm;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}
#define WS_LAUNCH(kernel, grid, block, smem, ...)                 \
  do {                                                            \
    kernel<<<(grid), (block), (smem), stream()>>>(__VA_ARGS__);   \
    WS_CK(cudaGetLastError());                                    \
    countLaunch();                                                \
  } while (0)

// ---------------------------------------------------------------- helper kernels
}  // namespace
// Identity values of one accumulator row (by value as a kernel parameter).
struct RowTemplate {
  u64 w[kMaxRowWords];
};
namespace {
// Result rows to their identities (hash rows empty: key word kEmpty, the extra row's claim flag 0) and the
// control words to 0.
struct FillSpec {
  u64* rows;
  int64_t words;       // rows x rw
  int64_t emptyWords;  // hash rows x rw: their word 0 is kEmpty, every other row's 0
  int rw;
  u64* ctl;            // kCtlWords words
  RowTemplate t;
};
// count u64 | ... | err int x3, occTicket u32 | ticket u32, pad: the flags that scans read are 128 bytes from the count
// that they add to, so that those reads do not queue behind its atomics.
constexpr int kCtlWords = 24, kCtlFlags = 128;
// Thread `tid` of `nthreads` (at least rw).  The threads step by a multiple of the row width, so each stays
// on one word of the rows (a constant) and a warp's stores are consecutive: 2^24 rows of 32 B take 79 us,
// against 310 us with a row per thread (and 345 us with a loop of its own for the key words).
__device__ __forceinline__ void fillRows(const FillSpec& f, int64_t tid, int64_t nthreads) {
  if (tid < kCtlWords) f.ctl[tid] = 0;
  const int64_t step = nthreads / f.rw * f.rw;
  if (tid >= step) return;
  const int j = (int)(tid % f.rw);
  const u64 v = j == 0 ? kEmpty : f.t.w[j];
  const int64_t plain = j == 0 ? f.emptyWords : f.words;  // one loop for every lane: whole sectors per store
  for (int64_t i = tid; i < f.words; i += step) f.rows[i] = i < plain ? v : 0ull;
}
__global__ void kFillRows(const __grid_constant__ FillSpec f) {
  fillRows(f, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}
__global__ void kFillRowsMany(const FillSpec* fs) {  // spec blockIdx.y
  fillRows(fs[blockIdx.y], blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// ---- result delivery.  Occupied result rows (hash rows [0, cap) by their key word, the extra row (cap) by
// its claim flag, dense rows by slot 0 (COUNT(*)) being non-zero) become groups in ascending row order:
// keys in the engine's format, accs in its slot format, exact words.
//
// A result table of at most kSmallRows rows is delivered by one CTA in one launch (kDeliver: occupancy,
// ranks, groups and the status), whole queries' worth of them by one launch of a CTA each (kDeliverMany); a
// larger one by two (kOccCount, whose last CTA also scans the chunks' counts; kEmitChunks).  The separate
// count, scan, status, index, emit and convert launches they replace cost a small query 13 to 25 us of
// launches and each read the table again.  The groups' row indices are listed in shared memory and the
// output is written by consecutive words, so that stores to pinned host memory go out as whole lines.
struct ResultSpec {
  const u64* rows;
  int64_t nrows, cap;  // cap: index of the extra hash row
  const int* err;
  const double* tkeys;
  int rw, mode;        // mode 0 no keys, 1 dense, 2 hash
  int cnt0;            // word of slot 0
  int nk, na;
  uint8_t kind[WS_MAX_AGGS];     // kind of the slot whose words the slot shows (its partner's for SK_NONE)
  uint8_t derived[WS_MAX_AGGS];  // SK_NONE: the high half of a split BIGINT SUM
  uint8_t aggBits[WS_MAX_AGGS], aggPart[WS_MAX_AGGS];
  int16_t woff[WS_MAX_AGGS];
  uint8_t keyInt[WS_MAX_KEYS];
  int64_t kmin[WS_MAX_KEYS], range[WS_MAX_KEYS], stride[WS_MAX_KEYS];
};
// Where groups [first, first + limit) go (null: not wanted): row-major from output row 0, or column-major
// in columns of colRows.
struct OutSpec {
  double* keys;
  double* accs;
  long long* exact;
  int64_t first, limit, colRows;
};
constexpr int64_t kSmallRows = 4097;
constexpr int kDeliverThreads = 1024, kDeliverIters = (int)((kSmallRows + kDeliverThreads - 1) / kDeliverThreads);
constexpr int kOccChunk = 2048, kOccThreads = 256;

__device__ __forceinline__ bool occupied(const ResultSpec& s, int64_t i) {
  const u64* r = s.rows + i * s.rw;
  if (s.mode == 0) return true;  // no GROUP BY: the one result row
  if (s.mode == 1) return r[s.cnt0] != 0;
  if (i == s.cap) return r[0] != 0;
  return r[0] != kEmpty;
}
__device__ __forceinline__ double keyOut(const ResultSpec& s, int64_t i, int k) {
  if (s.mode == 1) {
    const long long v = s.kmin[k] + (i / s.stride[k]) % s.range[k];
    return s.keyInt[k] ? __longlong_as_double(v) : (double)v;
  }
  if (s.nk == 1) return __longlong_as_double(i == s.cap ? (long long)kEmpty : (long long)s.rows[i * s.rw]);
  return s.tkeys[i * s.nk + k];
}
// Exact words of slot a of result row i: (lo, hi) of an integer SUM, (value, 0) otherwise.
__device__ __forceinline__ void exactOut(const ResultSpec& s, int64_t i, int a, long long& w0, long long& w1) {
  const u64* r = s.rows + i * s.rw + s.woff[a];
  const uint8_t k = s.kind[a];
  w0 = (long long)r[0];
  w1 = k == SK_ISUM ? (long long)r[1] : 0;
  if (k == SK_DMIN || k == SK_DMAX) w0 = __double_as_longlong(dunord(w0));
}
// The engine's double slot format of those words.
__device__ __forceinline__ double accOut(const ResultSpec& s, int a, long long w0, long long w1) {
  const uint8_t k = s.kind[a];
  if (k == SK_COUNT) return (double)w0;
  if (k == SK_ISUM) {
    const __int128 T = (__int128)(((unsigned __int128)(unsigned long long)w1 << 64) | (unsigned long long)w0);
    if (s.nk == 0) return __longlong_as_double(w0);
    if (s.aggBits[a])
      return __longlong_as_double(s.aggPart[a] == 2 || s.derived[a] ? (long long)(T >> 32)
                                  : s.aggPart[a] == 1 ? (long long)(T & 0xffffffff) : w0);
    return (double)T;
  }
  if (k == SK_IMIN || k == SK_IMAX) {
    if (s.nk == 0 || s.aggBits[a]) return __longlong_as_double(w0);
    if (k == SK_IMIN && w0 == 0x7fffffffffffffffll) return __longlong_as_double(0x7ff0000000000000ll);
    if (k == SK_IMAX && w0 == (long long)0x8000000000000000ull) return __longlong_as_double((long long)0xfff0000000000000ull);
    return (double)w0;
  }
  return __longlong_as_double(w0);
}
// Groups p0 .. p0 + n of the result, whose rows are base + list[0 .. n): those within [first, first + limit)
// to the outputs (all threads of the CTA).
__device__ __forceinline__ void emitGroups(const ResultSpec& s, const OutSpec& o, int64_t base, const int* list, int n,
                                           int64_t p0) {
  const int lo = (int)min((int64_t)n, max((int64_t)0, o.first - p0));
  const int hi = (int)max((int64_t)lo, min((int64_t)n, o.first + o.limit - p0));
  const int m = hi - lo;
  if (m <= 0) return;
  list += lo;
  const int64_t at = p0 + lo - o.first;  // output row of the first
  if (o.keys)
    for (int t = threadIdx.x; t < m * s.nk; t += blockDim.x) {
      const int p = o.colRows ? t % m : t / s.nk, k = o.colRows ? t / m : t % s.nk;
      o.keys[o.colRows ? k * o.colRows + at + p : (at + p) * s.nk + k] = keyOut(s, base + list[p], k);
    }
  if (o.accs || o.exact)
    for (int t = threadIdx.x; t < m * s.na; t += blockDim.x) {
      const int p = o.colRows ? t % m : t / s.na, a = o.colRows ? t / m : t % s.na;
      long long w0, w1;
      exactOut(s, base + list[p], a, w0, w1);
      const int64_t e = (at + p) * s.na + a;
      if (o.accs) o.accs[o.colRows ? a * o.colRows + at + p : e] = accOut(s, a, w0, w1);
      if (o.exact) o.exact[2 * e] = w0, o.exact[2 * e + 1] = w1;
    }
}
// Lists the occupied rows of [base, base + rows) in ascending order; returns their number (every thread).
// rows <= ITERS * blockDim.x, blockDim.x = 32 * WARPS; cnt: [ITERS * WARPS] words of shared memory.
template <int ITERS, int WARPS>
__device__ __forceinline__ int listOccupied(const ResultSpec& s, int64_t base, int rows, int* list, int* cnt, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned m[ITERS];
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int r = it * WARPS * 32 + threadIdx.x;
    m[it] = __ballot_sync(0xffffffffu, r < rows && occupied(s, base + r));
    if (lane == 0) cnt[it * WARPS + warp] = __popc(m[it]);
  }
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the ITERS * WARPS counts, E of them per lane
    constexpr int N = ITERS * WARPS, E = (N + 31) / 32;
    int c[E], sum = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int at = lane * E + e;
      c[e] = at < N ? cnt[at] : 0;
      sum += c[e];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    int run = incl - sum;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int at = lane * E + e;
      if (at < N) cnt[at] = run;
      run += c[e];
    }
    if (lane == 31) *total = incl;
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < ITERS; ++it)
    if ((m[it] >> lane) & 1u)
      list[cnt[it * WARPS + warp] + __popc(m[it] & ((1u << lane) - 1u))] = it * WARPS * 32 + threadIdx.x;
  __syncthreads();
  return *total;
}
__device__ __forceinline__ void writeStatus(const ResultSpec& s, int64_t groups, ws_fetch_status* st) {
  st->groups = groups;
  st->overflow = s.mode == 2 && s.err[1] ? 1 : 0;
  st->error = s.err[0] ? WS_ERR_RANGE : s.err[2] ? WS_ERR_INTERNAL : 0;
}

// Delivers a result of at most kSmallRows rows.  Nothing but the status is written when the run raised a flag
// (dense key out of range, staged-copy timeout; hash overflow unless evenOverflowed): the caller reads the
// status and reruns.
struct DeliverSpec {
  ResultSpec r;
  OutSpec o;
  ws_fetch_status* st;  // null: not wanted
  int evenOverflowed;
};
__device__ __forceinline__ void deliver(const DeliverSpec& d) {
  __shared__ int list[kDeliverIters * kDeliverThreads], cnt[kDeliverIters * 32], total;
  const int g = listOccupied<kDeliverIters, 32>(d.r, 0, (int)d.r.nrows, list, cnt, &total);
  if (threadIdx.x == 0 && d.st) writeStatus(d.r, g, d.st);
  if (d.r.err[0] || d.r.err[2] || (d.r.mode == 2 && d.r.err[1] && !d.evenOverflowed)) return;
  emitGroups(d.r, d.o, 0, list, g, 0);
}
__global__ void __launch_bounds__(kDeliverThreads) kDeliver(const __grid_constant__ DeliverSpec d) { deliver(d); }
__global__ void __launch_bounds__(kDeliverThreads) kDeliverMany(const DeliverSpec* ds) { deliver(ds[blockIdx.x]); }

// Groups of each chunk of kOccChunk result rows; the last CTA turns the counts into offsets (offs[nchunks]:
// the total) and writes the status (pinned host memory).  *ticket is 0 before and after.
__global__ void __launch_bounds__(kOccThreads) kOccCount(const __grid_constant__ ResultSpec s, int64_t* offs,
                                                         int64_t nchunks, unsigned* ticket, ws_fetch_status* st) {
  __shared__ int64_t wsum[kOccThreads / 32];
  __shared__ bool amLast;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t c0 = (int64_t)blockIdx.x * kOccChunk;
  int c = 0;
#pragma unroll
  for (int it = 0; it < kOccChunk / kOccThreads; ++it) {
    const int64_t i = c0 + it * kOccThreads + t;
    c += i < s.nrows && occupied(s, i);
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) wsum[warp] = c;
  __syncthreads();
  if (t == 0) {
    int64_t sum = 0;
    for (int w = 0; w < kOccThreads / 32; ++w) sum += wsum[w];
    offs[blockIdx.x] = sum;
    __threadfence();
    amLast = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!amLast) return;
  __threadfence();
  constexpr int E = 8;  // counts per thread and step
  int64_t run = 0;
  for (int64_t b = 0; b < nchunks; b += kOccThreads * E) {
    int64_t v[E], sum = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int64_t i = b + t * E + e;
      v[e] = i < nchunks ? __ldcg((const long long*)offs + i) : 0;
      sum += v[e];
    }
    int64_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int64_t before = 0, all = 0;
    for (int w = 0; w < kOccThreads / 32; ++w) {
      if (w < warp) before += wsum[w];
      all += wsum[w];
    }
    int64_t at = run + before + incl - sum;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int64_t i = b + t * E + e;
      if (i < nchunks) offs[i] = at;
      at += v[e];
    }
    run += all;
  }
  if (t == 0) {
    offs[nchunks] = run;
    *ticket = 0;
    writeStatus(s, run, st);
  }
}
// Groups of chunk blockIdx.x (the groups from offs[chunk] on) to the outputs; nothing when the run raised a
// flag (as kDeliver).
__global__ void __launch_bounds__(kOccThreads) kEmitChunks(const __grid_constant__ ResultSpec s,
                                                           const __grid_constant__ OutSpec o, const int64_t* offs,
                                                           int evenOverflowed) {
  constexpr int kIters = kOccChunk / kOccThreads, kWarps = kOccThreads / 32;
  __shared__ int list[kOccChunk], cnt[kIters * kWarps], total;
  if (s.err[0] || s.err[2] || (s.mode == 2 && s.err[1] && !evenOverflowed)) return;
  const int64_t p0 = offs[blockIdx.x], p1 = offs[blockIdx.x + 1];
  if (p0 == p1 || p1 <= o.first || p0 >= o.first + o.limit) return;  // none of this chunk's groups
  const int64_t base = (int64_t)blockIdx.x * kOccChunk;
  const int n = listOccupied<kIters, kWarps>(s, base, (int)min((int64_t)kOccChunk, s.nrows - base), list, cnt, &total);
  emitGroups(s, o, base, list, n, p0);
}
// The status alone (offsets known from an earlier range of the same run).
__global__ void kFetchStatus(const __grid_constant__ ResultSpec s, const int64_t* total, ws_fetch_status* st) {
  writeStatus(s, *total, st);
}

}  // namespace

// ---------------------------------------------------------------- batch descriptor
// Device copy of the batches of one launch: [cols nb*ncols][n nb][del nb][tileStart nb+1][rowStart nb+1]
// followed, for interpreted plans, by the typed programs and slot tables.
struct BatchDesc {
  DBuf<uint8_t> buf;
  int64_t ntiles = 0, rows = 0;
  const ws_col_view* cols = nullptr;
  const int64_t* n = nullptr;
  const uint32_t* const* del = nullptr;
  const int64_t* tileStart = nullptr;
  const int64_t* rowStart = nullptr;
  const TProgs* progs = nullptr;
  const uint8_t* kinds = nullptr;
  const int* woff = nullptr;
  const int* fwoff = nullptr;
  const uint8_t* aggNull = nullptr;
  const uint8_t* keyInt = nullptr;
};

static BatchDesc uploadBatches(int nb, int ncols, const int64_t* bn, const uint32_t* const* bdel, const ws_col_view* bcols,
                               const TProgs* progs, const SlotLayout* lay, const ws_agg_plan* plan) {
  BatchDesc d;
  const size_t colBytes = (size_t)nb * ncols * sizeof(ws_col_view);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = (off + 15) & ~(size_t)15;
    off = o + bytes;
    return o;
  };
  const size_t oCols = take(colBytes), oN = take(8 * nb), oDel = take(8 * nb), oTile = take(8 * (nb + 1)),
               oRow = take(8 * (nb + 1));
  size_t oProg = 0, oKinds = 0, oWoff = 0, oFwoff = 0, oNull = 0, oKeyInt = 0;
  if (progs) {
    oProg = take(sizeof(TProgs));
    oKinds = take(WS_MAX_AGGS);
    oWoff = take(4 * WS_MAX_AGGS);
    oFwoff = take(4 * WS_MAX_AGGS);
    oNull = take(WS_MAX_AGGS);
    oKeyInt = take(WS_MAX_KEYS);
  }
  uint8_t* st = pinnedStage(off);
  memcpy(st + oCols, bcols, colBytes);
  int64_t* n = (int64_t*)(st + oN);
  const uint32_t** del = (const uint32_t**)(st + oDel);
  int64_t* ts = (int64_t*)(st + oTile);
  int64_t* rs = (int64_t*)(st + oRow);
  ts[0] = 0;
  rs[0] = 0;
  for (int b = 0; b < nb; ++b) {
    n[b] = bn[b];
    del[b] = bdel ? bdel[b] : nullptr;
    ts[b + 1] = ts[b] + (bn[b] + kTile - 1) / kTile;
    rs[b + 1] = rs[b] + bn[b];
  }
  d.ntiles = ts[nb];
  d.rows = rs[nb];
  if (progs) {
    memcpy(st + oProg, progs, sizeof(TProgs));
    memcpy(st + oKinds, lay->kind, WS_MAX_AGGS);
    memcpy(st + oWoff, lay->woff, 4 * WS_MAX_AGGS);
    memcpy(st + oFwoff, lay->fwoff, 4 * WS_MAX_AGGS);
    memcpy(st + oNull, plan->aggNull, WS_MAX_AGGS);
    memcpy(st + oKeyInt, plan->keyInt, WS_MAX_KEYS);
  }
  d.buf = DBuf<uint8_t>((int64_t)off);
  h2dAsync(d.buf.p, st, off);
  stageCopied();
  uint8_t* p = d.buf.p;
  d.cols = (const ws_col_view*)(p + oCols);
  d.n = (const int64_t*)(p + oN);
  d.del = (const uint32_t* const*)(p + oDel);
  d.tileStart = (const int64_t*)(p + oTile);
  d.rowStart = (const int64_t*)(p + oRow);
  if (progs) {
    d.progs = (const TProgs*)(p + oProg);
    d.kinds = p + oKinds;
    d.woff = (const int*)(p + oWoff);
    d.fwoff = (const int*)(p + oFwoff);
    d.aggNull = p + oNull;
    d.keyInt = p + oKeyInt;
  }
  return d;
}

static void fillLaunch(Launch& L, const BatchDesc& d, int nb, int ncols, const ws_expr_env& env, const ws_agg_plan* plan,
                       const SlotLayout* lay) {
  memset(&L, 0, sizeof L);
  L.cols = d.cols;
  L.n = (const i64*)d.n;
  L.del = d.del;
  L.tileStart = (const i64*)d.tileStart;
  L.rowStart = (const i64*)d.rowStart;
  L.nb = nb;
  L.ncols = ncols;
  L.ntiles = d.ntiles;
  L.env = envK(env);
  L.progs = d.progs;
  L.kinds = d.kinds;
  L.woff = d.woff;
  L.fwoff = d.fwoff;
  L.aggNull = d.aggNull;
  L.keyInt = d.keyInt;
  if (plan) {
    L.nkeys = plan->nkeys;
    L.naggs = plan->naggs;
  }
  if (lay) {
    L.rowWords = lay->rw;
    L.fastWords = lay->frw;
  }
}

// A compiled plan can only run batches whose columns it was generated for: one generated for raw
// columns cannot decode an encoded segment (the engine's hint, env.cols[c].enc, says which may be).
static bool planCovers(const ws_expr_env& env, int nb, int ncols, const ws_col_view* bcols) {
  for (int b = 0; b < nb; ++b)
    for (int c = 0; c < ncols; ++c)
      if (bcols[(int64_t)b * ncols + c].enc && !env.cols[c].enc) return false;
  return true;
}

}  // namespace ws

using namespace ws;

// ================================================================ aggregation
struct ws_aggregator {
  ws_agg_plan plan{};
  ws_dense_spec dense{};
  bool isDense = false;
  SlotLayout lay;
  int64_t cap = 1;  // hash rows (power of two) / dense groups / 1
  int ncols = 0;
  std::vector<int64_t> bn;
  std::vector<const uint32_t*> bdel;
  std::vector<ws_col_view> bcols;
  int64_t rowsDone = 0;
  int batchesDone = 0, windows = 0;
  DBuf<u64> rows;
  DBuf<double> tkeys;
  // control words after the rows (kCtlWords)
  uint8_t* ctl() { return (uint8_t*)(rows.p + nrows() * lay.rw); }
  std::vector<int64_t> hi;
  // What the last fetch learned of the run's result, until the next run: the status (flags, groups), of a small
  // result also its groups in host memory (keys and engine-format doubles row-major, exact words [g][na][2]),
  // of a larger one the groups before each chunk of kOccChunk result rows.
  bool statusKnown = false, groupsOnHost = false, offsKnown = false;
  ws_fetch_status status{};
  std::vector<double> hostKeys, hostAccs;
  std::vector<int64_t> hostExact;
  DBuf<int64_t> offs;
  void newRun() { statusKnown = groupsOnHost = offsKnown = false; }

  u64* count() { return (u64*)ctl(); }
  int* err() { return (int*)(ctl() + kCtlFlags); }
  unsigned* occTicket() { return (unsigned*)(ctl() + kCtlFlags + 12); }
  unsigned* ticket() { return (unsigned*)(ctl() + kCtlFlags + 16); }
  int64_t nrows() const { return isDense ? dense.G : plan.nkeys ? cap + 1 : 1; }
};

namespace ws {

static RowTemplate rowTemplate(const SlotLayout& lay) {
  RowTemplate t{};
  for (int a = 0; a < lay.na; ++a) {
    const int o = lay.woff[a];
    switch (lay.kind[a]) {
      case SK_IMIN: t.w[o] = (u64)0x7fffffffffffffffll; break;
      case SK_IMAX: t.w[o] = (u64)0x8000000000000000ll; break;
      case SK_DMIN: {
        double inf = __builtin_inf();
        long long b;
        memcpy(&b, &inf, 8);
        t.w[o] = (u64)(b >= 0 ? b : (b ^ 0x7fffffffffffffffll));
        break;
      }
      case SK_DMAX: {
        double inf = -__builtin_inf();
        long long b;
        memcpy(&b, &inf, 8);
        t.w[o] = (u64)(b >= 0 ? b : (b ^ 0x7fffffffffffffffll));
        break;
      }
      default: break;
    }
  }
  return t;
}

static FillSpec fillSpec(ws_aggregator& A) {
  const int64_t emptyRows = A.plan.nkeys && !A.isDense ? A.cap : 0;
  return FillSpec{A.rows.p, A.nrows() * A.lay.rw, emptyRows * A.lay.rw, A.lay.rw, (u64*)A.ctl(), rowTemplate(A.lay)};
}

// Result rows to their identities (hash rows empty) and the control words (count, flags, tickets) to 0.
static void aggResetRows(ws_aggregator& A) {
  const FillSpec f = fillSpec(A);
  WS_LAUNCH(kFillRows, gridFor(f.words, 256, 16), 256, 0, f);
}

static void aggInitRows(ws_aggregator& A) {
  const int64_t nr = A.nrows();
  const int64_t words = nr * A.lay.rw + kCtlWords;
  A.rows = DBuf<u64>((u64*)tableAlloc(8 * (size_t)words), words);
  // key values beside the table: several keys only (a single key is its key word, in the extra row too: the empty
  // marker's bits)
  if (A.plan.nkeys > 1 && !A.isDense) A.tkeys = DBuf<double>((A.cap + 1) * A.plan.nkeys);
  aggResetRows(A);
}

static TuneChoice tuneScan(ws_aggregator& A, const std::string& key, const std::vector<TuneChoice>& cands,
                           const std::function<void(const TuneChoice&)>& launch);

// Bytes of a group's accumulators in a shared-memory table (compact words, ws_kern.cuh; the interpreter keeps
// accumulator rows), integer sums with top words or without.
static size_t groupBytes(const ws_aggregator& A, bool compact, bool tops = true) {
  if (!compact) return (size_t)A.lay.rw * 8;
  size_t b = 0;
  for (int a = 0; a < A.lay.na; ++a) {
    const int k = A.lay.kind[a];
    b += k == SK_COUNT ? 4 : k == SK_ISUM && tops ? 12 : k != SK_NONE ? 8 : 0;
  }
  return b;
}

// The hash scan's shared memory (ws_shape.h); f: its kernel; tableKB: the table's size where tuned or given
// (WARPSTORE_B200_HASH_SMEM_KB), 0: chosen.
static HashTable hashTableOf(const ws_aggregator& A, bool compiled, CUfunction f, int tableKB) {
  static const int envKB = [] {
    const char* e = getenv("WARPSTORE_B200_HASH_SMEM_KB");
    const int v = e ? atoi(e) : 0;
    return v >= 4 && v <= 160 ? v : 0;
  }();
  int resident = 0;
  WS_CKD(drv().occupancy(&resident, f, kThreads, 0));
  const size_t acc = groupBytes(A, compiled), keys = A.plan.nkeys > 1 ? (size_t)A.plan.nkeys * 8 : 0;
  return hashTable(A.cap, 9 + keys + acc, acc, kHotKeys, kHotCopies, resident, (size_t)(tableKB > 0 ? tableKB : envKB),
                   compiled);
}

// A scan prepared for launching elsewhere (a captured graph): kernel, shape, launch descriptor and the
// device buffers the descriptor points to.
struct PreparedScan {
  bool direct = false;    // in: direct loads only (a multi-query launch has no staged form)
  bool ready = false;     // false: the batches hold no tiles (nothing to launch)
  bool compiled = false;  // the plan's generated kernels (not the interpreter)
  bool hot = false;       // of the evaluator of hinted storage (ws_jit_program::kernels)
  int scan = -1;          // the scan kind's KernelId
  CUfunction f = nullptr;
  unsigned grid = 0;
  size_t smem = 0;
  int threads = kThreads;
  Launch L{};
  BatchDesc desc;
  DBuf<u64> part;
};

// The aggregation scan over the collected batches; with `prep`, everything up to the launch (descriptor
// upload, kernel and shape choice, tuning) is done and the launch is handed to the caller instead.
static void aggRun(ws_aggregator& A, const ws_expr_env& env, const ws_jit_program* jit, PreparedScan* prep = nullptr) {
  const int nb = (int)A.bn.size();
  if (nb == 0) return;
  A.newRun();
  const bool interpretable = A.plan.naggs <= WS_INTERP_AGGS && A.plan.nkeys <= WS_INTERP_KEYS;
  const KernelSet* compiled = jit && jit->state.load() == 1 && planCovers(env, nb, A.ncols, A.bcols.data())
                                  ? jit->kernelsFor(nb, A.ncols, A.bcols.data()) : nullptr;
  const bool useJit = compiled != nullptr;
  if (!useJit && !interpretable)
    throw Error("this aggregation needs a compiled plan (more than 16 aggregates or 4 GROUP BY keys); codegen failed or is off", WS_ERR_PLAN);
  std::unique_ptr<TProgs> progs;
  if (!useJit) {
    progs.reset(new TProgs);
    buildTProgs(env, A.ncols, A.plan, A.plan.hasWhere, *progs);
  }
  BatchDesc d = uploadBatches(nb, A.ncols, A.bn.data(), A.bdel.data(), A.bcols.data(), progs.get(), &A.lay, &A.plan);
  if (d.ntiles == 0) return;
  Launch L;
  fillLaunch(L, d, nb, A.ncols, env, &A.plan, &A.lay);
  L.rows = A.rows.p;
  L.err = A.err();
  L.ticket = A.ticket();
  const KernelSet& ks = useJit ? *compiled : interpKernels();
  // Staged scans: a ring of 2..4 tile stages in shared memory (compiled plans only).
  const int stageBytes = useJit ? jit->stageBytes : 0;
  static const int maxStages = [] {  // WARPSTORE_B200_STAGES: shared-memory tile stages (0: direct loads,
                                      // measured faster for the dense scan, which then fits 2 CTAs per SM)
    const char* e = getenv("WARPSTORE_B200_STAGES");
    return e ? std::max(0, std::min(8, atoi(e))) : 0;
  }();
  const int S = stageBytes > 0 ? (int)std::min<int64_t>(maxStages, (200 * 1024) / stageBytes) : 0;
  // The scan's launch shape as a function of a tuning choice: kernel, shared memory, block size and
  // the launch fields the shape changes.  Per-CTA partial rows (`part`: no-key and private-row scans)
  // are sized by the grid.
  struct Shape {
    CUfunction f = nullptr;
    size_t smem = 0;
    int threads = kThreads;
  };
  std::function<Shape(const TuneChoice&)> shapeOf;
  const char* name = "";
  int64_t partRows = 0;  // rows of `part` per CTA (0: none)
  int tilesPerCta = 1;   // tiles a CTA visits at a time
  std::vector<TuneChoice> cands(1);  // candidates for the autotuner; [0] = the default shape
  auto ctas = [](int c) {
    TuneChoice t;
    t.ctasPerSm = c;
    return t;
  };
  auto staged = [](int st) {
    TuneChoice t;
    t.stages = st;
    return t;
  };
  Launch* lp = &L;
  if (A.plan.nkeys == 0) {
    CUfunction f = ks.fn[K_NOKEYS];
    if (!f) throw Error("compiled plan has no aggregation kernel", WS_ERR_INTERNAL);
    shapeOf = [=](const TuneChoice& c) {
      // stage count: the choice's, else the default; within 200 KB of tile stages
      int st = c.stages >= 0 ? c.stages : S;
      if (stageBytes > 0) st = (int)std::min<int64_t>(st, (200 * 1024) / stageBytes);
      CUfunction stagedFn = st < 2 || stageBytes <= 0 ? nullptr : jit->stagedKernel(K_NOKEYS_STAGED);
      if (!stagedFn) st = 0;
      lp->stages = st;
      return Shape{st ? stagedFn : f, (size_t)st * stageBytes, st ? kStagedThreads : kThreads};
    };
    name = "nokeys";
    partRows = 1;
    cands.push_back(ctas(2));
    cands.push_back(ctas(1));
    if (stageBytes > 0)
      for (int st : {0, 2, 3})
        if (st != (S >= 2 ? S : 0)) cands.push_back(staged(st));
  } else if (A.isDense) {
    for (int k = 0; k < A.plan.nkeys; ++k) {
      L.kmin[k] = A.dense.kmin[k];
      L.range[k] = A.dense.range[k];
      L.stride[k] = A.dense.stride[k];
    }
    L.G = A.dense.G;
    L.kmin32 = 1;
    for (int k = 0; k < A.plan.nkeys; ++k)
      if (A.dense.kmin[k] > (1 << 30) || A.dense.kmin[k] < -(1 << 30)) L.kmin32 = 0;
    const int64_t G = A.dense.G;
    // few groups: private register rows per thread in shared memory (+ staged tiles when they fit)
    // private rows [G][frw][kThreads] + int128 spill counters [G][NA][2] (NA: the evaluator's slot bound)
    const int naEv = ks.interp ? WS_INTERP_AGGS : A.plan.naggs;
    const size_t privBytes = (size_t)G * A.lay.frw * kThreads * 8 + (size_t)G * naEv * 16;
    // compact accumulators per group (ws_kern.cuh), in copies while they are small: few groups meet in a warp
    size_t perGroup = groupBytes(A, !ks.interp);
    int copies = 1;
    // A table an SM holds once pays when the CTA brings the SM's warps with it (denseV: 5000 groups of 24 B, 12M rows:
    // 83 us against 377 us of L2 atomics), and where the rows well outnumber the groups each CTA merges
    const int denseV = ks.denseV;
    const size_t sharedLimit = denseV > 1 ? 200 * 1024 : 96 * 1024;
    // Sums without top words where only they fit: rows of large arguments then go to the global rows, which take them
    // all otherwise.
    const bool tops = (size_t)G * perGroup <= sharedLimit;
    if (!tops) perGroup = groupBytes(A, !ks.interp, false);
    while (!ks.interp && copies < 8 && (size_t)G * copies * 2 * perGroup <= 24 * 1024) copies <<= 1;
    const size_t sharedSmem = (size_t)G * copies * perGroup;
    const bool sharedPays = sharedSmem <= 48 * 1024 || d.rows >= 16 * G;
    if (G * A.lay.frw <= 48 && ks.fn[K_DENSE_PRIV]) {
      // tile stages fit beside the private rows within 220 KB; the staged body is its own entry
      const int64_t room = std::max<int64_t>(0, (int64_t)(220 * 1024) - (int64_t)privBytes);
      const int fitStages = stageBytes > 0 ? (int)std::min<int64_t>(8, room / stageBytes) : 0;
      CUfunction direct = ks.fn[K_DENSE_PRIV];
      shapeOf = [=](const TuneChoice& c) {
        int st = std::min(c.stages >= 0 ? c.stages : maxStages, fitStages);
        CUfunction stagedFn = st < 2 ? nullptr : jit->stagedKernel(K_DENSE_PRIV_STAGED);
        if (!stagedFn) st = 0;
        lp->stages = st;
        return Shape{st ? stagedFn : direct, (size_t)st * stageBytes + privBytes, st ? kStagedThreads : kThreads};
      };
      name = "dense_priv";
      partRows = G;
      cands.push_back(ctas(1));
      if (fitStages >= 2)
        for (int st : {0, 2, 3})
          if (st <= fitStages && st != (std::min(maxStages, fitStages) >= 2 ? std::min(maxStages, fitStages) : 0))
            cands.push_back(staged(st));
    } else if (sharedSmem <= sharedLimit && sharedPays && ks.fn[K_DENSE_SHARED]) {
      CUfunction f = ks.fn[tops && ks.fn[K_DENSE_TOPS] ? K_DENSE_TOPS : K_DENSE_SHARED];
      L.copies = copies;
      tilesPerCta = denseV;
      shapeOf = [=](const TuneChoice&) { return Shape{f, sharedSmem, kThreads * denseV}; };
      name = "dense_shared";
      cands.push_back(ctas(2));
      cands.push_back(ctas(1));
    } else {
      CUfunction f = ks.fn[K_DENSE_GLOBAL];
      if (!f) throw Error("compiled plan has no dense kernel", WS_ERR_INTERNAL);
      shapeOf = [=](const TuneChoice&) { return Shape{f, 0, kThreads}; };
      name = "dense_global";
      cands.push_back(ctas(4));
      cands.push_back(ctas(2));
    }
  } else {
    CUfunction f = ks.fn[K_HASH];
    if (!f) throw Error("compiled plan has no hash aggregation kernel", WS_ERR_INTERNAL);
    L.table = A.rows.p;
    L.tkeys = A.tkeys.p;
    L.mask = (u64)(A.cap - 1);
    L.count = A.count();
    L.probeLimit = (int)std::min<int64_t>(A.cap, 1 << 16);
    const size_t per = (size_t)A.lay.rw * 8 + (A.plan.nkeys > 1 ? (size_t)A.plan.nkeys * 8 : 0);
    ws_aggregator* ap = &A;
    const bool compiledPlan = !ks.interp;
    shapeOf = [=](const TuneChoice& c) {
      const HashTable t = hashTableOf(*ap, compiledPlan, f, c.smemKB);
      lp->smemSlots = (int)t.slots;
      lp->copies = t.copies;
      lp->spillRows = (int)std::min<size_t>(kTile, t.spill / per);
      return Shape{f, t.bytes + (size_t)lp->spillRows * per, kThreads};
    };
    name = "hash";
    for (int kb : {16, 32, 96}) {
      TuneChoice t;
      t.smemKB = kb;
      cands.push_back(t);
    }
    cands.push_back(ctas(2));
  }
  DBuf<u64> part;
  int64_t partCap = 0;
  auto launchOnce = [&](const TuneChoice& c) {
    const Shape sh = shapeOf(c);
    unsigned grid = persistentGrid(sh.f, sh.smem, (d.ntiles + tilesPerCta - 1) / tilesPerCta, sh.threads);
    if (c.ctasPerSm > 0) grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(grid, (int64_t)c.ctasPerSm * smCount()));
    if (partRows) {
      if ((int64_t)grid * partRows > partCap) {
        partCap = (int64_t)grid * partRows;
        part = DBuf<u64>(partCap * A.lay.rw);
      }
      L.part = part.p;
      WS_CK(cudaMemsetAsync(A.ticket(), 0, 4, stream()));
    }
    launchScan(sh.f, grid, sh.smem, L, sh.threads);
  };
  const std::string key = tuneKey(name, useJit ? jit : nullptr, A.plan, d.ntiles);
  TuneChoice choice;
  if (prep && prep->direct) {  // tuned without staged candidates: a multi-query launch loads directly
    std::vector<TuneChoice> directOnly;
    for (const TuneChoice& c : cands)
      if (c.stages <= 0) directOnly.push_back(c);
    for (TuneChoice& c : directOnly) c.stages = 0;
    cands.swap(directOnly);
  }
  if (!tuneLookup(key, choice) && tuneMode() == WS_TUNE_ON && A.windows == 0 && A.rowsDone == 0)
    choice = tuneScan(A, key, cands, launchOnce);
  if (prep && prep->direct) choice.stages = 0;
  if (prep) {
    const Shape sh = shapeOf(choice);
    unsigned grid = persistentGrid(sh.f, sh.smem, (d.ntiles + tilesPerCta - 1) / tilesPerCta, sh.threads);
    if (choice.ctasPerSm > 0)
      grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(grid, (int64_t)choice.ctasPerSm * smCount()));
    if (partRows) {
      part = DBuf<u64>((int64_t)grid * partRows * A.lay.rw);
      L.part = part.p;
    }
    prep->compiled = useJit;
    prep->hot = useJit && &ks == &jit->kernels;
    for (int k : {K_NOKEYS, K_DENSE_PRIV, K_HASH})
      if (sh.f == ks.fn[k]) prep->scan = k;
    prep->f = sh.f;
    prep->grid = grid;
    prep->smem = sh.smem;
    prep->threads = sh.threads;
    prep->L = L;
    prep->L.sumShift = sumShiftFor(L.ntiles, grid);
    prep->L.waitLog2 = stagedWaitLog2();
    prep->desc = std::move(d);
    prep->part = std::move(part);
    prep->ready = true;
    return;
  }
  launchOnce(choice);
}

// Times each candidate launch shape of a scan on the aggregation's own batches (best of two runs,
// CUDA events on the calling stream, the result rows reset before each run) and records the fastest;
// the rows are reset again for the caller's final run.  A run that raised a flag (overflow, key out of
// range) records nothing: the final run raises it again and the caller decides.
static TuneChoice tuneScan(ws_aggregator& A, const std::string& key, const std::vector<TuneChoice>& cands,
                           const std::function<void(const TuneChoice&)>& launch) {
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  WS_CK(cudaEventCreate(&e0));
  WS_CK(cudaEventCreate(&e1));
  TuneChoice best;
  double bestMs = 1e300;
  bool flagged = false;
  try {
    for (const TuneChoice& c : cands) {
      double ms = 1e300;
      for (int rep = 0; rep < 2; ++rep) {
        aggResetRows(A);
        WS_CK(cudaEventRecord(e0, stream()));
        launch(c);
        WS_CK(cudaEventRecord(e1, stream()));
        WS_CK(cudaEventSynchronize(e1));
        float t = 0;
        WS_CK(cudaEventElapsedTime(&t, e0, e1));
        ms = std::min(ms, (double)t);
      }
      int e[3] = {0, 0, 0};
      d2hSync(e, A.err(), 12);
      flagged |= e[0] || e[1] || e[2];
      if (ms < bestMs) bestMs = ms, best = c;
    }
  } catch (...) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    throw;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  aggResetRows(A);
  if (flagged) return TuneChoice{};
  tuneStore(key, best, bestMs * 1000);
  best.found = true;
  return best;
}

static ResultSpec resultSpec(ws_aggregator& A) {
  ResultSpec s{};
  s.rows = A.rows.p;
  s.nrows = A.nrows();
  s.cap = A.cap;
  s.err = A.err();
  s.tkeys = A.tkeys.p;
  s.rw = A.lay.rw;
  s.mode = A.plan.nkeys == 0 ? 0 : A.isDense ? 1 : 2;
  s.cnt0 = A.lay.woff[0];
  s.nk = A.plan.nkeys;
  s.na = A.plan.naggs;
  for (int a = 0; a < s.na; ++a) {
    s.derived[a] = A.lay.kind[a] == SK_NONE;
    const int src = s.derived[a] ? A.lay.partner[a] : a;
    s.kind[a] = A.lay.kind[src];
    s.woff[a] = (int16_t)A.lay.woff[src];
    s.aggBits[a] = A.plan.aggBits[a];
    s.aggPart[a] = A.plan.aggPart[a];
  }
  for (int k = 0; k < s.nk; ++k) {
    s.keyInt[k] = A.plan.keyInt[k];
    s.kmin[k] = A.dense.kmin[k];
    s.range[k] = A.isDense ? A.dense.range[k] : 1;
    s.stride[k] = A.isDense ? A.dense.stride[k] : 1;
  }
  return s;
}

// Pinned and mapped memory that small results are delivered into, one block per thread (its size is bounded
// by kHostResultBytes; freed when the thread ends).  Its contents are copied out before the call returns.
constexpr size_t kHostResultBytes = 1u << 20;
static uint8_t* hostResult() {
  struct Block {
    uint8_t* p = nullptr;
    ~Block() {
      if (p) cudaFreeHost(p);
    }
  };
  static thread_local Block b;
  if (!b.p) WS_CK(cudaHostAlloc((void**)&b.p, kHostResultBytes, cudaHostAllocMapped));
  return b.p;
}
template <class T>
static T* mappedPtr(T* host) {
  void* d = nullptr;
  WS_CK(cudaHostGetDevicePointer(&d, (void*)host, 0));
  return (T*)d;
}

constexpr size_t kStatusBytes = 64;  // the status at the start of a host result block
// A result delivered whole into the thread's host block: few rows, all of whose groups fit it.
static bool smallResult(const ws_aggregator& A) {
  return A.nrows() <= kSmallRows &&
         kStatusBytes + (size_t)A.nrows() * 8 * (size_t)(A.plan.nkeys + 3 * A.plan.naggs) <= kHostResultBytes;
}

// The run's status (flags and number of groups) on the host: a small result is delivered whole, a larger
// one's chunks are counted.  One wait.
static const ws_fetch_status& learnStatus(ws_aggregator& A) {
  if (A.statusKnown) return A.status;
  uint8_t* h = hostResult();
  uint8_t* d = mappedPtr(h);
  const size_t nk = (size_t)A.plan.nkeys, na = (size_t)A.plan.naggs, nr = (size_t)A.nrows();
  const size_t oKeys = kStatusBytes, oAccs = oKeys + 8 * nk * nr, oExact = oAccs + 8 * na * nr;
  const bool small = smallResult(A);
  if (small) {
    DeliverSpec ds{resultSpec(A),
                   {nk ? (double*)(d + oKeys) : nullptr, (double*)(d + oAccs), (long long*)(d + oExact), 0, (int64_t)nr, 0},
                   (ws_fetch_status*)d, 1};
    WS_LAUNCH(kDeliver, 1, kDeliverThreads, 0, ds);
  } else {
    const int64_t nchunks = ((int64_t)nr + kOccChunk - 1) / kOccChunk;
    A.offs = DBuf<int64_t>(nchunks + 1);
    WS_LAUNCH(kOccCount, (unsigned)nchunks, kOccThreads, 0, resultSpec(A), A.offs.p, nchunks, A.occTicket(),
              (ws_fetch_status*)d);
    A.offsKnown = true;
  }
  sync();
  memcpy(&A.status, h, sizeof A.status);
  if (small && !A.status.error) {
    const size_t g = (size_t)A.status.groups;
    A.hostKeys.assign((const double*)(h + oKeys), (const double*)(h + oKeys) + g * nk);
    A.hostAccs.assign((const double*)(h + oAccs), (const double*)(h + oAccs) + g * na);
    A.hostExact.assign((const int64_t*)(h + oExact), (const int64_t*)(h + oExact) + g * na * 2);
    A.groupsOnHost = true;
  }
  A.statusKnown = true;
  return A.status;
}

static void throwFlags(const ws_fetch_status& st) {
  if (st.error == WS_ERR_RANGE) throw Error("dense GROUP BY key outside its declared range", WS_ERR_RANGE);
  if (st.error) throw Error("a staged tile copy did not complete in time", WS_ERR_INTERNAL);
}

// Queues the groups of a counted result (offs known) to device or mapped memory.
static void emitChunks(ws_aggregator& A, const int64_t* offs, const OutSpec& o, bool evenOverflowed) {
  WS_LAUNCH(kEmitChunks, (unsigned)((A.nrows() + kOccChunk - 1) / kOccChunk), kOccThreads, 0, resultSpec(A), o, offs,
            evenOverflowed ? 1 : 0);
}

// One multi-query scan over prepared queries (ws_agg_run_many, ws_exec_group_*): the kernel of the
// queries' common scan kind, its shared memory and block, the queries that have tiles, their CTA
// starts (the launch's resident CTAs shared out by tiles: each query at least one CTA, at most its own
// persistent grid, which its partial rows were sized for) and their launch descriptors.
struct MultiPlan {
  CUfunction f = nullptr;
  size_t smem = 0;
  int threads = 0;
  std::vector<int> live;    // indices of the queries with tiles
  std::vector<int> start;   // CTA starts, live.size() + 1
  std::vector<Launch> L;    // per live query, ctaBase / ctaGrid left for the kernel
};

static MultiPlan planMulti(const std::vector<const PreparedScan*>& preps, const ws_jit_program* jit, const char* who) {
  MultiPlan mp;
  // queries whose batches all are stored as hinted run that evaluator's kernel, else all run the generic one
  bool hot = true;
  for (const PreparedScan* p : preps) hot = hot && (!p->ready || p->hot);
  const KernelSet* ks = nullptr;
  int multi = -1;
  int64_t tiles = 0;
  for (size_t i = 0; i < preps.size(); ++i) {
    const PreparedScan& p = *preps[i];
    if (!p.ready) continue;  // no tiles: nothing to scan
    if (p.compiled && !jit) throw Error(std::string(who) + ": compiled queries need their plan", WS_ERR_ARG);
    const KernelSet& own = !p.compiled ? interpKernels() : p.hot ? jit->kernels : jit->any;
    const KernelSet& k = !p.compiled ? interpKernels() : hot ? jit->kernels : jit->any;
    const int m = p.scan < 0 || p.f != own.fn[p.scan] ? -1
                : p.scan == K_NOKEYS ? K_MULTI_NOKEYS : p.scan == K_DENSE_PRIV ? K_MULTI_DENSE_PRIV : K_MULTI_HASH;
    if (m < 0 || !k.fn[m] || p.L.stages)
      throw Error(std::string(who) + ": a query's scan has no multi-query form (dense shared / global rows, staged tiles)",
                  WS_ERR_ARG);
    if (multi >= 0 && (m != multi || &k != ks))
      throw Error(std::string(who) + ": the queries need one scan kind and one plan (or all interpreted)", WS_ERR_ARG);
    ks = &k, multi = m;
    mp.smem = std::max(mp.smem, p.smem);
    mp.threads = p.threads;
    tiles += p.L.ntiles;
    mp.live.push_back((int)i);
  }
  if (mp.live.empty()) return mp;
  mp.f = ks->fn[multi];
  const unsigned total = persistentGrid(mp.f, mp.smem, std::max<int64_t>(tiles, (int64_t)mp.live.size()), mp.threads);
  mp.start.assign(mp.live.size() + 1, 0);
  for (size_t j = 0; j < mp.live.size(); ++j) {
    const PreparedScan& p = *preps[(size_t)mp.live[j]];
    int64_t share = (int64_t)((double)total * (double)p.L.ntiles / (double)tiles);
    share = std::max<int64_t>(1, std::min<int64_t>(share, std::min<int64_t>(p.grid, p.L.ntiles)));
    mp.start[j + 1] = mp.start[j] + (int)share;
    Launch L = p.L;
    L.sumShift = sumShiftFor(L.ntiles, (unsigned)share);
    L.waitLog2 = stagedWaitLog2();
    L.ctaBase = L.ctaGrid = 0;  // set per CTA by the kernel
    mp.L.push_back(L);
  }
  return mp;
}

}  // namespace ws

extern "C" {

int ws_agg_create(const ws_agg_plan* plan, int64_t capacity, const ws_dense_spec* dense, ws_aggregator** out) {
  return guardedCall([&] {
    *out = nullptr;
    std::unique_ptr<ws_aggregator> A(new ws_aggregator);
    A->plan = *plan;
    A->lay = layoutOf(*plan);
    if (dense && dense->G > 0 && plan->nkeys) {
      A->dense = *dense;
      A->isDense = true;
      A->cap = dense->G;
    } else if (plan->nkeys) {
      int64_t c = 1;
      while (c < capacity) c <<= 1;
      A->cap = std::max<int64_t>(c, 2);
    } else {
      A->cap = 1;
    }
    aggInitRows(*A);
    *out = A.release();
  });
}

void ws_agg_destroy(ws_aggregator* agg) { delete agg; }

int ws_agg_add_batch(ws_aggregator* A, const ws_expr_env* env, int ncols, int64_t n, const uint32_t* del) {
  return guardedCall([&] {
    if (n <= 0) return;
    if (ncols < 0 || ncols > WS_MAX_COLS) throw Error("bad column count", WS_ERR_ARG);
    if (!A->bn.empty() && ncols != A->ncols) throw Error("batches must have the same column count", WS_ERR_ARG);
    A->ncols = ncols;
    A->bn.push_back(n);
    A->bdel.push_back(del);
    for (int i = 0; i < ncols; ++i) A->bcols.push_back(env->cols[i]);
  });
}

int ws_agg_add_batches(ws_aggregator* A, int ncols, int nb, const int64_t* bn, const uint32_t* const* bdel,
                       const ws_col_view* bcols) {
  return guardedCall([&] {
    if (ncols < 0 || ncols > WS_MAX_COLS || nb < 0) throw Error("bad column or batch count", WS_ERR_ARG);
    for (int b = 0; b < nb; ++b) {
      if (bn[b] <= 0) continue;
      if (!A->bn.empty() && ncols != A->ncols) throw Error("batches must have the same column count", WS_ERR_ARG);
      A->ncols = ncols;
      A->bn.push_back(bn[b]);
      A->bdel.push_back(bdel ? bdel[b] : nullptr);
      A->bcols.insert(A->bcols.end(), bcols + (int64_t)b * ncols, bcols + (int64_t)(b + 1) * ncols);
    }
  });
}

int ws_agg_run(ws_aggregator* A, const ws_expr_env* env, const ws_jit_program* jit) {
  return guardedCall([&] { aggRun(*A, *env, jit); });
}

int ws_agg_run_many(ws_aggregator* const* aggs, const ws_expr_env* const* envs, const ws_jit_program* jit, int n) {
  return guardedCall([&] {
    if (n < 1 || n > 1024 || !aggs || !envs) throw Error("ws_agg_run_many: 1..1024 aggregators", WS_ERR_ARG);
    // each query prepared as for its own launch (descriptor uploaded, kernel and shape chosen)
    std::vector<PreparedScan> preps((size_t)n);
    for (int i = 0; i < n; ++i) {
      preps[(size_t)i].direct = true;
      aggRun(*aggs[i], *envs[i], jit, &preps[(size_t)i]);
    }
    std::vector<const PreparedScan*> pp;
    for (const PreparedScan& p : preps) pp.push_back(&p);
    const MultiPlan mp = planMulti(pp, jit, "ws_agg_run_many");
    if (mp.live.empty()) return;
    const size_t nl = mp.live.size();
    const size_t launchBytes = nl * sizeof(Launch), startBytes = (nl + 1) * sizeof(int);
    uint8_t* st = pinnedStage(launchBytes + startBytes);
    memcpy(st, mp.L.data(), launchBytes);
    memcpy(st + launchBytes, mp.start.data(), startBytes);
    for (const Launch& L : mp.L)
      if (L.ticket) WS_CK(cudaMemsetAsync(L.ticket, 0, 4, stream()));
    DBuf<uint8_t> dl((int64_t)(launchBytes + startBytes));
    h2dAsync(dl.p, st, launchBytes + startBytes);
    stageCopied();
    MultiLaunch M{(const Launch*)dl.p, (const int*)(dl.p + launchBytes), (int)nl};
    allowDynamicSmem(mp.f, mp.smem);
    void* args[] = {(void*)&M};
    WS_CKD(drv().launchKernel(mp.f, (unsigned)mp.start[nl], 1, 1, (unsigned)mp.threads, 1, 1, (unsigned)mp.smem,
                              (CUstream)stream(), args, nullptr));
    countLaunch();
  });
}

int ws_agg_run_window(ws_aggregator* A, const ws_expr_env* env, const ws_jit_program* jit) {
  return guardedCall([&] {
    if (A->bn.empty()) return;
    aggRun(*A, *env, jit);
    ++A->windows;
    for (int64_t n : A->bn) A->rowsDone += n;
    A->batchesDone += (int)A->bn.size();
    A->bn.clear();
    A->bdel.clear();
    A->bcols.clear();
  });
}

int ws_agg_batches(const ws_aggregator* A) { return A->batchesDone + (int)A->bn.size(); }
int ws_agg_windows(const ws_aggregator* A) { return A->windows; }
int64_t ws_agg_rows_in(const ws_aggregator* A) {
  int64_t r = A->rowsDone;
  for (int64_t n : A->bn) r += n;
  return r;
}
int ws_agg_is_dense(const ws_aggregator* A) { return A->isDense ? 1 : 0; }
int64_t ws_agg_capacity(const ws_aggregator* A) { return A->cap; }

int ws_agg_overflowed(ws_aggregator* A, int* out) {
  return guardedCall([&] {
    if (smallResult(*A) || A->statusKnown) {  // the groups come along: a fetch usually follows
      const ws_fetch_status& st = learnStatus(*A);
      throwFlags(st);
      *out = st.overflow;
      return;
    }
    int e[3] = {0, 0, 0};
    d2hSync(e, A->err(), 12);
    throwFlags(ws_fetch_status{0, 0, e[0] ? WS_ERR_RANGE : e[2] ? WS_ERR_INTERNAL : 0});
    *out = A->plan.nkeys && !A->isDense && e[1] ? 1 : 0;
  });
}

int ws_agg_group_count(ws_aggregator* A, int64_t* out) {
  return guardedCall([&] {
    if (!A->plan.nkeys) {
      *out = 1;
      return;
    }
    if (A->isDense) {
      *out = learnStatus(*A).groups;
      return;
    }
    u64 c = 0;
    d2hSync(&c, A->count(), 8);
    *out = (int64_t)c;
  });
}

int ws_agg_fetch(ws_aggregator* A, int64_t max_groups, double* keys, double* accs, int64_t* exact, int64_t* ngroups) {
  return guardedCall([&] {
    const int nk = A->plan.nkeys, na = A->plan.naggs;
    const ws_fetch_status& st = learnStatus(*A);
    throwFlags(st);
    const int64_t g = st.groups;
    *ngroups = g;
    if (g > max_groups) throw Error("output buffer too small for " + std::to_string(g) + " groups", WS_ERR_SIZE);
    if (!nk) keys = nullptr;
    if (A->groupsOnHost) {
      if (keys) memcpy(keys, A->hostKeys.data(), sizeof(double) * g * nk);
      if (accs) memcpy(accs, A->hostAccs.data(), sizeof(double) * g * na);
      if (exact) memcpy(exact, A->hostExact.data(), sizeof(int64_t) * g * na * 2);
    } else if (g && (keys || accs || exact)) {
      DBuf<double> dk(keys ? g * nk : 0), da(accs ? g * na : 0);
      DBuf<int64_t> dx(exact ? g * na * 2 : 0);
      emitChunks(*A, A->offs.p, OutSpec{dk.p, da.p, (long long*)dx.p, 0, g, 0}, true);
      if (keys) d2hLarge(keys, dk.p, sizeof(double) * g * nk);
      if (accs) d2hLarge(accs, da.p, sizeof(double) * g * na);
      if (exact) d2hLarge(exact, dx.p, sizeof(int64_t) * g * na * 2);
    }
    A->hi.assign(na, 0);
    if (!nk && A->groupsOnHost)  // high words of exact no-key integer sums (sumHigh)
      for (int a = 0; a < na; ++a) {
        const uint8_t k = A->lay.kind[a] == SK_NONE ? A->lay.kind[A->lay.partner[a]] : A->lay.kind[a];
        A->hi[a] = k == SK_ISUM ? A->hostExact[2 * a + 1] : 0;
      }
  });
}

int ws_agg_fetch_async(ws_aggregator* A, int64_t first_group, int64_t max_groups, double* keys, int64_t* exact,
                       ws_fetch_status* status) {
  return guardedCall([&] {
    const int nk = A->plan.nkeys;
    auto mapped = [](void* h, const char* what) -> void* {
      if (!h) throw Error(std::string("fetch_async: ") + what + " is null", WS_ERR_ARG);
      cudaPointerAttributes at{};
      if (cudaPointerGetAttributes(&at, h) != cudaSuccess || at.type != cudaMemoryTypeHost || !at.devicePointer) {
        cudaGetLastError();
        throw Error(std::string("fetch_async: ") + what + " is not pinned host memory", WS_ERR_ARG);
      }
      return at.devicePointer;
    };
    auto* st = (ws_fetch_status*)mapped(status, "status");
    double* dk = nk ? (double*)mapped(keys, "keys") : nullptr;
    auto* dx = (long long*)mapped(exact, "exact");
    if (first_group < 0 || max_groups < 0) throw Error("fetch_async: negative group range", WS_ERR_ARG);
    const OutSpec o{dk, nullptr, dx, first_group, max_groups, 0};
    if (A->nrows() <= kSmallRows) {
      WS_LAUNCH(kDeliver, 1, kDeliverThreads, 0, DeliverSpec{resultSpec(*A), o, st, 0});
      return;
    }
    const int64_t nchunks = (A->nrows() + kOccChunk - 1) / kOccChunk;
    if (!A->offsKnown) {  // group offsets per chunk, kept for the later ranges of the same run
      A->offs = DBuf<int64_t>(nchunks + 1);
      WS_LAUNCH(kOccCount, (unsigned)nchunks, kOccThreads, 0, resultSpec(*A), A->offs.p, nchunks, A->occTicket(), st);
      A->offsKnown = true;
    } else {
      WS_LAUNCH(kFetchStatus, 1, 1, 0, resultSpec(*A), A->offs.p + nchunks, st);
    }
    if (max_groups) emitChunks(*A, A->offs.p, o, false);
  });
}

}  // extern "C"

// A prepared query (ws_exec_*): the aggregation's result rows, its batch descriptor and one CUDA graph
// of the whole query — result rows reset, the scan, compaction, the groups and the status written into
// pinned host memory — captured once; each run updates the scan node's launch descriptor (the plan's
// constants) and launches the graph.
struct ws_executor {
  ws_aggregator* A = nullptr;
  ws::PreparedScan ps;
  uint64_t code = 0;  // digest of the expressions the graph was built for
  int64_t maxGroups = 0;
  double* keys = nullptr;
  int64_t* exact = nullptr;
  ws_fetch_status* st = nullptr;
  ws::DBuf<int64_t> offs;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaGraphNode_t scanNode = nullptr;
  int kernels = 0;  // kernel nodes per run
  ~ws_executor() {
    cudaStreamSynchronize(ws::stream());  // a run queued on this thread's stream may still be in flight
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (keys) cudaFreeHost(keys);
    if (exact) cudaFreeHost(exact);
    if (st) cudaFreeHost(st);
    if (A) ws_agg_destroy(A);
  }
};

namespace {
OutSpec execOut(ws_executor& X) {
  return OutSpec{X.A->plan.nkeys ? mappedPtr(X.keys) : nullptr, nullptr, (long long*)mappedPtr(X.exact), 0, X.maxGroups, 0};
}
// Queues on this thread's stream the part of a prepared query after its scan: compaction of the
// result rows, the status word and the groups written into the executor's pinned memory.  Returns the
// kernels queued.
int queueExecTail(ws_executor& X) {
  ws_aggregator& A = *X.A;
  ws_fetch_status* st = mappedPtr(X.st);
  if (A.nrows() <= kSmallRows) {
    WS_LAUNCH(kDeliver, 1, kDeliverThreads, 0, DeliverSpec{resultSpec(A), execOut(X), st, 0});
    return 1;
  }
  const int64_t nchunks = (A.nrows() + kOccChunk - 1) / kOccChunk;
  WS_LAUNCH(kOccCount, (unsigned)nchunks, kOccThreads, 0, resultSpec(A), X.offs.p, nchunks, A.occTicket(), st);
  emitChunks(A, X.offs.p, execOut(X), false);
  return 2;
}

uint64_t codeDigest(const ws_expr_env& env) {
  uint64_t h = 0xcbf29ce484222325ull;
  const unsigned char* b = (const unsigned char*)env.code;
  for (size_t i = 0; i < sizeof env.code; ++i) h = (h ^ b[i]) * 0x100000001b3ull;
  return h;
}
}  // namespace

extern "C" {

int ws_exec_create(const ws_agg_plan* plan, int64_t capacity, const ws_dense_spec* dense, const ws_expr_env* env,
                   int ncols, int nb, const int64_t* bn, const uint32_t* const* bdel, const ws_col_view* bcols,
                   const ws_jit_program* jit, int64_t max_groups, ws_executor** out) {
  return guardedCall([&] {
    *out = nullptr;
    if (max_groups < 1) throw Error("exec: max_groups must be positive", WS_ERR_ARG);
    if (!jit || jit->state.load() != 1) throw Error("exec: a prepared query needs a compiled plan", WS_ERR_PLAN);
    std::unique_ptr<ws_executor> X(new ws_executor);
    if (int rc = ws_agg_create(plan, capacity, dense, &X->A)) throw Error(ws_last_error(), rc);
    if (int rc = ws_agg_add_batches(X->A, ncols, nb, bn, bdel, bcols)) throw Error(ws_last_error(), rc);
    ws_aggregator& A = *X->A;
    aggRun(A, *env, jit, &X->ps);
    if (X->ps.ready && !X->ps.compiled)
      throw Error("exec: the compiled plan does not cover these batches (encodings)", WS_ERR_PLAN);
    X->code = codeDigest(*env);
    X->maxGroups = max_groups;
    const int nk = A.plan.nkeys, na = A.plan.naggs;
    auto pinned = [](size_t bytes, void** p) {
      if (cudaHostAlloc(p, std::max<size_t>(bytes, 8), cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        throw Error("exec: pinned result buffers", WS_ERR_OOM);
      }
    };
    pinned(sizeof(double) * max_groups * std::max(nk, 1), (void**)&X->keys);
    pinned(sizeof(int64_t) * max_groups * na * 2, (void**)&X->exact);
    pinned(sizeof(ws_fetch_status), (void**)&X->st);
    X->offs = DBuf<int64_t>((A.nrows() + kOccChunk - 1) / kOccChunk + 1);
    sync();  // the preparation's copies and allocations are done before the capture starts
    // capture on a private stream (nothing else of this thread's work joins the graph)
    cudaStream_t cs = nullptr;
    WS_CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaStream_t prev = stream();
    auto restore = [&] { ws_set_stream(prev == cudaStreamPerThread ? nullptr : (void*)prev); };
    ws_set_stream(cs);
    bool capturing = false;
    try {
      WS_CK(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
      capturing = true;
      aggResetRows(A);
      X->kernels = 1;
      if (X->ps.ready) {
        const PreparedScan& p = X->ps;
        allowDynamicSmem(p.f, p.smem);
        void* args[] = {(void*)&X->ps.L};
        WS_CKD(drv().launchKernel(p.f, p.grid, 1, 1, (unsigned)p.threads, 1, 1, (unsigned)p.smem, (CUstream)cs, args,
                                  nullptr));
        countLaunch();
        cudaStreamCaptureStatus cst;
        const cudaGraphNode_t* deps = nullptr;
        size_t ndeps = 0;
        WS_CK(cudaStreamGetCaptureInfo(cs, &cst, nullptr, nullptr, &deps, &ndeps));
        if (ndeps != 1) throw Error("exec: could not find the scan in the captured graph", WS_ERR_INTERNAL);
        X->scanNode = deps[0];
        ++X->kernels;
      }
      X->kernels += queueExecTail(*X);
      capturing = false;
      WS_CK(cudaStreamEndCapture(cs, &X->graph));
      WS_CK(cudaGraphInstantiate(&X->exec, X->graph, 0));
    } catch (...) {
      if (capturing) {
        cudaGraph_t g = nullptr;
        cudaStreamEndCapture(cs, &g);
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
      }
      restore();
      cudaStreamDestroy(cs);
      throw;
    }
    countLaunch(-X->kernels);  // captured, not launched
    restore();
    WS_CK(cudaStreamDestroy(cs));
    *out = X.release();
  });
}

int ws_exec_run(ws_executor* X, const ws_expr_env* env) {
  return guardedCall([&] {
    if (codeDigest(*env) != X->code) throw Error("exec: the expressions differ from the prepared query's", WS_ERR_ARG);
    if (X->scanNode) {
      X->ps.L.env = envK(*env);
      void* args[] = {(void*)&X->ps.L};
      CUDA_KERNEL_NODE_PARAMS kp{};
      kp.func = X->ps.f;
      kp.gridDimX = X->ps.grid;
      kp.gridDimY = kp.gridDimZ = 1;
      kp.blockDimX = (unsigned)X->ps.threads;
      kp.blockDimY = kp.blockDimZ = 1;
      kp.sharedMemBytes = (unsigned)X->ps.smem;
      kp.kernelParams = args;
      WS_CKD(drv().graphExecKernelNodeSetParams((CUgraphExec)X->exec, (CUgraphNode)X->scanNode, &kp));
    }
    WS_CK(cudaGraphLaunch(X->exec, stream()));
    countLaunch(X->kernels);
  });
}

int ws_exec_results(ws_executor* X, const double** keys, const int64_t** exact, const ws_fetch_status** status) {
  if (keys) *keys = X->keys;
  if (exact) *exact = X->exact;
  if (status) *status = X->st;
  return WS_OK;
}

void ws_exec_destroy(ws_executor* X) { delete X; }

}  // extern "C"

// Prepared queries of one plan run together (ws_exec_group_*): one CUDA graph that resets every
// query's result rows, copies the queries' launch descriptors from pinned memory (each run writes the
// new constants there first), runs ONE multi-query scan over all of them and then each query's
// compaction and delivery into its own executor's pinned memory.
struct ws_exec_group {
  std::vector<ws_executor*> xs;
  ws::MultiPlan mp;
  uint8_t* stage = nullptr;  // pinned: [Launch per live query][CTA starts]
  size_t stageBytes = 0;
  ws::DBuf<uint8_t> dl;      // the device copy the scan reads
  ws::DBuf<uint8_t> specs;   // the queries' reset specs, then the delivery specs of those with small results
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t done = nullptr;  // the last run's end: its copy of `stage` has been made
  int kernels = 0;
  ~ws_exec_group() {
    if (done) cudaEventSynchronize(done);
    cudaStreamSynchronize(ws::stream());
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (done) cudaEventDestroy(done);
    if (stage) cudaFreeHost(stage);
  }
};

extern "C" {

int ws_exec_group_create(ws_executor* const* xs, int n, const ws_jit_program* jit, ws_exec_group** out) {
  return guardedCall([&] {
    *out = nullptr;
    if (n < 1 || n > 1024 || !xs) throw Error("exec group: 1..1024 prepared queries", WS_ERR_ARG);
    std::unique_ptr<ws_exec_group> G(new ws_exec_group);
    std::vector<const PreparedScan*> pp;
    for (int i = 0; i < n; ++i) {
      if (!xs[i]) throw Error("exec group: a null prepared query", WS_ERR_ARG);
      for (int j = 0; j < i; ++j)
        if (xs[j] == xs[i]) throw Error("exec group: a prepared query given twice", WS_ERR_ARG);
      G->xs.push_back(xs[i]);
      pp.push_back(&xs[i]->ps);
    }
    G->mp = planMulti(pp, jit, "exec group");
    const MultiPlan& mp = G->mp;
    const size_t nl = mp.live.size();
    const size_t launchBytes = nl * sizeof(Launch), startBytes = (nl + 1) * sizeof(int);
    G->stageBytes = launchBytes + startBytes;
    if (cudaHostAlloc((void**)&G->stage, std::max<size_t>(G->stageBytes, 8), cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      G->stage = nullptr;
      throw Error("exec group: pinned descriptor buffer", WS_ERR_OOM);
    }
    if (nl) {
      memcpy(G->stage, mp.L.data(), launchBytes);
      memcpy(G->stage + launchBytes, mp.start.data(), startBytes);
      G->dl = DBuf<uint8_t>((int64_t)G->stageBytes);
    }
    WS_CK(cudaEventCreateWithFlags(&G->done, cudaEventDisableTiming));
    // every query's rows are reset by one launch, and the small results delivered by one (a CTA each)
    std::vector<FillSpec> fills;
    std::vector<DeliverSpec> small;
    int64_t fillWords = 1;
    for (ws_executor* X : G->xs) {
      fills.push_back(fillSpec(*X->A));
      fillWords = std::max(fillWords, fills.back().words);
      if (X->A->nrows() <= kSmallRows) small.push_back(DeliverSpec{resultSpec(*X->A), execOut(*X), mappedPtr(X->st), 0});
    }
    const size_t fillBytes = fills.size() * sizeof(FillSpec), smallBytes = small.size() * sizeof(DeliverSpec);
    G->specs = DBuf<uint8_t>((int64_t)(fillBytes + smallBytes));
    WS_CK(cudaMemcpyAsync(G->specs.p, fills.data(), fillBytes, cudaMemcpyHostToDevice, stream()));
    WS_CK(cudaMemcpyAsync(G->specs.p + fillBytes, small.data(), smallBytes, cudaMemcpyHostToDevice, stream()));
    sync();  // allocations done before the capture starts
    cudaStream_t cs = nullptr;
    WS_CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaStream_t prev = stream();
    auto restore = [&] { ws_set_stream(prev == cudaStreamPerThread ? nullptr : (void*)prev); };
    ws_set_stream(cs);
    const int64_t launches0 = ws_kernel_launches();
    bool capturing = false;
    try {
      WS_CK(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
      capturing = true;
      WS_LAUNCH(kFillRowsMany, dim3(gridFor(fillWords), (unsigned)fills.size()), 256, 0, (const FillSpec*)G->specs.p);
      if (nl) {
        WS_CK(cudaMemcpyAsync(G->dl.p, G->stage, G->stageBytes, cudaMemcpyHostToDevice, cs));
        MultiLaunch M{(const Launch*)G->dl.p, (const int*)(G->dl.p + launchBytes), (int)nl};
        allowDynamicSmem(mp.f, mp.smem);
        void* args[] = {(void*)&M};
        WS_CKD(drv().launchKernel(mp.f, (unsigned)mp.start[nl], 1, 1, (unsigned)mp.threads, 1, 1, (unsigned)mp.smem,
                                  (CUstream)cs, args, nullptr));
        countLaunch();
      }
      if (!small.empty())
        WS_LAUNCH(kDeliverMany, (unsigned)small.size(), kDeliverThreads, 0,
                  (const DeliverSpec*)(G->specs.p + fillBytes));
      for (ws_executor* X : G->xs)
        if (X->A->nrows() > kSmallRows) queueExecTail(*X);
      capturing = false;
      WS_CK(cudaStreamEndCapture(cs, &G->graph));
      WS_CK(cudaGraphInstantiate(&G->exec, G->graph, 0));
    } catch (...) {
      if (capturing) {
        cudaGraph_t g = nullptr;
        cudaStreamEndCapture(cs, &g);
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
      }
      restore();
      cudaStreamDestroy(cs);
      throw;
    }
    G->kernels = (int)(ws_kernel_launches() - launches0);
    countLaunch(-G->kernels);  // captured, not launched
    restore();
    WS_CK(cudaStreamDestroy(cs));
    *out = G.release();
  });
}

int ws_exec_group_run(ws_exec_group* G, const ws_expr_env* const* envs) {
  return guardedCall([&] {
    if (!envs) throw Error("exec group: no constants", WS_ERR_ARG);
    for (size_t i = 0; i < G->xs.size(); ++i)
      if (!envs[i] || codeDigest(*envs[i]) != G->xs[i]->code)
        throw Error("exec group: query " + std::to_string(i) + "'s expressions differ from its prepared query's",
                    WS_ERR_ARG);
    // the previous run's graph copies `stage` when it runs: wait for it before overwriting
    WS_CK(cudaEventSynchronize(G->done));
    for (size_t j = 0; j < G->mp.live.size(); ++j) {
      Launch L = G->mp.L[j];
      L.env = envK(*envs[(size_t)G->mp.live[j]]);
      memcpy(G->stage + j * sizeof(Launch), &L, sizeof(Launch));
    }
    WS_CK(cudaGraphLaunch(G->exec, stream()));
    WS_CK(cudaEventRecord(G->done, stream()));
    countLaunch(G->kernels);
  });
}

void ws_exec_group_destroy(ws_exec_group* G) { delete G; }

int ws_host_alloc(size_t bytes, void** out) {
  return guardedCall([&] {
    *out = nullptr;
    ws_gpu_init();
    if (cudaHostAlloc(out, std::max<size_t>(bytes, 1), cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      *out = nullptr;
      throw Error("pinned host allocation of " + std::to_string(bytes) + " bytes failed", WS_ERR_OOM);
    }
  });
}

int ws_host_free(void* p) {
  return guardedCall([&] {
    if (p) WS_CK(cudaFreeHost(p));
  });
}

int ws_agg_sum_bits_slots(const ws_aggregator* A, uint8_t* out) {
  for (int a = 0; a < A->plan.naggs; ++a) {
    if (A->plan.nkeys) out[a] = A->plan.aggBits[a];
    else
      out[a] = (A->plan.ops[a] == WS_AGG_SUM || A->plan.ops[a] == WS_AGG_MIN || A->plan.ops[a] == WS_AGG_MAX) && A->plan.aggInt[a];
  }
  return WS_OK;
}

int ws_agg_sum_high(const ws_aggregator* A, int64_t* out) {
  for (int a = 0; a < A->plan.naggs; ++a) out[a] = a < (int)A->hi.size() ? A->hi[a] : 0;
  return WS_OK;
}

int ws_agg_compact(ws_aggregator* A, double** keys, double** accs, int64_t* ngroups) {
  return guardedCall([&] {
    const int nk = A->plan.nkeys, na = A->plan.naggs;
    const ws_fetch_status& st = learnStatus(*A);
    throwFlags(st);
    const int64_t g = st.groups;
    DBuf<double> dk(std::max<int64_t>(g * nk, 1)), da(std::max<int64_t>(g * na, 1));
    if (g && A->groupsOnHost) {
      // a small result again, now into device memory
      WS_LAUNCH(kDeliver, 1, kDeliverThreads, 0,
                DeliverSpec{resultSpec(*A), {nk ? dk.p : nullptr, da.p, nullptr, 0, g, g}, nullptr, 1});
    } else if (g) {
      emitChunks(*A, A->offs.p, OutSpec{nk ? dk.p : nullptr, da.p, nullptr, 0, g, g}, true);
    }
    *keys = dk.release();
    *accs = da.release();
    *ngroups = g;
  });
}

}  // extern "C"
