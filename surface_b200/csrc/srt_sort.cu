// srt_sort.cu -- stable sort of (Morton code, index) pairs.
//
// The order is the reference's: ascending 30-bit code, ties in input order
// (RadixSort30OMP, render/render_prefix_tree_util.h:296-402, is a stable LSD
// sort whose keys start as index = i).  Both sorts here are one-sweep radix
// sorts (Adinets and Merrill, 2022; the look-back is Merrill and Garland's,
// 2016): one kernel per LSD pass instead of a count, a scan and a scatter.
// sort_codes30, up to 2^18 codes, takes three passes of 10 bits; its digit
// counts come from the build's Morton kernel.
//
//   os_pass_kernel   per pass, tiles of 1,024 keys in tile order (tile ids from
//                    a ticket counter, so a tile only waits on tiles that are
//                    already running): rank every key within its tile (warps
//                    own consecutive chunks, one ballot per digit bit ranks
//                    lanes in order), publish the tile's digit counts, add the
//                    counts of earlier tiles (look-back over their published
//                    aggregates / inclusive prefixes), stage the tile in shared
//                    memory in (digit, input) order and write it out in runs of
//                    equal digits.
//
// sort_codes30_large (below) takes longer tiles and shorter digits.
//
// Look-back words are 64 bits: the pass's epoch (a per-context counter, so
// the status array is never cleared between passes) and a 32-bit value
// (flag in bits 30-31: aggregate or inclusive prefix; count in bits 0-29).
// Every wait is bounded: a tile that waits longer than kSpinLimit polls sets
// the context's error flag and gives up (SRT_ERR_LIMIT), it never hangs.
#include <algorithm>

#include "srt_internal.cuh"

namespace srt {
namespace {

constexpr int kOsBits = 10;
constexpr int kOsBins = 1 << kOsBits;
constexpr int kOsWarps = 8;
constexpr int kOsThreads = kOsWarps * 32;
constexpr int kOsPerThread = kOsBins / kOsThreads;  // 4 bins per thread
constexpr int kOsRounds = 4;  // keys per thread: short tiles keep every SM busy
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kCountMask30 = (1u << 30) - 1u;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr uint32_t kErrSort = kErrSortWait;

// Exclusive scan of kOsBins values held 4 per thread (bins 4t..4t+3), in
// place; returns the total.  Uses `tmp` (kOsWarps words) of shared memory.
__device__ __forceinline__ uint32_t block_scan4(uint32_t x[kOsPerThread], uint32_t *tmp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t s = 0;
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) {
    const uint32_t t = x[q];
    x[q] = s;
    s += t;
  }
  uint32_t inc = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) tmp[w] = inc;
  __syncthreads();
  uint32_t wbase = 0, total = 0;
#pragma unroll
  for (int k = 0; k < kOsWarps; k++) {
    const uint32_t v = tmp[k];
    if (k < w) wbase += v;
    total += v;
  }
  const uint32_t base = wbase + inc - s;
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) x[q] += base;
  __syncthreads();
  return total;
}

__device__ __forceinline__ unsigned long long ld_status(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_status(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_word(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(uint32_t *p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Shared memory of one pass block (dynamic): per-warp digit counts, then the
// staged tile.
struct PassSmem {
  static constexpr int kTile = kOsThreads * kOsRounds;
  uint32_t wc[kOsWarps][kOsBins];  // counts, then exclusive offsets per warp
  uint32_t tloc[kOsBins];          // tile-local start of each digit
  uint32_t gdst[kOsBins];          // global position of tile slot 0 per digit
  uint32_t tmp[kOsWarps];
  uint32_t tile;
  uint32_t key[kTile];
  uint32_t val[kTile];
};

__global__ void __launch_bounds__(kOsThreads)
os_pass_kernel(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
               uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, uint32_t n, int shift,
               const uint32_t *__restrict__ ghist, unsigned long long *__restrict__ status,
               unsigned long long *__restrict__ ticket, uint32_t epoch,
               uint32_t *__restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PassSmem &S = *reinterpret_cast<PassSmem *>(smem_raw);
  constexpr int ROUNDS = kOsRounds, kTile = PassSmem::kTile;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) S.tile = (uint32_t)atomicAdd(ticket, 1ull);
  for (int i = threadIdx.x; i < kOsWarps * kOsBins; i += kOsThreads) (&S.wc[0][0])[i] = 0;
  __syncthreads();
  const uint32_t tile = S.tile;
  if (tile >= gridDim.x) {  // a counter left over from a failed launch
    if (threadIdx.x == 0) atomicOr(err, kErrSort);
    return;
  }
  const uint32_t base = tile * (uint32_t)kTile + (uint32_t)w * (32u * ROUNDS);

  // load, digits, in-warp ranks (peers: lanes of the round with this digit)
  uint32_t k[ROUNDS], v[ROUNDS], dg[ROUNDS], rk[ROUNDS];
  bool ok[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const uint32_t idx = base + (uint32_t)r * 32u + (uint32_t)lane;
    ok[r] = idx < n;
    k[r] = ok[r] ? kin[idx] : 0u;
    v[r] = ok[r] ? (vin ? vin[idx] : idx) : 0u;
  }
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    unsigned pm = __ballot_sync(0xffffffffu, ok[r]);
    const uint32_t d = (k[r] >> shift) & (kOsBins - 1);
#pragma unroll
    for (int b = 0; b < kOsBits; b++) {
      const bool bit = (d >> b) & 1u;
      const unsigned m = __ballot_sync(0xffffffffu, bit);
      pm &= bit ? m : ~m;
    }
    dg[r] = d;
    // rank among this warp's earlier keys of the same digit
    uint32_t before = 0;
    if (ok[r]) before = S.wc[w][d];
    __syncwarp();
    rk[r] = before + (uint32_t)__popc(pm & lt);
    if (ok[r] && lane == __ffs(pm) - 1) S.wc[w][d] = before + (uint32_t)__popc(pm);
    __syncwarp();
  }
  __syncthreads();

  // tile counts; per-warp exclusive offsets within each digit
  uint32_t c[kOsPerThread];
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) {
    const int d = kOsPerThread * threadIdx.x + q;
    uint32_t run = 0;
#pragma unroll
    for (int ww = 0; ww < kOsWarps; ww++) {
      const uint32_t t = S.wc[ww][d];
      S.wc[ww][d] = run;
      run += t;
    }
    c[q] = run;
  }
  // publish this tile's counts before anything else, so later tiles can go on
  unsigned long long *st = status + (size_t)tile * kOsBins;
  const unsigned long long ep = (unsigned long long)epoch << 32;
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) {
    const int d = kOsPerThread * threadIdx.x + q;
    st_status(&st[d], ep | (tile == 0 ? kFlagInc : kFlagAgg) | c[q]);
  }
  // global digit starts (exclusive scan of this pass's histogram)
  uint32_t g[kOsPerThread];
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) g[q] = __ldg(&ghist[kOsPerThread * threadIdx.x + q]);
  block_scan4(g, S.tmp);
  // tile-local digit starts
  uint32_t tl[kOsPerThread];
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) tl[q] = c[q];
  block_scan4(tl, S.tmp);
  // look-back: keys of each digit in earlier tiles.  The thread's four bins
  // walk back together, kWin predecessor words per bin per round, all loads
  // of a round in flight at once; a window is consumed up to its nearest
  // inclusive prefix, or retried while a word in it is not yet published.
  constexpr int kWin = 4;
  bool failed = false;
  uint32_t prefix[kOsPerThread];
  int jnext[kOsPerThread];  // next predecessor to read, -1: done
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) {
    prefix[q] = 0;
    jnext[q] = (int)tile - 1;
  }
  uint32_t spins = 0;
  while (true) {
    bool pending = false;
#pragma unroll
    for (int q = 0; q < kOsPerThread; q++) pending |= jnext[q] >= 0;
    if (!pending) break;
    unsigned long long wv[kOsPerThread][kWin];
#pragma unroll
    for (int q = 0; q < kOsPerThread; q++) {
      const int d = kOsPerThread * threadIdx.x + q;
#pragma unroll
      for (int w = 0; w < kWin; w++) {
        const int j = jnext[q] - w;
        wv[q][w] = j >= 0 ? ld_status(&status[(size_t)j * kOsBins + d])
                          : (((unsigned long long)epoch << 32) | kFlagInc);  // tile -1: 0
      }
    }
    bool stalled = false;
#pragma unroll
    for (int q = 0; q < kOsPerThread; q++) {
      if (jnext[q] < 0) continue;
      uint32_t add = 0;
      int consumed = 0;
      bool fin = false, wait = false;
#pragma unroll
      for (int w = 0; w < kWin; w++) {
        if (fin || wait) continue;
        if ((uint32_t)(wv[q][w] >> 32) != epoch) {
          wait = true;
          continue;
        }
        const uint32_t x = (uint32_t)wv[q][w];
        add += x & kCountMask30;
        consumed = w + 1;
        if (x & kFlagInc) fin = true;
      }
      prefix[q] += add;
      jnext[q] = fin ? -1 : jnext[q] - consumed;
      stalled |= wait && consumed == 0;
    }
    if (stalled) {
      if (++spins > kSpinLimit) {
        failed = true;
        break;
      }
      __nanosleep(64);
    }
  }
#pragma unroll
  for (int q = 0; q < kOsPerThread; q++) {
    const int d = kOsPerThread * threadIdx.x + q;
    if (tile > 0) st_status(&st[d], ep | kFlagInc | ((prefix[q] + c[q]) & kCountMask30));
    S.tloc[d] = tl[q];
    S.gdst[d] = g[q] + prefix[q] - tl[q];
  }
  if (failed) atomicOr(err, kErrSort);
  __syncthreads();

  // stage the tile in (digit, input) order
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    if (!ok[r]) continue;
    const uint32_t d = dg[r];
    const uint32_t pos = S.tloc[d] + S.wc[w][d] + rk[r];
    S.key[pos] = k[r];
    S.val[pos] = v[r];
  }
  __syncthreads();
  // write out: consecutive slots of one digit go to consecutive addresses
  const uint32_t cnt = min((uint32_t)kTile, n - tile * (uint32_t)kTile);
  for (uint32_t j = threadIdx.x; j < cnt; j += kOsThreads) {
    const uint32_t kk = S.key[j];
    const uint32_t d = (kk >> shift) & (kOsBins - 1);
    const uint32_t gp = S.gdst[d] + j;
    if (gp < n) {  // holds unless a look-back gave up (error flag set)
      kout[gp] = kk;
      vout[gp] = S.val[j];
    }
  }
}

// ------------------------------------------------------------ large arrays
// What counts above some 10^5 keys is how the keys leave a pass: a tile of
// 4,096 keys in 1,024 digits writes runs of 4 keys, half of every 32-byte
// sector wasted, and its 8 KB of look-back words are an eighth of its traffic.
// Here digits have 8 bits and tiles 8,192 keys: runs of 32 keys, 1 KB of
// words, four passes of 16 bytes a key.  A pass is bound by its tiles' chains
// (ranks, look-back), so long tiles in two blocks per SM do best, a shared
// word per digit finds the lanes that share one (8 votes: 162 instructions
// per 32 keys, 40 % more time), and a tile is staged before the look-back to
// free its registers.  16.8 M codes: 1,085 us (histogram, scan and scatter per
// 10-bit pass) -> 578; 1 M: 113 -> 62; 9.4 M in 64 scenes: 783 -> 440.  (Tiles
// of 4,096 and 6,144 keys: 927 and 665 us; windows of 32 and 64 words in the
// look-back: no gain.)
constexpr int kLgBits = 8;
constexpr int kLgBins = 1 << kLgBits;
constexpr int kLgWarps = 16;
constexpr int kLgThreads = kLgWarps * 32;
constexpr int kLgRounds = 16;
constexpr int kLgTile = kLgThreads * kLgRounds;
constexpr int kLgPasses = 4;  // digits of 8, 8, 8 and 6 bits: 30

// Counts of every digit of the passes.
__global__ void __launch_bounds__(kLgThreads)
lg_hist_kernel(const uint32_t *__restrict__ keys, size_t n, uint32_t *__restrict__ ghist,
               const uint32_t *__restrict__ skip) {
  if (skip && *skip) return;
  __shared__ uint32_t h[2][kLgPasses][kLgBins];  // (two copies: half the conflicts)
  for (int i = threadIdx.x; i < 2 * kLgPasses * kLgBins; i += kLgThreads) (&h[0][0][0])[i] = 0;
  __syncthreads();
  const size_t stride = (size_t)gridDim.x * kLgThreads * 4;
  uint32_t(*mine)[kLgBins] = h[threadIdx.x & 1];
  for (size_t i = ((size_t)blockIdx.x * kLgThreads + threadIdx.x) * 4; i < n; i += stride) {
    uint32_t k[4];
    const int cnt = n - i < 4 ? (int)(n - i) : 4;
    if (cnt == 4) {
      const uint4 q = __ldg(reinterpret_cast<const uint4 *>(keys + i));
      k[0] = q.x; k[1] = q.y; k[2] = q.z; k[3] = q.w;
    } else {
      for (int q = 0; q < cnt; q++) k[q] = __ldg(&keys[i + q]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q < cnt) {
#pragma unroll
        for (int p = 0; p < kLgPasses; p++)
          atomicAdd(&mine[p][(k[q] >> (kLgBits * p)) & (kLgBins - 1)], 1u);
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kLgPasses * kLgBins; i += kLgThreads) {
    const uint32_t c = (&h[0][0][0])[i] + (&h[1][0][0])[i];
    if (c) atomicAdd(&ghist[i], c);
  }
}

struct LgSmem {
  uint32_t wc[kLgWarps][kLgBins];  // per-warp digit counts, then offsets
  uint32_t tloc[kLgBins];          // tile-local start of each digit
  uint32_t gdst[kLgBins];          // global position of tile slot 0 per digit
  uint32_t tmp[kLgWarps];
  uint32_t tile;
  union {  // match: zero between rounds; the tile follows when ranks are known
    uint32_t match[kLgWarps][kLgBins];
    struct {
      uint32_t key[kLgTile], val[kLgTile];
      uint8_t dig[kLgTile];
    };
  };
};

// Exclusive scan of one value per bin, held by the first kLgBins threads.
__device__ __forceinline__ uint32_t lg_scan(uint32_t x, uint32_t *tmp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) tmp[w] = inc;
  __syncthreads();
  uint32_t base = 0;
#pragma unroll
  for (int k = 0; k < kLgBins / 32; k++)
    if (k < w) base += tmp[k];
  __syncthreads();
  return base + inc - x;
}

// One stable pass (as os_pass_kernel): the digit at `shift`, or (SEG) the
// segment of the value, whose counts are the differences of the offsets seg.
template <bool SEG>
__global__ void __launch_bounds__(kLgThreads, 2)
lg_pass_kernel(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
               uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, uint32_t n, int shift,
               const uint32_t *__restrict__ ghist, const uint32_t *__restrict__ seg, int nseg,
               uint32_t *__restrict__ status, unsigned long long *__restrict__ ticket,
               uint32_t *__restrict__ err, const uint32_t *__restrict__ skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  LgSmem &S = *reinterpret_cast<LgSmem *>(smem_raw);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) S.tile = (uint32_t)atomicAdd(ticket, 1ull);
  for (int i = threadIdx.x; i < kLgWarps * kLgBins; i += kLgThreads) {
    (&S.wc[0][0])[i] = 0;
    (&S.match[0][0])[i] = 0;
  }
  __syncthreads();
  const uint32_t tile = S.tile;
  if (tile >= gridDim.x) {  // a counter left over from a failed launch
    if (threadIdx.x == 0) atomicOr(err, kErrSort);
    return;
  }
  const uint32_t first = tile * (uint32_t)kLgTile;
  const uint32_t base = first + (uint32_t)w * (32u * kLgRounds) + (uint32_t)lane;
  uint32_t k[kLgRounds], v[kLgRounds], rk[kLgRounds];  // rk: rank | digit << 16
#pragma unroll
  for (int r = 0; r < kLgRounds; r++) {
    const uint32_t idx = base + (uint32_t)r * 32u;
    k[r] = idx < n ? __ldg(&kin[idx]) : 0u;
    v[r] = idx < n ? (vin ? __ldg(&vin[idx]) : idx) : 0u;
  }
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < kLgRounds; r++) {
    const bool ok = base + (uint32_t)r * 32u < n;
    uint32_t d = (k[r] >> shift) & (kLgBins - 1);
    if (SEG) d = ok ? (uint32_t)seg_of(seg, nseg, v[r]) : 0u;
    // lanes of this round with the digit, through a shared word per digit
    if (ok) atomicOr(&S.match[w][d], 1u << lane);
    __syncwarp();
    // rank among this warp's earlier keys of the same digit
    unsigned pm = 0;
    uint32_t before = 0;
    if (ok) {
      pm = S.match[w][d];
      before = S.wc[w][d];
    }
    __syncwarp();
    rk[r] = (before + (uint32_t)__popc(pm & lt)) | d << 16;
    if (ok && (pm & lt) == 0) {  // the first of them
      S.match[w][d] = 0u;
      S.wc[w][d] = before + (uint32_t)__popc(pm);
    }
    __syncwarp();
  }
  __syncthreads();
  // a thread per digit: tile count, per-warp offsets, published at once
  const uint32_t d = threadIdx.x;
  uint32_t cnt = 0, g = 0;
  if (d < kLgBins) {
#pragma unroll
    for (int q = 0; q < kLgWarps; q++) {
      const uint32_t t = S.wc[q][d];
      S.wc[q][d] = cnt;
      cnt += t;
    }
    st_word(&status[(size_t)tile * kLgBins + d], (tile == 0 ? kFlagInc : kFlagAgg) | cnt);
    g = SEG ? (d < (uint32_t)nseg ? __ldg(&seg[d + 1]) - __ldg(&seg[d]) : 0u) : __ldg(&ghist[d]);
  }
  g = lg_scan(g, S.tmp);
  const uint32_t tl = lg_scan(cnt, S.tmp);
  if (d < kLgBins) S.tloc[d] = tl;
  __syncthreads();
  // stage the tile in (digit, input) order: its registers are free for the
  // look-back
#pragma unroll
  for (int r = 0; r < kLgRounds; r++) {
    if (base + (uint32_t)r * 32u >= n) continue;
    const uint32_t dd = rk[r] >> 16;
    const uint32_t pos = S.tloc[dd] + S.wc[w][dd] + (rk[r] & 0xffffu);
    S.key[pos] = k[r];
    S.val[pos] = v[r];
    S.dig[pos] = (uint8_t)dd;
  }
  if (d < kLgBins) {
    // look-back: some hundred tiles are under way, so the words of many
    // predecessors are read at once
    constexpr int kWin = 16;
    uint32_t prefix = 0, spins = 0;
    int j = (int)tile - 1;
    bool failed = false;
    while (j >= 0) {
      uint32_t x[kWin];
#pragma unroll
      for (int q = 0; q < kWin; q++)
        x[q] = j - q >= 0 ? ld_word(&status[(size_t)(j - q) * kLgBins + d]) : kFlagInc;
      int used = 0;
      bool fin = false, wait = false;
#pragma unroll
      for (int q = 0; q < kWin; q++) {
        if (fin || wait) continue;
        if (x[q] == 0u) {  // not published
          wait = true;
          continue;
        }
        prefix += x[q] & kCountMask30;
        used = q + 1;
        if (x[q] & kFlagInc) fin = true;
      }
      j = fin ? -1 : j - used;
      if (wait && used == 0) {
        if (++spins > kSpinLimit) {
          failed = true;
          break;
        }
        __nanosleep(32);
      }
    }
    if (tile > 0)
      st_word(&status[(size_t)tile * kLgBins + d], kFlagInc | ((prefix + cnt) & kCountMask30));
    S.gdst[d] = g + prefix - tl;
    if (failed) atomicOr(err, kErrSort);
  }
  __syncthreads();
  // write it out in runs of a digit
  const uint32_t mine = min((uint32_t)kLgTile, n - first);
  for (uint32_t j = threadIdx.x; j < mine; j += kLgThreads) {
    const uint32_t gp = S.gdst[S.dig[j]] + j;
    if (gp < n) {  // holds unless a look-back gave up (error flag set)
      kout[gp] = S.key[j];
      vout[gp] = S.val[j];
    }
  }
}

}  // namespace

srt_status sort_codes30_large(srt_ctx *ctx, uint32_t *keys, uint32_t *vals, size_t n,
                              bool identity_vals, const uint32_t *seg, int nseg,
                              const uint32_t *skip) {
  const uint32_t ntiles = (uint32_t)((n + kLgTile - 1) / kLgTile);
  const bool by_seg = nseg > 1;
  cudaStream_t st = ctx->stream;
  cudaError_t e;
  if ((e = ctx->s_keys2.ensure(n * 4)) != cudaSuccess ||
      (e = ctx->s_vals2.ensure(n * 4)) != cudaSuccess ||
      (by_seg && (e = ctx->s_keys3.ensure(n * 4)) != cudaSuccess) ||
      (by_seg && (e = ctx->s_vals3.ensure(n * 4)) != cudaSuccess))
    return cuda_status(e, "sort");
  // tile counters, digit counts and each pass's look-back words (0: not
  // published), zeroed by every sort
  constexpr size_t kHead = 256 + kLgPasses * kLgBins * 4;
  const int passes = kLgPasses + (by_seg ? 1 : 0);
  const size_t sbytes = kHead + (size_t)passes * ntiles * kLgBins * 4;
  if ((e = ctx->s_status_lg.ensure(sbytes)) != cudaSuccess ||
      (e = cudaMemsetAsync(ctx->s_status_lg.p, 0, sbytes, st)) != cudaSuccess)
    return cuda_status(e, "sort");
  static bool attr_set[64] = {};
  if (ctx->device >= 0 && ctx->device < 64 && !attr_set[ctx->device]) {
    for (const void *fn : {(const void *)lg_pass_kernel<false>, (const void *)lg_pass_kernel<true>})
      if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(LgSmem))) != cudaSuccess)
        return cuda_status(e, "sort pass attributes");
    attr_set[ctx->device] = true;
  }
  unsigned long long *tickets = ctx->s_status_lg.as<unsigned long long>();
  uint32_t *ghist = reinterpret_cast<uint32_t *>(tickets + 32);
  uint32_t *status = ghist + kLgPasses * kLgBins;
  const int hgrid = (int)std::min<size_t>((n + 8191) / 8192, (size_t)ctx->num_sms * 4);
  lg_hist_kernel<<<hgrid, kLgThreads, 0, st>>>(keys, n, ghist, skip);
  ctx->launches++;
  // four passes go to and fro; a fifth (segments) takes a third buffer
  uint32_t *kb[3] = {keys, ctx->s_keys2.as<uint32_t>(), ctx->s_keys3.as<uint32_t>()};
  uint32_t *vb[3] = {vals, ctx->s_vals2.as<uint32_t>(), ctx->s_vals3.as<uint32_t>()};
  static const int even[] = {0, 1, 0, 1, 0}, odd[] = {0, 1, 2, 1, 2, 0};
  const int *way = by_seg ? odd : even;
  for (int p = 0; p < passes; p++) {
    const uint32_t *vin = (p == 0 && identity_vals) ? nullptr : vb[way[p]];
    const auto kern = p < kLgPasses ? lg_pass_kernel<false> : lg_pass_kernel<true>;
    kern<<<ntiles, kLgThreads, sizeof(LgSmem), st>>>(
        kb[way[p]], vin, kb[way[p + 1]], vb[way[p + 1]], (uint32_t)n,
        p < kLgPasses ? kLgBits * p : 0, ghist + kLgBins * (p % kLgPasses), seg, nseg, status + (size_t)p * ntiles * kLgBins, tickets + p,
        ctx->d_err, skip);
    ctx->launches++;
  }
  return cuda_status(cudaGetLastError(), "sort passes");
}

// Scratch of sort_codes30 for n keys: ping-pong buffers, the digit
// histograms (3 x 1024 words) and the look-back words behind a 256-byte
// header whose first three 64-bit words are the passes' tile counters.
srt_status sort_codes30_scratch(srt_ctx *ctx, size_t n, uint32_t **hist,
                                unsigned long long **tickets) {
  cudaError_t e;
  if ((e = ctx->s_keys2.ensure(n * 4)) != cudaSuccess) return cuda_status(e, "sort");
  if ((e = ctx->s_vals2.ensure(n * 4)) != cudaSuccess) return cuda_status(e, "sort");
  if ((e = ctx->s_keys3.ensure(n * 4)) != cudaSuccess) return cuda_status(e, "sort");
  if ((e = ctx->s_vals3.ensure(n * 4)) != cudaSuccess) return cuda_status(e, "sort");
  if ((e = ctx->s_hist.ensure(3 * kOsBins * 4)) != cudaSuccess) return cuda_status(e, "sort");
  const size_t ntiles = (n + kOsThreads * 4 - 1) / (kOsThreads * 4);  // the smallest tiles
  const size_t sbytes = 256 + ntiles * kOsBins * 8;
  if (sbytes > ctx->s_status.cap || !ctx->s_status.p) {
    // fresh words: epoch 0 never matches a pass
    if ((e = ctx->s_status.ensure(sbytes)) != cudaSuccess) return cuda_status(e, "sort");
    if ((e = cudaMemsetAsync(ctx->s_status.p, 0, ctx->s_status.cap, ctx->stream)) !=
        cudaSuccess)
      return cuda_status(e, "sort");
  }
  *hist = ctx->s_hist.as<uint32_t>();
  *tickets = ctx->s_status.as<unsigned long long>();
  return SRT_OK;
}

// Stable sort of (30-bit code, value) pairs by code, in place.  identity_vals:
// the values are 0..n-1 on entry (not read).  The digit histograms of the three
// passes are already in the scratch and the tile counters zeroed (the Morton
// kernel of a build does both).
srt_status sort_codes30(srt_ctx *ctx, uint32_t *keys, uint32_t *vals, size_t n,
                        bool identity_vals) {
  if (n == 0) return SRT_OK;
  if (n >= (1u << 30)) {
    set_error("sort: at most 2^30 - 1 keys");
    return SRT_ERR_INVALID;
  }
  const uint32_t ntiles = (uint32_t)((n + PassSmem::kTile - 1) / PassSmem::kTile);
  const size_t smem = sizeof(PassSmem);
  static bool attr_set[64] = {};
  if (ctx->device >= 0 && ctx->device < 64 && !attr_set[ctx->device]) {
    cudaError_t e = cudaFuncSetAttribute(os_pass_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return cuda_status(e, "sort pass attributes");
    attr_set[ctx->device] = true;
  }
  uint32_t *ghist = nullptr;
  unsigned long long *tickets = nullptr;
  srt_status s = sort_codes30_scratch(ctx, n, &ghist, &tickets);
  if (s != SRT_OK) return s;
  unsigned long long *status = tickets + 32;  // after the 256-byte header
  // keys -> 2 -> 3 -> keys: three passes end where they started
  uint32_t *ksrc[3] = {keys, ctx->s_keys2.as<uint32_t>(), ctx->s_keys3.as<uint32_t>()};
  uint32_t *vsrc[3] = {vals, ctx->s_vals2.as<uint32_t>(), ctx->s_vals3.as<uint32_t>()};
  for (int p = 0; p < 3; p++) {
    const uint32_t epoch = ++ctx->os_epoch == 0 ? ++ctx->os_epoch : ctx->os_epoch;
    const uint32_t *vin = (p == 0 && identity_vals) ? nullptr : vsrc[p];
    os_pass_kernel<<<ntiles, kOsThreads, smem, ctx->stream>>>(
        ksrc[p], vin, ksrc[(p + 1) % 3], vsrc[(p + 1) % 3], (uint32_t)n, kOsBits * p,
        ghist + kOsBins * p, status, tickets + p, epoch, ctx->d_err);
    ctx->launches++;
  }
  return cuda_status(cudaGetLastError(), "sort passes");
}

}  // namespace srt
