// srt_raysort.cu -- coherent ray order for traversal (SRT_TRACE_SORT_RAYS).
//
// Rays that start close together and point the same way visit the same
// nodes; a warp of such rays diverges less.  The order is a Morton curve over
// the six ray coordinates (origin and direction), each quantized within the
// rays' own bounding range, with the 30 key bits shared among the
// coordinates that vary (an orthographic view orders by origin, a pinhole
// view by direction, bounce rays by both).  A stable sort of (key, ray
// index) gives the order; traversal reads ray order[k] in thread k and writes
// its hit at the ray's own index, so results do not depend on the order.
#include <algorithm>
#include <climits>

#include "srt_internal.cuh"

namespace srt {
namespace {

__device__ __forceinline__ int ord_f(float f) {  // order-preserving float -> int
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float ord_i(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// box[0..5]: min of o.xyz, d.xyz; box[6..11]: max
__global__ void ray_box_init_kernel(int *__restrict__ box) {
  const int k = threadIdx.x;
  if (k < 12) box[k] = k < 6 ? INT_MAX : INT_MIN;
}

// (these kernels return when *skip is set)
__global__ void ray_box_kernel(const srt_ray *__restrict__ rays, size_t n, int *__restrict__ box,
                               const uint32_t *__restrict__ skip = nullptr) {
  if (skip && *skip) return;
  float lo[6], hi[6];
#pragma unroll
  for (int a = 0; a < 6; a++) {
    lo[a] = FLT_MAX;
    hi[a] = -FLT_MAX;
  }
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const float4 *r4 = reinterpret_cast<const float4 *>(rays + i);
    const float4 a = __ldg(r4), b = __ldg(r4 + 1);
    const float x[6] = {a.x, a.y, a.z, b.x, b.y, b.z};
#pragma unroll
    for (int k = 0; k < 6; k++) {
      lo[k] = fminf(lo[k], x[k]);  // NaN coordinates are ignored
      hi[k] = fmaxf(hi[k], x[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = fminf(lo[k], __shfl_down_sync(0xffffffffu, lo[k], o));
      hi[k] = fmaxf(hi[k], __shfl_down_sync(0xffffffffu, hi[k], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 6; k++) {
      atomicMin(&box[k], ord_f(lo[k]));
      atomicMax(&box[6 + k], ord_f(hi[k]));
    }
  }
}

// The rays' quantization: per coordinate its low end and scale, the
// coordinates that vary (dims[0..nd)) and the bits each gets (30 / nd).
struct RayQuant {
  float lo[6], scale[6];
  int dims[6], nd, bits;
  __device__ __forceinline__ explicit RayQuant(const int *__restrict__ box) {
    nd = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      lo[k] = ord_i(box[k]);
      const float ext = ord_i(box[6 + k]) - lo[k];
      scale[k] = ext > 0.0f ? 1.0f / ext : 0.0f;
      if (ext > 0.0f) dims[nd++] = k;
    }
    bits = nd ? 30 / nd : 0;  // bits per varying coordinate (<= 30 total)
  }
  // Morton code (up to 30 bits) of ray i
  __device__ __forceinline__ uint32_t key(const srt_ray *__restrict__ rays, size_t i) const {
    const float qmax = (float)((1u << bits) - 1u);
    const float4 *r4 = reinterpret_cast<const float4 *>(rays + i);
    const float4 a = __ldg(r4), b = __ldg(r4 + 1);
    const float x[6] = {a.x, a.y, a.z, b.x, b.y, b.z};
    uint32_t q[6];
    for (int c = 0; c < nd; c++) {
      const int k = dims[c];
      // fmaxf(NaN, 0) = 0: NaN coordinates land in cell 0
      const float v = fminf(fmaxf((x[k] - lo[k]) * scale[k] * (qmax + 1.0f), 0.0f), qmax);
      q[c] = (uint32_t)v;
    }
    uint32_t key = 0;
    for (int bit = bits - 1; bit >= 0; bit--)
      for (int c = 0; c < nd; c++) key = (key << 1) | ((q[c] >> bit) & 1u);
    return key;
  }
};

__global__ void ray_key_kernel(const srt_ray *__restrict__ rays, size_t n,
                               const int *__restrict__ box, uint32_t *__restrict__ keys,
                               const uint32_t *__restrict__ skip = nullptr) {
  if (skip && *skip) return;
  const RayQuant Q(box);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    keys[i] = Q.key(rays, i);
}

// Batch keys: the ray's scene above the top mbits of its Morton code, so
// that the order keeps every scene's rays together.
__global__ void batch_ray_key_kernel(const srt_ray *__restrict__ rays, size_t n,
                                     const int *__restrict__ box,
                                     const uint32_t *__restrict__ roff, int nseg, int mbits,
                                     uint32_t *__restrict__ keys) {
  const RayQuant Q(box);
  const int used = Q.nd * Q.bits;  // significant bits of a Morton code
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t m = Q.key(rays, i);
    const uint32_t top = used > mbits ? m >> (used - mbits) : m << (mbits - used);
    keys[i] = ((uint32_t)seg_of(roff, nseg, (uint32_t)i) << mbits) | top;
  }
}

// ---------------------------------------------------------------- rasters
// Ray sets of a camera come row by row.  Taken that way the 32 rays of a
// warp are a 32 x 1 strip and a block's neighbours lie a whole row away; in
// square tiles, each in Z order, both warp and cache see nearby rays:
// 16,777,216 spheres, 2048^2 rays 4.31 -> 2.55 ms, 64^3 x 5 tetrahedra,
// 1024^2 rays 1.37 -> 1.07 ms, 64 triangle scenes 7.65 -> 6.06 ms.  Where
// rays were sorted before (lines, solids) the sort goes, and its key, ten
// bits per direction coordinate, was the worse order: 262,144 hexahedra,
// 512^2 rays 5.50 -> 3.10 ms, 1.6 M lines, 1024^2 2.88 -> 2.60 ms.

// Row length of the rays of segment b (rays roff[b] .. roff[b + 1]; one
// segment of n rays without roff), 0 when they are not rows: the first step
// between consecutive rays eight times longer than those before ends the
// first row, and rows spread over the set must end the same way and lie
// nearer to the row above than a quarter of that step.  Only the order of
// the walks depends on it.  One block per segment, a few microseconds.
constexpr int kProbeThreads = 1024;
constexpr int kProbeItems = 4;
constexpr uint32_t kProbeRows = 16384;  // longest row looked for
constexpr uint32_t kProbeLeast = 64;    // shortest (rays already in small tiles stay so)

__device__ __forceinline__ float ray_gap(const srt_ray *__restrict__ rays, size_t i, size_t j) {
  const float4 *p = reinterpret_cast<const float4 *>(rays + i);
  const float4 *q = reinterpret_cast<const float4 *>(rays + j);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(q), d = __ldg(q + 1);
  // (NaN differences count as none)
  return fmaxf(fmaxf(fmaxf(fabsf(a.x - c.x), fabsf(a.y - c.y)), fabsf(a.z - c.z)),
               fmaxf(fmaxf(fabsf(b.x - d.x), fabsf(b.y - d.y)), fabsf(b.z - d.z)));
}

__global__ void __launch_bounds__(kProbeThreads)
raster_probe_kernel(const srt_ray *__restrict__ rays, size_t n,
                    const uint32_t *__restrict__ roff, uint32_t *__restrict__ width) {
  __shared__ uint32_t s_end, s_bad;
  const size_t first = roff ? roff[blockIdx.x] : 0;
  if (roff) n = roff[blockIdx.x + 1] - first;
  rays += first;
  if (threadIdx.x == 0) {
    s_end = 0xffffffffu;
    s_bad = 0u;
  }
  __syncthreads();
  uint32_t w = 0;
  if (n >= 64) {
    const float step = 8.0f * fmaxf(ray_gap(rays, 0, 1), ray_gap(rays, 1, 2));
    const uint32_t most = (uint32_t)(n - 1 < kProbeRows ? n - 1 : kProbeRows);
    for (uint32_t base = 2; base < most; base += kProbeThreads * kProbeItems) {
#pragma unroll
      for (int q = 0; q < kProbeItems; q++) {
        const uint32_t k = base + q * kProbeThreads + threadIdx.x;
        if (k < most && ray_gap(rays, k, k + 1) > step) atomicMin(&s_end, k + 1);
      }
      __syncthreads();
      const bool found = s_end != 0xffffffffu;
      __syncthreads();  // read by all before the next turn writes it
      if (found) break;
    }
    w = s_end;
    if (w == 0xffffffffu || w < kProbeLeast || n / w < 4) {
      w = 0;
    } else if (threadIdx.x < 64) {
      // rows spread evenly from the second to the last full one
      const size_t rows = n / w;
      const size_t r = 1 + (rows - 1) * (size_t)threadIdx.x / 64;
      const float jump = ray_gap(rays, r * w - 1, r * w);
      const size_t c = threadIdx.x & 1 ? w / 2 : 0;
      if (!(jump > step) || !(ray_gap(rays, (r - 1) * w + c, r * w + c) < 0.25f * jump)) s_bad = 1u;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) width[blockIdx.x] = s_bad ? 0u : w;
}

// The even bits of a number below 2^16, packed: a coordinate of a Z order.
__device__ __forceinline__ uint32_t z_coord(uint32_t v) {
  v &= 0x5555u;
  v = (v | (v >> 1)) & 0x3333u;
  v = (v | (v >> 2)) & 0x0f0fu;
  return (v | (v >> 4)) & 0xffu;
}

// Ray at place k of n rays in rows of w: 32 x 32 tiles row by row, a tile's
// rays in Z order; then the columns right of the tiles, the rows below them
// and the rays of an unfinished row.  (Squares of 8 x 8 tiles in Z order
// measured the same, and 3.10 -> 4.26 ms for hexahedra, whose blocks take
// rays a grid apart.)
__device__ __forceinline__ uint32_t raster_ray(uint32_t k, uint32_t n, uint32_t w) {
  const uint32_t h = n / w, tw = w >> 5, th = h >> 5, core = tw * th * 1024u;
  if (k < core) {
    const uint32_t tile = k >> 10, ty = tile / tw, tx = tile - ty * tw;
    return (ty * 32u + z_coord((k & 1023u) >> 1)) * w + tx * 32u + z_coord(k & 1023u);
  }
  k -= core;
  const uint32_t rw = w & 31u, rh = th * 32u;
  if (k < rw * rh) return (k / rw) * w + tw * 32u + k % rw;
  k -= rw * rh;
  const uint32_t bh = h & 31u;
  if (k < bh * w) return (rh + k % bh) * w + k / bh;
  return h * w + (k - bh * w);
}

// order[k] for rays in rows; the array order otherwise, or (ordered) left as
// it is.  Four places per thread: their segment is looked up once.
__global__ void raster_fill_kernel(size_t n, const uint32_t *__restrict__ roff, int nseg,
                                   const uint32_t *__restrict__ width,
                                   uint32_t *__restrict__ order, bool ordered) {
  for (size_t g0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) * 4; g0 < n;
       g0 += (size_t)gridDim.x * blockDim.x * 4) {
    uint32_t sg = 0, first = 0, end = (uint32_t)n, w = 0, o[4];
    if (!roff) w = __ldg(width);
    if (ordered && !w) return;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t g = (uint32_t)g0 + q;
      if (roff && (q == 0 || g >= end) && g < n) {
        sg = (uint32_t)seg_of(roff, nseg, g);
        first = __ldg(&roff[sg]);
        end = __ldg(&roff[sg + 1]);
        w = __ldg(&width[sg]);
      }
      o[q] = w && g < n ? first + raster_ray(g - first, end - first, w) : g;
    }
    if (g0 + 4 <= n) {
      *reinterpret_cast<uint4 *>(order + g0) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
      for (int q = 0; g0 + q < n; q++) order[g0 + q] = o[q];
    }
  }
}

}  // namespace

static srt_status find_rows(srt_ctx *ctx, const srt_ray *rays, size_t n, const uint32_t *roff,
                            int nseg, uint32_t *width, uint32_t *order) {
  if (n == 0) return SRT_OK;
  raster_probe_kernel<<<(unsigned)nseg, kProbeThreads, 0, ctx->stream>>>(rays, n, roff, width);
  const unsigned grid = (unsigned)std::min<size_t>((n + 1023) / 1024, (size_t)ctx->num_sms * 8);
  raster_fill_kernel<<<grid, 256, 0, ctx->stream>>>(n, roff, nseg, width, order, false);
  ctx->launches += 2;
  return cuda_status(cudaGetLastError(), "ray rows");
}

srt_status raster_order(srt_ctx *ctx, const srt_ray *rays, size_t n, const uint32_t **order) {
  *order = nullptr;
  if (ctx->s_rorder.ensure(n * 4) != cudaSuccess ||
      ctx->s_raster.ensure(4) != cudaSuccess)
    return SRT_OK;  // array order does as well
  *order = ctx->s_rorder.as<uint32_t>();
  return find_rows(ctx, rays, n, nullptr, 1, ctx->s_raster.as<uint32_t>(),
                   ctx->s_rorder.as<uint32_t>());
}

srt_status batch_raster_order(srt_ctx *ctx, const srt_ray *rays, size_t n, const uint32_t *roff,
                              int nseg, uint32_t *width, uint32_t *order) {
  return find_rows(ctx, rays, n, roff, nseg, width, order);
}

srt_status batch_ray_order(srt_ctx *ctx, const srt_ray *rays, size_t n, const uint32_t *roff,
                           int nseg, int mbits, uint32_t *keys, uint32_t *order) {
  int segbits = 0;
  while ((1 << segbits) < nseg) segbits++;
  if (mbits < 1 || segbits + mbits > 30) {
    set_error("ray order: scene and Morton bits exceed 30");
    return SRT_ERR_INVALID;
  }
  int *box = reinterpret_cast<int *>(keys + n);  // 12 ints after the keys
  cudaStream_t st = ctx->stream;
  const int grid = ctx->num_sms * 4;
  ray_box_init_kernel<<<1, 32, 0, st>>>(box);
  ray_box_kernel<<<grid, 256, 0, st>>>(rays, n, box);
  batch_ray_key_kernel<<<grid, 256, 0, st>>>(rays, n, box, roff, nseg, mbits, keys);
  ctx->launches += 3;
  srt_status s = cuda_status(cudaGetLastError(), "batch ray keys");
  if (s != SRT_OK) return s;
  return sort_pairs(ctx, keys, order, n, true, segbits + mbits);
}

srt_status ray_order(srt_ctx *ctx, const srt_ray *rays, size_t n, const uint32_t **order) {
  cudaError_t e;
  if ((e = ctx->s_rkey.ensure(n * 4 + 64)) != cudaSuccess ||
      (e = ctx->s_rorder.ensure(n * 4)) != cudaSuccess ||
      (e = ctx->s_raster.ensure(4)) != cudaSuccess)
    return cuda_status(e, "ray order scratch");
  uint32_t *keys = ctx->s_rkey.as<uint32_t>();
  int *box = reinterpret_cast<int *>(keys + n);  // 12 ints after the keys
  uint32_t *ord = ctx->s_rorder.as<uint32_t>();
  // Rays in rows need no sort: its kernels then return at once.  Few rays are
  // sorted without a look (1,000 rays and 70,000 tetrahedra: 312 us, with it 318).
  const bool look = n >= ((size_t)1 << 15);
  uint32_t *width = look ? ctx->s_raster.as<uint32_t>() : nullptr;
  cudaStream_t st = ctx->stream;
  const int grid = ctx->num_sms * 4;
  if (look) {
    raster_probe_kernel<<<1, kProbeThreads, 0, st>>>(rays, n, nullptr, width);
    ctx->launches++;
  }
  ray_box_init_kernel<<<1, 32, 0, st>>>(box);
  ray_box_kernel<<<grid, 256, 0, st>>>(rays, n, box, width);
  ray_key_kernel<<<grid, 256, 0, st>>>(rays, n, box, keys, width);
  ctx->launches += 3;
  srt_status s = cuda_status(cudaGetLastError(), "ray keys");
  if (s != SRT_OK) return s;
  if ((s = sort_pairs(ctx, keys, ord, n, true, 30, width)) != SRT_OK) return s;
  if (look) {
    raster_fill_kernel<<<grid, 256, 0, st>>>(n, nullptr, 1, width, ord, true);
    ctx->launches++;
  }
  *order = ord;
  return cuda_status(cudaGetLastError(), "ray order");
}

}  // namespace srt
