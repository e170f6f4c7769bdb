// k-nearest-neighbour scale initialisation: knn_init (knn-init.wgsl:40-90,
// dispatched by initializeKnn, gaussian-renderer.ts:2131-2171) without its
// O(N^2) scan.  Points (positions read through f16, as the reference's
// packed buffer holds them) are binned into a uniform grid and sorted by
// cell; each point then searches its own cell, the rows of cells around it,
// and shells of growing Chebyshev radius r until its third-smallest distance
// is below the distance to any unvisited cell, (r - 0.001) h: cell assignment
// in f32 places a point at most 2.4e-4 cells from its true cell, so no
// unvisited point can be closer.  The three smallest distances are the ones
// the brute-force scan finds (the insertion keeps values; ties do not
// reorder them), so the result is bit-identical to it.
#include <cstring>

#include "chain.cuh"
#include "knn.cuh"
#include "sky_math.cuh"

namespace sky {
namespace {

SKY_DEV uint32_t enc(float f) {  // order-preserving float -> u32
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

SKY_DEV float pos16(const float* P, uint32_t stride, int k, uint32_t i) {
  return round_f16(P[(size_t)k * stride + i]);
}

__global__ void __launch_bounds__(256)
k_knn_bounds(const float* __restrict__ P, uint32_t stride, uint32_t n, uint32_t* __restrict__ out) {
  uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) {
      const float v = pos16(P, stride, k, i);
      if (v != v) continue;
      const uint32_t e = enc(v);
      mn[k] = min(mn[k], e);
      mx[k] = max(mx[k], e);
    }
  // one atomic per block and bound (one per warp serialised on the six words)
  __shared__ uint32_t s_mn[3][8], s_mx[3][8];
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
  for (int k = 0; k < 3; ++k) {
    const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, mn[k]), hi = __reduce_max_sync(0xFFFFFFFFu, mx[k]);
    if (lane == 0) {
      s_mn[k][warp] = lo;
      s_mx[k][warp] = hi;
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    uint32_t lo = 0xFFFFFFFFu, hi = 0u;
    for (int w = 0; w < 8; ++w) {
      lo = min(lo, s_mn[threadIdx.x][w]);
      hi = max(hi, s_mx[threadIdx.x][w]);
    }
    atomicMin(&out[threadIdx.x], lo);
    atomicMax(&out[3 + threadIdx.x], hi);
  }
}

SKY_DEV uint32_t cell_of(float v, float lo, float h, uint32_t dim) {
  const float q = (v - lo) / h;
  if (!(q > 0.0f)) return 0u;
  const float c = floorf(q);
  return c >= (float)(dim - 1) ? dim - 1 : (uint32_t)c;
}

__global__ void __launch_bounds__(256)
k_knn_keys(const float* __restrict__ P, uint32_t stride, uint32_t n, KnnGrid g,
           uint32_t* __restrict__ keys) {
  chain_wait(P, keys);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t cx = cell_of(pos16(P, stride, 0, i), g.lo[0], g.h, g.dims[0]);
  const uint32_t cy = cell_of(pos16(P, stride, 1, i), g.lo[1], g.h, g.dims[1]);
  const uint32_t cz = cell_of(pos16(P, stride, 2, i), g.lo[2], g.h, g.dims[2]);
  keys[i] = (cz * g.dims[1] + cy) * g.dims[0] + cx;
}

__global__ void k_knn_cell_ranges(const uint32_t* __restrict__ keys, uint32_t n, uint32_t cells,
                                  uint32_t* __restrict__ start) {
  chain_wait(keys, start);
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > cells) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (keys[mid] < c) lo = mid + 1;
    else hi = mid;
  }
  start[c] = lo;
}

// The points in cell order: position and, as bits, the point's index.
__global__ void __launch_bounds__(256)
k_knn_gather(const float* __restrict__ P, uint32_t stride, uint32_t n,
             const uint32_t* __restrict__ order, float4* __restrict__ pos) {
  chain_wait(P, order, pos);
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t i = order[k];
  pos[k] = make_float4(pos16(P, stride, 0, i), pos16(P, stride, 1, i), pos16(P, stride, 2, i),
                       __uint_as_float(i));
}

SKY_DEV void insert3(float d[3], float v) {  // insert_sorted (knn-init.wgsl:27-38)
  if (v < d[0]) {
    d[2] = d[1];
    d[1] = d[0];
    d[0] = v;
  } else if (v < d[1]) {
    d[2] = d[1];
    d[1] = v;
  } else if (v < d[2]) {
    d[2] = v;
  }
}

// One thread per point, in cell order, so a warp's searches share cells.  The
// candidates are read as 16-byte records in cell order: the cells of a row
// are neighbours there, so three of them are one range.  Squared distances
// are kept (the square root is monotone, and sqrt(1e20f) is the scan's initial
// 1e10f).  Rows and cells further than the third-smallest distance so far,
// less the 0.001 h of the cell rounding, are skipped.  Bound by latency: 500k
// clustered points 736 -> 228 us against three scattered 4-byte reads per
// candidate and every cell of each shell.
__global__ void __launch_bounds__(256)
k_knn_query(uint32_t n, KnnGrid g, const float4* __restrict__ pos, const uint32_t* __restrict__ start,
            float extent, float* __restrict__ density, float* __restrict__ log_sigma) {
  chain_wait(pos, start, density, log_sigma);
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const float4 p = pos[k];
  const int cx = (int)cell_of(p.x, g.lo[0], g.h, g.dims[0]);
  const int cy = (int)cell_of(p.y, g.lo[1], g.h, g.dims[1]);
  const int cz = (int)cell_of(p.z, g.lo[2], g.h, g.dims[2]);
  const int DX = (int)g.dims[0], DY = (int)g.dims[1], DZ = (int)g.dims[2];
  float d[3] = {1e20f, 1e20f, 1e20f};
  // the cells [x0, x1] of row (y, z)
  auto visit = [&](int x0, int x1, int y, int z) {
    const uint32_t row = ((uint32_t)z * g.dims[1] + (uint32_t)y) * g.dims[0];
    const uint32_t e = start[row + (uint32_t)x1 + 1u];
    for (uint32_t j = start[row + (uint32_t)x0]; j < e; ++j) {
      const float4 o = pos[j];
      const float dx = p.x - o.x, dy = p.y - o.y, dz = p.z - o.z;
      float s = dx * dx + dy * dy;
      s = s + dz * dz;
      if (j != k) insert3(d, s);
    }
  };
  // (a point that is not finite is no distance from any other)
  const bool finite = fabsf(p.x) + fabsf(p.y) + fabsf(p.z) < INFINITY;
  if (finite) {
    visit(cx, cx, cy, cz);
    // lower bounds of the distance along an axis to the cells `o` away:
    // below[a] to the previous cell, above[a] to the next, h per further cell
    const float slack = 0.001f * g.h;
    const int c[3] = {cx, cy, cz};
    const float q[3] = {p.x, p.y, p.z};
    float below[3], above[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // relative to the grid's origin, where the rounding is that of at most
      // 1024 cells (1e-4 h), not of the coordinates
      const float t = q[a] - g.lo[a];
      below[a] = t - (float)c[a] * g.h - slack;
      above[a] = (float)(c[a] + 1) * g.h - t - slack;
    }
    auto far2 = [&](int a, int o) {  // squared bound, offset o along axis a
      const float t = o == 0 ? 0.0f
                             : fmaxf((o < 0 ? below[a] : above[a]) + (float)(abs(o) - 1) * g.h, 0.0f);
      return t * t;
    };
    const int rmax = max(DX, max(DY, DZ));
    for (int r = 1; r <= rmax; ++r) {
      for (int oz = -r; oz <= r; ++oz) {
        const int z = cz + oz;
        if (z < 0 || z >= DZ) continue;
        const float z2 = far2(2, oz);
        if (z2 > d[2]) continue;
        for (int oy = -r; oy <= r; ++oy) {
          const int y = cy + oy;
          if (y < 0 || y >= DY) continue;
          const float yz2 = z2 + far2(1, oy);
          if (yz2 > d[2]) continue;
          const bool lo = cx - r >= 0 && yz2 + far2(0, -r) <= d[2];
          const bool hi = cx + r < DX && yz2 + far2(0, r) <= d[2];
          if (abs(oz) == r || abs(oy) == r) {
            // the whole row of the shell, its end cells where they can matter
            const int x0 = lo ? cx - r : max(cx - r + 1, 0), x1 = hi ? cx + r : min(cx + r - 1, DX - 1);
            if (x0 <= x1) visit(x0, x1, y, z);
          } else {
            if (lo) visit(cx - r, cx - r, y, z);
            if (hi) visit(cx + r, cx + r, y, z);
          }
        }
      }
      if ((double)sqrtf(d[2]) <= ((double)r - 0.001) * (double)g.h) break;
      if (cx - r <= 0 && cy - r <= 0 && cz - r <= 0 && cx + r >= DX - 1 && cy + r >= DY - 1 &&
          cz + r >= DZ - 1)
        break;  // every cell visited
    }
  }
  const float mean = ((sqrtf(d[0]) + sqrtf(d[1])) + sqrtf(d[2])) / 3.0f;
  const float lo_s = extent * 0.0007f, hi_s = extent * 0.007f, bias = extent * 0.0015f;
  float sig = fmax_(mean / 3.0f, bias);
  sig = clampf_(sig, lo_s, hi_s);
  sig = fmin_(sig, 0.1f);
  const uint32_t self = __float_as_uint(p.w);
  if (density) density[self] = mean;
  log_sigma[self] = round_f16(sky_logf(fmax_(sig, 1e-6f)));
}

// One row of blocks per plane, four points per thread (the planes' padding up
// to a multiple of four is the caller's stride): 236 bytes read and written per
// point at 7.4 TB/s (part of them in L2), 62 -> 32 us for 500k against one
// thread walking a point's 59 planes.
__global__ void __launch_bounds__(256)
k_knn_write(float* __restrict__ P, uint32_t stride, uint32_t n, const float* __restrict__ ls) {
  chain_wait(P, ls);
  const uint32_t i = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
  const uint32_t k = blockIdx.y;
  if (i >= n) return;
  float* v = P + (size_t)k * stride + i;
  const bool scale = k >= 3u && k < 6u;
  if (i + 4u <= n) {
    float4 x = *reinterpret_cast<const float4*>(scale ? ls + i : v);
    if (!scale) x = make_float4(round_f16(x.x), round_f16(x.y), round_f16(x.z), round_f16(x.w));
    *reinterpret_cast<float4*>(v) = x;
  } else {
    for (uint32_t j = 0; i + j < n; ++j) v[j] = scale ? ls[i + j] : round_f16(v[j]);
  }
}

uint32_t blocks(uint32_t n) { return (n + 255) / 256; }

}  // namespace

uint32_t knn_bounds_init(int k) { return k < 3 ? 0xFFFFFFFFu : 0u; }

float knn_bounds_decode(uint32_t u) {
  const uint32_t b = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
  float f;
  memcpy(&f, &b, 4);
  return f;
}

void launch_knn_bounds(const float* params, uint32_t stride, uint32_t n, uint32_t* out,
                       cudaStream_t s) {
  if (n) k_knn_bounds<<<min(blocks(n), 1024u), 256, 0, s>>>(params, stride, n, out);
}

void launch_knn_keys(const float* params, uint32_t stride, uint32_t n, const KnnGrid& g,
                     uint32_t* keys, cudaStream_t s) {
  if (n) chain(k_knn_keys, blocks(n), 256, 0, s, params, stride, n, g, keys);
}

void launch_knn_cell_ranges(const uint32_t* keys_sorted, uint32_t n, uint32_t cells,
                            uint32_t* cell_start, cudaStream_t s) {
  chain(k_knn_cell_ranges, blocks(cells + 1), 256, 0, s, keys_sorted, n, cells, cell_start);
}

void launch_knn_query(const float* params, uint32_t stride, uint32_t n, const KnnGrid& g,
                      const uint32_t* order, const uint32_t* cell_start, float4* pos, float extent,
                      float* density, float* log_sigma, cudaStream_t s) {
  if (!n) return;
  chain(k_knn_gather, blocks(n), 256, 0, s, params, stride, n, order, pos);
  chain(k_knn_query, blocks(n), 256, 0, s, n, g, pos, cell_start, extent, density, log_sigma);
}

void launch_knn_write(float* params, uint32_t stride, uint32_t n, const float* log_sigma,
                      cudaStream_t s) {
  if (n) chain(k_knn_write, dim3((n + 1023) / 1024, 59), 256, 0, s, params, stride, n, log_sigma);
}

}  // namespace sky
