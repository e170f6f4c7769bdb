// Headless viewer render: the reference's frame() path -- preprocess
// (preprocess.wgsl:116-215), a global depth sort (radix_sort.wgsl), one
// screen-space quad per splat (gaussian.wgsl:15-52) blended back to front
// with src-alpha / one-minus-src-alpha (gaussian-renderer.ts:863-868) into a
// cleared target -- as CUDA kernels writing an f32 RGBA device buffer.
//
// The quads are binned into 16x16 pixel tiles in depth order, and every
// pixel blends, in that order, each splat whose quad covers its centre: the
// same sequence of blend operations the rasterizer performs per pixel, so
// the result matches a per-quad CPU restatement bit for bit.  Coverage is
// tested at pixel centres in f32 with the top-left rule (left and top quad
// edges inside); a hardware rasterizer snaps quad corners to its sub-pixel
// grid, so pixels within that snap of a quad edge can differ from it.
#include "chain.cuh"
#include "sky_math.cuh"
#include "viewer.cuh"

namespace sky {
namespace {

SKY_DEV float load_param(const float* P, uint32_t stride, int plane, uint32_t g, bool r16) {
  const float v = P[(size_t)plane * stride + g];
  return r16 ? round_f16(v) : v;
}

// float_to_ordered_uint (preprocess.wgsl:101-105) of -z_camera: ascending key
// = far to near.
SKY_DEV uint32_t ordered_key(float x) {
  const uint32_t bits = __float_as_uint(x);
  const uint32_t mask = (bits & 0x80000000u) ? 0xFFFFFFFFu : 0x80000000u;
  return bits ^ mask;
}

// One Gaussian: its splat, depth key and tile rectangle; returns its tiles.
SKY_DEV uint32_t project_splat(const ViewerParams& vp, const float* __restrict__ P, uint32_t g,
                               float4* __restrict__ splats, uint32_t* __restrict__ keys,
                               uint2* __restrict__ rects) {
  const bool r16 = vp.round_f16 != 0;
  auto get = [&](int plane) { return load_param(P, vp.plane_stride, plane, g, r16); };
  keys[g] = 0xFFFFFFFFu;
  rects[g] = make_uint2(0u, 0u);
  const float px = get(0), py = get(1), pz = get(2);
  float pc[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) pc[r] = mat4_row(vp.view, r, px, py, pz, 1.0f);
  float clip[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) clip[r] = mat4_row(vp.proj, r, pc[0], pc[1], pc[2], pc[3]);
  const float w = clip[3];
  const float ndc_x = clip[0] / w, ndc_y = clip[1] / w;
  if (fabsf(ndc_x) > 1.2f || fabsf(ndc_y) > 1.2f || pc[2] < 0.0f) return 0u;
  const float opacity = 1.0f / (1.0f + sky_expf(-get(10)));
  float sig[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    sig[k] = vp.gaussian_scaling * sky_expf(clampf_(get(3 + k), -10.0f, 10.0f));
  const float q0 = get(6), q1 = get(7), q2 = get(8), q3 = get(9);
  float qq = q0 * q0 + q1 * q1;
  qq = qq + q2 * q2;
  qq = qq + q3 * q3;
  const float ql = sqrtf(qq);
  const float rx = q0 / ql, ry = q1 / ql, rz = q2 / ql, rw = q3 / ql;
  float R[3][3];  // WGSL column-major R[col][row] (quat_to_mat3, :100-107)
  R[0][0] = 1.0f - 2.0f * (ry * ry + rz * rz);
  R[0][1] = 2.0f * (rx * ry - rw * rz);
  R[0][2] = 2.0f * (rx * rz + rw * ry);
  R[1][0] = 2.0f * (rx * ry + rw * rz);
  R[1][1] = 1.0f - 2.0f * (rx * rx + rz * rz);
  R[1][2] = 2.0f * (ry * rz - rw * rx);
  R[2][0] = 2.0f * (rx * rz - rw * ry);
  R[2][1] = 2.0f * (ry * rz + rw * rx);
  R[2][2] = 1.0f - 2.0f * (rx * rx + ry * ry);
  // C3D = transpose(S R) S R with S = diag(scaling * sigma)
  float A[3][3];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int r = 0; r < 3; ++r) A[j][r] = (sig[j] * R[r][j]) * sig[j];
  float C3[3][3];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      float acc = A[0][r] * R[j][0];
      acc = acc + A[1][r] * R[j][1];
      acc = acc + A[2][r] * R[j][2];
      C3[j][r] = acc;
    }
  // C2D = T C3D T^T with T = J Rwc (J as the WGSL constructor lays it out)
  const float tx = pc[0], ty = pc[1], tz = pc[2];
  const float fx = vp.focal[0], fy = vp.focal[1];
  const float tz2 = tz * tz;
  const float J00 = fx / tz, J11 = fy / tz;
  const float J02 = -(fx * tx) / tz2, J12 = -(fy * ty) / tz2;
  float T[3][3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float v0 = vp.view[j * 4 + 0], v1 = vp.view[j * 4 + 1];
    T[j][0] = J00 * v0;
    T[j][1] = J11 * v1;
    T[j][2] = J02 * v0 + J12 * v1;
  }
  float B0[3], B1[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    float a0 = T[0][0] * C3[j][0];
    a0 = a0 + T[1][0] * C3[j][1];
    a0 = a0 + T[2][0] * C3[j][2];
    B0[j] = a0;
    float a1 = T[0][1] * C3[j][0];
    a1 = a1 + T[1][1] * C3[j][1];
    a1 = a1 + T[2][1] * C3[j][2];
    B1[j] = a1;
  }
  float c00 = B0[0] * T[0][0];
  c00 = c00 + B0[1] * T[1][0];
  c00 = c00 + B0[2] * T[2][0];
  float c11 = B1[0] * T[0][1];
  c11 = c11 + B1[1] * T[1][1];
  c11 = c11 + B1[2] * T[2][1];
  float c01 = B1[0] * T[0][0];
  c01 = c01 + B1[1] * T[1][0];
  c01 = c01 + B1[2] * T[2][0];
  c00 = c00 + 0.3f;
  c11 = c11 + 0.3f;
  const float det = c00 * c11 - c01 * c01;
  if (det <= 0.0f) return 0u;
  const float det_inv = 1.0f / det;
  const float ca = c11 * det_inv, cb = (-c01) * det_inv, cc = c00 * det_inv;
  const float v0 = -pc[0], v1 = -pc[1], v2 = -pc[2];
  float vv = v0 * v0 + v1 * v1;
  vv = vv + v2 * v2;
  const float vl = sqrtf(vv);
  const float d0 = v0 / vl, d1 = v1 / vl, d2 = v2 / vl;
  float col[3];
  const int deg = (int)min(vp.sh_deg, 3u);
  auto sh = [&](int k, int c) { return get(11 + 3 * k + c); };
  sh_color_raw(sh, d0, d1, d2, deg, col);
#pragma unroll
  for (int c = 0; c < 3; ++c) col[c] = fmax_(0.0f, col[c]);
  const float mid = 0.5f * (c00 + c11);
  const float disc = sqrtf(fmax_(mid * mid - det, 0.0f));
  const float l1 = mid + disc, l2 = mid - disc;
  const float radius = ceilf(3.0f * sqrtf(fmax_(l1, l2)));
  const float cx = (ndc_x * 0.5f + 0.5f) * vp.viewport[0];
  const float cy = (ndc_y * -0.5f + 0.5f) * vp.viewport[1];
  splats[(size_t)g * 3 + 0] = make_float4(cx, cy, ca, cb);
  splats[(size_t)g * 3 + 1] = make_float4(cc, opacity, col[0], col[1]);
  splats[(size_t)g * 3 + 2] = make_float4(col[2], radius, 0.0f, 0.0f);
  keys[g] = ordered_key(-pc[2]);
  // tiles holding a pixel centre the quad may cover (one pixel of margin
  // each side; the raster kernel tests coverage exactly)
  const float X0 = cx - radius, X1 = cx + radius, Y0 = cy - radius, Y1 = cy + radius;
  if (!(X1 > 0.0f) || !(Y1 > 0.0f) || !(X0 < (float)vp.width) || !(Y0 < (float)vp.height)) return 0u;
  // clamped in f32 before the conversions (the bounds may be huge or infinite)
  const int xlo = (int)fmax_(floorf(X0 - 0.5f) - 1.0f, 0.0f);
  const int ylo = (int)fmax_(floorf(Y0 - 0.5f) - 1.0f, 0.0f);
  const int xhi = (int)fmin_(ceilf(X1 - 0.5f) + 1.0f, (float)vp.width - 1.0f);
  const int yhi = (int)fmin_(ceilf(Y1 - 0.5f) + 1.0f, (float)vp.height - 1.0f);
  if (xhi < xlo || yhi < ylo) return 0u;
  const uint32_t tx0 = (uint32_t)xlo / kViewTile, tx1 = (uint32_t)xhi / kViewTile + 1;
  const uint32_t ty0 = (uint32_t)ylo / kViewTile, ty1 = (uint32_t)yhi / kViewTile + 1;
  const uint32_t cnt = (tx1 - tx0) * (ty1 - ty0);
  rects[g] = make_uint2(tx0 | (ty0 << 16), tx1 | (ty1 << 16));
  return cnt;
}

// Bound by the parameter reads (236 bytes per Gaussian).  The frame's pair
// count is summed per block before it goes to the one 64-bit total: an atomic
// per Gaussian serialised on that address (1M Gaussians: 643 -> 70 us).
__global__ void __launch_bounds__(256)
k_viewer_project(ViewerParams vp, const float* __restrict__ P, float4* __restrict__ splats,
                 uint32_t* __restrict__ keys, uint32_t* __restrict__ counts,
                 uint2* __restrict__ rects, unsigned long long* __restrict__ total) {
  __shared__ unsigned long long s_sum[8];
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t cnt = 0u;
  if (g < vp.n) {
    cnt = project_splat(vp, P, g, splats, keys, rects);
    counts[g] = cnt;
  }
  unsigned long long sum = cnt;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) sum += s_sum[w];
    if (sum) atomicAdd(total, sum);
  }
}


__global__ void k_viewer_gather_counts(const uint32_t* __restrict__ order,
                                       const uint32_t* __restrict__ counts, uint32_t n,
                                       uint32_t* __restrict__ out) {
  chain_wait(order, counts, out);
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) out[k] = counts[order[k]];
}

// One thread per Gaussian in depth order; a warp's keys are consecutive, and
// where it has at most kEmitStage of them they go through shared memory, so
// that lanes write neighbouring words: 1M Gaussians at 1920x1080 47 -> 22.5 us.
constexpr uint32_t kEmitStage = 384;

__global__ void __launch_bounds__(256)
k_viewer_emit(ViewerParams vp, const uint32_t* __restrict__ order, const uint32_t* __restrict__ cum,
              const uint32_t* __restrict__ counts_sorted, const uint2* __restrict__ rects,
              uint32_t n, uint32_t* __restrict__ tile_keys, uint32_t* __restrict__ gidx) {
  chain_wait(order, cum, counts_sorted, rects, tile_keys, gidx);
  __shared__ uint32_t s_key[8][kEmitStage];
  __shared__ uint8_t s_own[8][kEmitStage];  // the lane whose Gaussian a staged key is
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t c = k < n ? counts_sorted[k] : 0u;
  const uint32_t g = k < n ? order[k] : 0u;
  const uint32_t first = k < n ? cum[k] - c : 0u;
  const uint2 rc = c ? rects[g] : make_uint2(0u, 0u);
  const uint32_t x0 = rc.x & 0xFFFFu, y0 = rc.x >> 16, x1 = rc.y & 0xFFFFu, y1 = rc.y >> 16;
  // the warp's keys are consecutive: [base, base + total)
  const uint32_t base = __shfl_sync(0xFFFFFFFFu, first, 0);
  uint32_t total = min(c, kEmitStage + 1u);  // (the sum does not wrap)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
  if (total <= kEmitStage) {
    uint32_t o = first - base;
    for (uint32_t ty = y0; ty < y1; ++ty)
      for (uint32_t tx = x0; tx < x1; ++tx, ++o) {
        s_key[warp][o] = ty * vp.tiles_x + tx;
        s_own[warp][o] = (uint8_t)lane;
      }
    __syncwarp();
    for (uint32_t t = 0; t < total; t += 32) {
      const uint32_t q = t + lane;
      const uint32_t w = q < total ? s_own[warp][q] : 0u;
      const uint32_t gw = __shfl_sync(0xFFFFFFFFu, g, (int)w);
      if (q < total) {
        tile_keys[base + q] = s_key[warp][q];
        gidx[base + q] = gw;
      }
    }
  } else {
    uint32_t o = first;
    for (uint32_t ty = y0; ty < y1; ++ty)
      for (uint32_t tx = x0; tx < x1; ++tx, ++o) {
        tile_keys[o] = ty * vp.tiles_x + tx;
        gidx[o] = g;
      }
  }
}

__global__ void k_viewer_ranges(const uint32_t* __restrict__ keys, uint32_t total, uint32_t tiles,
                                uint32_t* __restrict__ offsets) {
  chain_wait(keys, offsets);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t > tiles) return;
  uint32_t lo = 0, hi = total;  // first index with key >= t
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (keys[mid] < t) lo = mid + 1;
    else hi = mid;
  }
  offsets[t] = t == tiles ? total : lo;
}

constexpr int kViewBatch = 256;

// Two splats of a warp's list side by side, so that a lane evaluates both with
// packed operations: each float2 holds the first and the second splat's value.
struct __align__(16) SplatPair {
  float2 nmx, nmy;     // negated means
  float2 a, c;         // conic
  float2 b, opacity;
  float2 bits, blue;   // coverage bits, blue
  float2 rg[2];        // red and green of either splat
};

// One CTA per 16x16 tile, warp w on its 8x4 pixel block (w & 1, w >> 1).  The
// thread that stages a splat runs the quad's coverage test once per pixel
// column (low half of a word) and row (high half) of the tile; each warp
// lists the splats with a column and a row in its block and blends them in
// order, a pixel's test being its two bits.  The list is walked two splats at
// a time, copied side by side into shared memory 32 entries ahead (one per
// lane): exponents and exponentials are packed f32x2 operations, the blends
// follow in order.  Issue-bound: every covered (pixel, splat) pair has to be
// blended, back to front, with no early exit.  1M Gaussians at 1920x1080:
// 2184 us with warps that tested every quad of the tile at every pixel, 1595
// with lists and coverage bits, 1276 with pairs.
__global__ void __launch_bounds__(kViewTile* kViewTile, 5)
k_viewer_raster(ViewerParams vp, const float4* __restrict__ splats,
                const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ gidx,
                float4* __restrict__ rgba, uchar4* __restrict__ rgba8) {
  chain_wait(splats, offsets, gidx, rgba, rgba8);
  constexpr int NT = kViewTile * kViewTile;
  static_assert(kViewTile == 16 && kViewBatch == NT, "16-bit masks; one staged splat per thread");
  __shared__ float4 s_sp[kViewBatch][2];   // mean, conic a, b | conic c, opacity, red, green
  __shared__ float2 s_bc[kViewBatch];      // blue, coverage bits
  __shared__ uint8_t s_list[NT / 32][kViewBatch];
  __shared__ SplatPair s_pair[NT / 32][16];
  const uint32_t tile = blockIdx.x;
  const uint32_t tx = tile % vp.tiles_x, ty = tile / vp.tiles_x;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lx = 8u * (warp & 1u) + (lane & 7u), ly = 4u * (warp >> 1) + (lane >> 3);
  const uint32_t x = tx * kViewTile + lx, y = ty * kViewTile + ly;
  const bool inside = x < vp.width && y < vp.height;
  const float2 px2 = make_float2((float)x + 0.5f, (float)x + 0.5f);
  const float2 py2 = make_float2((float)y + 0.5f, (float)y + 0.5f);
  const uint32_t block_cols = 0xFFu << (8u * (warp & 1u));
  const uint32_t block_rows = 0xF0000u << (4u * (warp >> 1));
  const uint32_t my_bits = (1u << lx) | (0x10000u << ly);
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t start = offsets[tile], end = offsets[tile + 1];
  float C0 = 0.0f, C1 = 0.0f, C2 = 0.0f, A = 0.0f;  // cleared to transparent black
  for (uint32_t bs = start; bs < end; bs += kViewBatch) {
    const uint32_t cnt = min((uint32_t)kViewBatch, end - bs);
    __syncthreads();
    if (tid < cnt) {
      const size_t g = gidx[bs + tid];
      const float4 q0 = splats[g * 3 + 0], q2 = splats[g * 3 + 2];
      s_sp[tid][1] = splats[g * 3 + 1];
      s_sp[tid][0] = q0;
      const float r = q2.y;
      const float X0 = q0.x - r, X1 = q0.x + r, Y0 = q0.y - r, Y1 = q0.y + r;
      uint32_t bits = 0u;
#pragma unroll 4
      for (uint32_t k = 0; k < (uint32_t)kViewTile; ++k) {
        const float cx = (float)(tx * kViewTile + k) + 0.5f, cy = (float)(ty * kViewTile + k) + 0.5f;
        if (cx >= X0 && cx < X1) bits |= 1u << k;
        if (cy >= Y0 && cy < Y1) bits |= 0x10000u << k;
      }
      s_bc[tid] = make_float2(q2.x, __uint_as_float(bits));
    }
    __syncthreads();
    uint32_t nlist = 0;
    for (uint32_t base = 0; base < cnt; base += 32) {
      const uint32_t j = base + lane;
      const uint32_t bits = j < cnt ? __float_as_uint(s_bc[j].y) : 0u;
      const bool in = (bits & block_cols) != 0u && (bits & block_rows) != 0u;
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, in);
      if (in) s_list[warp][nlist + __popc(m & lt)] = (uint8_t)j;
      nlist += __popc(m);
    }
    for (uint32_t base = 0; base < nlist; base += 32) {
      __syncwarp();  // the list is written; the pairs before have been read
      {
        float* dst = reinterpret_cast<float*>(&s_pair[warp][lane >> 1]) + (lane & 1u);
        if (base + lane < nlist) {
          const uint32_t k = s_list[warp][base + lane];
          const float4 q0 = s_sp[k][0], q1 = s_sp[k][1];
          const float2 bc = s_bc[k];
          dst[0] = -q0.x; dst[2] = -q0.y; dst[4] = q0.z; dst[6] = q1.x;
          dst[8] = q0.w; dst[10] = q1.y; dst[12] = bc.y; dst[14] = bc.x;
          s_pair[warp][lane >> 1].rg[lane & 1u] = make_float2(q1.z, q1.w);
        } else {
          dst[12] = 0.0f;  // covers nothing
        }
      }
      __syncwarp();
      const uint32_t np = (min(32u, nlist - base) + 1u) / 2u;
      for (uint32_t p = 0; p < np; ++p) {
        const SplatPair& q = s_pair[warp][p];
        const float2 bits = q.bits;
        const bool in0 = (~__float_as_uint(bits.x) & my_bits) == 0u;
        const bool in1 = (~__float_as_uint(bits.y) & my_bits) == 0u;
        if (!in0 && !in1) continue;  // outside both quads
        const float2 dx = __fadd2_rn(px2, q.nmx), dy = __fadd2_rn(py2, q.nmy);
        const float nz = vp.neg_zero;
        const float2 s1 = mul2_rounded(__fmul2_rn(q.a, dx), dx, nz);
        const float2 s2 = mul2_rounded(__fmul2_rn(q.c, dy), dy, nz);
        float2 s = mul2_rounded(make_float2(0.5f, 0.5f), __fadd2_rn(s1, s2), nz);
        s = __fadd2_rn(s, mul2_rounded(__fmul2_rn(q.b, dx), dy, nz));
        float2 G = sky_expf_neg_pair(s, nz);
        // (beyond the exponential's range, and NaN)
        if (!(s.x <= 87.0f)) G.x = s.x != s.x ? s.x : 0.0f;
        if (!(s.y <= 87.0f)) G.y = s.y != s.y ? s.y : 0.0f;
        const float2 al = __fmul2_rn(q.opacity, G);
        auto blend = [&](float a_raw, float2 rg, float blue) {
          const float a = clampf_(a_raw, 0.0f, 1.0f);
          const float om = 1.0f - a;
          C0 = rg.x * a + C0 * om;
          C1 = rg.y * a + C1 * om;
          C2 = blue * a + C2 * om;
          A = a + A * om;
        };
        if (in0 && !(s.x < 0.0f)) blend(al.x, q.rg[0], q.blue.x);
        if (in1 && !(s.y < 0.0f)) blend(al.y, q.rg[1], q.blue.y);
      }
    }
  }
  if (inside) {
    const size_t p = (size_t)y * vp.width + x;
    rgba[p] = make_float4(C0, C1, C2, A);
    // round(clamp(v, 0, 1) * 255), halves away from zero
    auto u8 = [](float v) { return (unsigned char)lroundf(clampf_(v, 0.0f, 1.0f) * 255.0f); };
    if (rgba8) rgba8[p] = make_uchar4(u8(C0), u8(C1), u8(C2), u8(A));
  }
}

uint32_t blocks(uint32_t n, uint32_t t) { return (n + t - 1) / t; }

}  // namespace

void launch_viewer_project(const ViewerParams& vp, const float* params, float4* splats,
                           uint32_t* keys, uint32_t* counts, uint2* rects,
                           unsigned long long* total, cudaStream_t s) {
  if (vp.n)
    k_viewer_project<<<blocks(vp.n, 256), 256, 0, s>>>(vp, params, splats, keys, counts, rects, total);
}

void launch_viewer_gather_counts(const uint32_t* order, const uint32_t* counts, uint32_t n,
                                 uint32_t* counts_sorted, cudaStream_t s) {
  if (n) chain(k_viewer_gather_counts, blocks(n, 256), 256, 0, s, order, counts, n, counts_sorted);
}

void launch_viewer_emit(const ViewerParams& vp, const uint32_t* order, const uint32_t* cum,
                        const uint32_t* counts_sorted, const uint2* rects, uint32_t n,
                        uint32_t* tile_keys, uint32_t* gidx, cudaStream_t s) {
  if (n)
    chain(k_viewer_emit, blocks(n, 256), 256, 0, s, vp, order, cum, counts_sorted, rects, n, tile_keys,
                                                 gidx);
}

void launch_viewer_ranges(const uint32_t* tile_keys, uint32_t total, uint32_t tiles,
                          uint32_t* offsets, cudaStream_t s) {
  chain(k_viewer_ranges, blocks(tiles + 1, 256), 256, 0, s, tile_keys, total, tiles, offsets);
}

void launch_viewer_raster(const ViewerParams& vp, const float4* splats, const uint32_t* offsets,
                          const uint32_t* gidx, float4* rgba, uchar4* rgba8, cudaStream_t s) {
  const uint32_t tiles = vp.tiles_x * vp.tiles_y;
  if (tiles)
    chain(k_viewer_raster, tiles, kViewTile * kViewTile, 0, s, vp, splats, offsets, gidx, rgba, rgba8);
}

}  // namespace sky
