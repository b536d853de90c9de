// Memory-bound kernels for sm_100a: RMSNorm (+ per-head QK-norm with RoPE), gated
// activations, the dual-orientation MXFP8 quantiser, cross-entropy over a logits
// chunk, flat AdamW (fp32 / bf16 / block-scaled 8-bit moments), and the MoE row
// gather / weighted combine. All use 128-bit accesses and fp32 math; none allocates.
//
// Reference counterparts: norm_rope Pallas kernel (architecture/attention/norm_rope.py),
// MXFP8 quantiser (architecture/precision/blockscaled.py:386-445), chunked
// cross-entropy (architecture/logits.py:209-353), optax AdamW (train/optim.py:403),
// token_rows / token_sums (architecture/experts/moe.py:992-1071).
#include "common.cuh"
#include "elementwise.h"

#include <cuda_fp4.h>

namespace bux {

// ---------------------------------------------------------------- RMSNorm
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t* u = &v.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 t = unpack_bf16(u[j]); f[2 * j] = t.x; f[2 * j + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
// Eight fp32 gains from column 8 i (1 without gains); `w16`: w starts on a 16-byte boundary.
__device__ __forceinline__ void load_gain8(const float* __restrict__ w, bool w16, int i, float (&g)[8]) {
  if (w == nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = 1.f;
  } else if (w16) {
    const float4 lo = reinterpret_cast<const float4*>(w)[2 * i], hi = reinterpret_cast<const float4*>(w)[2 * i + 1];
    g[0] = lo.x; g[1] = lo.y; g[2] = lo.z; g[3] = lo.w; g[4] = hi.x; g[5] = hi.y; g[6] = hi.z; g[7] = hi.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = w[i * 8 + j];
  }
}

// One warp per row. x, y: [rows, d] bf16; w: [d] fp32 or null; rstd: [rows] fp32 out. NV > 0: the
// row stays in registers, NV 16-byte loads per lane all in flight (rows up to 32 * 8 * NV wide); it
// is a stream, bound by the bytes it keeps in flight: 16384 x 2048 took 49 us with the row read
// a second time and one load in flight at a time, 31 now. NV = 0: rows of any width, read twice.
template <int NV>
__global__ void __launch_bounds__(256, NV > 0 ? 3 : 2)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, bool w16,
                   __nv_bfloat16* __restrict__ y, float* __restrict__ rstd, int rows, int d, float eps) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * d);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * d);
  const int nvec = d / 8;
  constexpr int HELD = NV > 0 ? NV : 1;
  uint4 held[HELD];
  float ss = 0.f;
  if (NV > 0) {
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
      const int i = lane + 32 * k;
      held[k] = i < nvec ? xr[i] : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
      float f[8];
      unpack8(held[k], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
  } else {
    for (int i = lane; i < nvec; i += 32) {
      float f[8];
      unpack8(xr[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / d + eps);
  if (lane == 0 && rstd) rstd[row] = r;
  auto emit = [&](int i, const uint4& v) {
    float f[8], g[8];
    unpack8(v, f);
    load_gain8(w, w16, i, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * r * g[j];
    yr[i] = pack8(f);
  };
  if (NV > 0) {
#pragma unroll
    for (int k = 0; k < HELD; ++k)
      if (lane + 32 * k < nvec) emit(lane + 32 * k, held[k]);
  } else {
    for (int i = lane; i < nvec; i += 32) emit(i, xr[i]);
  }
}

// Rows wider than a warp holds (d <= 8192), and few rows of 1024 and more: a thread owns PIECES times eight
// columns of ROWS rows, loaded together; the squares meet in shared memory. 8192 x 4096: 55 us with a
// warp per row, 38 so (two rows; with four, 8192 x 2880 takes 31 instead of 27). Beyond 4096 columns two
// pieces per thread keep two blocks on an SM, one loading while the other waits for its sums (32768 x 8192: a
// warp per row 341 us, one block of 1024 threads 400, so 211; 32768 x 6144 257, 309, 174).
template <int PIECES, int ROWS>
__global__ void __launch_bounds__(512, PIECES > 1 ? 2 : 3)
rmsnorm_fwd_columns_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, bool w16,
                           __nv_bfloat16* __restrict__ y, float* __restrict__ rstd, int rows, int d, float eps) {
  __shared__ float part[16][ROWS];
  const int nvec = d / 8, nw = blockDim.x >> 5, r0 = blockIdx.x * ROWS;
  uint4 v[ROWS][PIECES];
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int i = threadIdx.x + p * blockDim.x;
      v[k][p] = i < nvec && r0 + k < rows ? reinterpret_cast<const uint4*>(x)[(size_t)(r0 + k) * nvec + i] : make_uint4(0, 0, 0, 0);
    }
  }
  float g[PIECES][8];
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
    if (threadIdx.x + p * blockDim.x < nvec) load_gain8(w, w16, threadIdx.x + p * blockDim.x, g[p]);
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    float ss = 0.f;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      float f[8];
      unpack8(v[k][p], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][k] = ss;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    float ss = 0.f;
    for (int q = 0; q < nw; ++q) ss += part[q][k];
    const float r = rsqrtf(ss / d + eps);
    if (r0 + k >= rows) break;
    if (threadIdx.x == 0 && rstd) rstd[r0 + k] = r;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int i = threadIdx.x + p * blockDim.x;
      float f[8];
      unpack8(v[k][p], f);
      if (i < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * r * g[p][j];
        reinterpret_cast<uint4*>(y)[(size_t)(r0 + k) * nvec + i] = pack8(f);
      }
    }
  }
}

// Backward: dx = r * (w*dy) - x * r^3 * mean(w*dy*x); dw += sum_rows dy * x * r.
// A thread owns eight columns of every row its block walks, so dw stays in eight registers; the
// block takes ROWS rows at a time (2 * ROWS 16-byte loads in flight per thread, each element
// read once) and shares their dot products through shared memory, one barrier per step (the sums
// alternate between two buffers). For 512 <= d <= 8192 (a block of d / 8 threads, 2 to 32 warps);
// beyond 512 threads a thread has 64 registers, which hold two rows.
// 16384 x 2048: 80 us with a warp per row, rows read twice and dw in shared memory, 48 now.
template <int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS, THREADS > 512 ? 1 : 512 / THREADS)
rmsnorm_bwd_columns_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, bool w16,
                           const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd,
                           __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part, int rows, int d) {
  __shared__ float part[2][32][ROWS];
  const int nvec = d / 8, i = threadIdx.x, nw = blockDim.x >> 5;
  const bool mine = i < nvec;
  float g[8], acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { g[j] = 0.f; acc[j] = 0.f; }
  if (mine) load_gain8(w, w16, i, g);
  const int groups = (rows + ROWS - 1) / ROWS;
  int buf = 0;
  for (int gr = blockIdx.x; gr < groups; gr += gridDim.x, buf ^= 1) {
    const int r0 = gr * ROWS;
    uint4 xv[ROWS], gv[ROWS];
    float r[ROWS], dot[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const bool live = mine && r0 + k < rows;
      const size_t at = (size_t)(r0 + k) * nvec + i;
      xv[k] = live ? reinterpret_cast<const uint4*>(x)[at] : make_uint4(0, 0, 0, 0);
      gv[k] = live ? reinterpret_cast<const uint4*>(dy)[at] : make_uint4(0, 0, 0, 0);
      r[k] = r0 + k < rows ? rstd[r0 + k] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      float a[8], b[8];
      unpack8(xv[k], a); unpack8(gv[k], b);
      dot[k] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) dot[k] += a[j] * b[j] * g[j];
      dot[k] = warp_sum(dot[k]);
    }
    if ((i & 31) == 0) {
#pragma unroll
      for (int k = 0; k < ROWS; ++k) part[buf][i >> 5][k] = dot[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ROWS; ++k) dot[k] = 0.f;
    for (int q = 0; q < nw; ++q) {
#pragma unroll
      for (int k = 0; k < ROWS; ++k) dot[k] += part[buf][q][k];
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      if (!mine || r0 + k >= rows) continue;
      const float c = dot[k] * r[k] * r[k] * r[k] / d;
      float a[8], b[8], o[8];
      unpack8(xv[k], a); unpack8(gv[k], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = r[k] * g[j] * b[j] - a[j] * c;
        acc[j] += b[j] * a[j] * r[k];
      }
      reinterpret_cast<uint4*>(dx)[(size_t)(r0 + k) * nvec + i] = pack8(o);
    }
  }
  if (dw_part && mine) {
    float4* out = reinterpret_cast<float4*>(dw_part + (size_t)blockIdx.x * d + i * 8);
    out[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    out[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
  }
}

// out[c] = sum of part[0..n)[c]: a block per 32 columns, 32 rows side by side.
__global__ void __launch_bounds__(1024)
sum_rows_kernel(const float* __restrict__ part, float* __restrict__ out, int n, int d) {
  __shared__ float sums[32][33];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
  float acc = 0.f;
  if (c < d) {
#pragma unroll 4
    for (int r = w; r < n; r += 32) acc += part[(size_t)r * d + c];
  }
  sums[w][threadIdx.x & 31] = acc;
  __syncthreads();
  acc = warp_sum(sums[threadIdx.x & 31][w]);
  const int oc = blockIdx.x * 32 + w;
  if ((threadIdx.x & 31) == 0 && oc < d) out[oc] = acc;
}

// The other widths: a warp per row.
// Each block walks rows grid-stride, keeps its dw partial in shared memory (fp32) and
// adds it to the global fp32 dw once at the end.
__global__ void rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w,
                                   const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd,
                                   __nv_bfloat16* __restrict__ dx, float* __restrict__ dw,
                                   int rows, int d) {
  extern __shared__ float dw_part[];
  for (int i = threadIdx.x; i < d; i += blockDim.x) dw_part[i] = 0.f;
  __syncthreads();
  const int warps_per_block = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = d / 8;
  for (int row = blockIdx.x * warps_per_block + warp; row < rows; row += gridDim.x * warps_per_block) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * d);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + (size_t)row * d);
    const float r = rstd[row];
    float dot = 0.f;
    for (int i = lane; i < nvec; i += 32) {
      uint4 xv = xr[i], gv = gr[i];
      const uint32_t* xu = &xv.x; const uint32_t* gu = &gv.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 a = unpack_bf16(xu[j]), g = unpack_bf16(gu[j]);
        const float w0 = w ? w[i * 8 + 2 * j] : 1.f, w1 = w ? w[i * 8 + 2 * j + 1] : 1.f;
        dot += a.x * g.x * w0 + a.y * g.y * w1;
      }
    }
    dot = warp_sum(dot);
    const float c = dot * r * r * r / d;
    uint4* dxr = reinterpret_cast<uint4*>(dx + (size_t)row * d);
    for (int i = lane; i < nvec; i += 32) {
      uint4 xv = xr[i], gv = gr[i], o;
      const uint32_t* xu = &xv.x; const uint32_t* gu = &gv.x; uint32_t* ou = &o.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 a = unpack_bf16(xu[j]), g = unpack_bf16(gu[j]);
        const int col = i * 8 + 2 * j;
        const float w0 = w ? w[col] : 1.f, w1 = w ? w[col + 1] : 1.f;
        ou[j] = pack_bf16(r * w0 * g.x - a.x * c, r * w1 * g.y - a.y * c);
        if (dw) {
          atomicAdd(&dw_part[col], g.x * a.x * r);
          atomicAdd(&dw_part[col + 1], g.y * a.y * r);
        }
      }
      dxr[i] = o;
    }
  }
  __syncthreads();
  if (dw)
    for (int i = threadIdx.x; i < d; i += blockDim.x) atomicAdd(&dw[i], dw_part[i]);
}

// The same backward with one private fp32 slab of dw per warp in shared memory: a lane owns
// its columns of the slab, so the per-row update is a plain vector read-modify-write (no
// atomics); the slabs are summed once at the end. Needs 8 warps · d · 4 bytes of shared memory.
__global__ void __launch_bounds__(256)
rmsnorm_bwd_slab_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w,
                        const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd,
                        __nv_bfloat16* __restrict__ dx, float* __restrict__ dw, int rows, int d) {
  extern __shared__ __align__(16) float slabs[];  // [warps][d]
  const int warps_per_block = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < warps_per_block * d; i += blockDim.x) slabs[i] = 0.f;
  __syncthreads();
  float4* mine = reinterpret_cast<float4*>(slabs + (size_t)warp * d);
  const float4* w4 = reinterpret_cast<const float4*>(w);
  const int nvec = d / 8;
  for (int row = blockIdx.x * warps_per_block + warp; row < rows; row += gridDim.x * warps_per_block) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * d);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + (size_t)row * d);
    const float r = rstd[row];
    float dot = 0.f;
    for (int i = lane; i < nvec; i += 32) {
      const uint4 xv = xr[i], gv = gr[i];
      const uint32_t* xu = &xv.x; const uint32_t* gu = &gv.x;
      float wl[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
      if (w) {
        const float4 lo = w4[2 * i], hi = w4[2 * i + 1];
        wl[0] = lo.x; wl[1] = lo.y; wl[2] = lo.z; wl[3] = lo.w; wl[4] = hi.x; wl[5] = hi.y; wl[6] = hi.z; wl[7] = hi.w;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = unpack_bf16(xu[j]), g = unpack_bf16(gu[j]);
        dot += a.x * g.x * wl[2 * j] + a.y * g.y * wl[2 * j + 1];
      }
    }
    dot = warp_sum(dot);
    const float c = dot * r * r * r / d;
    uint4* dxr = reinterpret_cast<uint4*>(dx + (size_t)row * d);
    for (int i = lane; i < nvec; i += 32) {
      const uint4 xv = xr[i], gv = gr[i];  // second read of the row: L1 / L2
      const uint32_t* xu = &xv.x; const uint32_t* gu = &gv.x;
      float wl[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
      if (w) {
        const float4 lo = w4[2 * i], hi = w4[2 * i + 1];
        wl[0] = lo.x; wl[1] = lo.y; wl[2] = lo.z; wl[3] = lo.w; wl[4] = hi.x; wl[5] = hi.y; wl[6] = hi.z; wl[7] = hi.w;
      }
      uint4 o; uint32_t* ou = &o.x;
      float p[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = unpack_bf16(xu[j]), g = unpack_bf16(gu[j]);
        ou[j] = pack_bf16(r * wl[2 * j] * g.x - a.x * c, r * wl[2 * j + 1] * g.y - a.y * c);
        p[2 * j] = g.x * a.x * r;
        p[2 * j + 1] = g.y * a.y * r;
      }
      dxr[i] = o;
      if (dw) {
        float4 lo = mine[2 * i], hi = mine[2 * i + 1];
        lo.x += p[0]; lo.y += p[1]; lo.z += p[2]; lo.w += p[3];
        hi.x += p[4]; hi.y += p[5]; hi.z += p[6]; hi.w += p[7];
        mine[2 * i] = lo; mine[2 * i + 1] = hi;
      }
    }
  }
  __syncthreads();
  if (dw)
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
      float total = 0.f;
      for (int k = 0; k < warps_per_block; ++k) total += slabs[(size_t)k * d + i];
      atomicAdd(&dw[i], total);
    }
}

// ---------------------------------------------------------------- QK-norm + RoPE
// x: [tokens, heads, D] bf16 (row stride `stride_tok` elements so it may be a slice of
// a fused qkv buffer); cos/sin: [tokens, D/2] fp32; w: [D] fp32 or null (no norm).
__device__ __forceinline__ void load_f32x8(const float* p, float (&out)[8]) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float4 t = reinterpret_cast<const float4*>(p)[j];
    out[4 * j] = t.x; out[4 * j + 1] = t.y; out[4 * j + 2] = t.z; out[4 * j + 3] = t.w;
  }
}

// D / 16 lanes per (token, head): a lane holds eight elements of the lower half and the eight they
// rotate with, so the rotation needs no exchange and one set of cos / sin serves sixteen elements.
// A lane group takes HC heads of a token at a time: their loads are in flight together and share the
// token's cos / sin (which were four fifths of what it loaded with one head at a time and halves
// in different lanes). 8192 tokens x 32 heads of 128: forward 45 -> 28 us, backward 90 -> 45.
// A single head, or so few that their lanes do not fill the GPU, goes one per lane group.
template <int D, bool BWD, int HC>
__global__ void __launch_bounds__(256)
norm_rope_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, bool w16,
                 const float* __restrict__ cs, const float* __restrict__ sn,
                 __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_io,
                 const __nv_bfloat16* __restrict__ dy, float* __restrict__ dw,
                 long tokens, int heads, long stride_tok_x, long stride_tok_y, float eps) {
  constexpr int LPI = D / 16;         // lanes per item: 4, 8 or 16
  constexpr int IPW = 32 / LPI;       // items (token, HC heads) per warp
  __shared__ float dw_part[D];
  if (BWD) {
    for (int i = threadIdx.x; i < D; i += blockDim.x) dw_part[i] = 0.f;
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const int sub = lane / LPI, li = lane % LPI;
  const long nwarps = (long)gridDim.x * (blockDim.x >> 5);
  const int chunks = (heads + HC - 1) / HC;
  const long total = tokens * chunks;
  const long steps = (total + IPW - 1) / IPW;   // whole warps iterate together (shuffles stay converged)
  float dwa[8], dwb[8], wa[8], wb[8];           // a = lower half, b = upper half
#pragma unroll
  for (int j = 0; j < 8; ++j) { dwa[j] = 0.f; dwb[j] = 0.f; }
  load_gain8(w, w16, li, wa);
  load_gain8(w, w16, li + LPI, wb);
  for (long step = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); step < steps; step += nwarps) {
    const long item = step * IPW + sub;
    const bool live = item < total;
    const long tok = live ? item / chunks : 0;
    const int h0 = live ? (int)(item % chunks) * HC : 0;
    const __nv_bfloat16* xp = x + tok * stride_tok_x + (long)h0 * D + li * 8;
    const __nv_bfloat16* gp = BWD ? dy + tok * stride_tok_y + (long)h0 * D + li * 8 : nullptr;
    __nv_bfloat16* yp = y + tok * stride_tok_y + (long)h0 * D + li * 8;   // backward: dx (dense, like dy)
    uint4 xa[HC], xb[HC], ga[HC], gb[HC];
    float r[HC];
#pragma unroll
    for (int k = 0; k < HC; ++k) {
      const bool on = live && h0 + k < heads;
      if (!BWD || w) {
        xa[k] = on ? *reinterpret_cast<const uint4*>(xp + k * D) : make_uint4(0, 0, 0, 0);
        xb[k] = on ? *reinterpret_cast<const uint4*>(xp + k * D + D / 2) : make_uint4(0, 0, 0, 0);
      }
      if (BWD) {
        ga[k] = on ? *reinterpret_cast<const uint4*>(gp + k * D) : make_uint4(0, 0, 0, 0);
        gb[k] = on ? *reinterpret_cast<const uint4*>(gp + k * D + D / 2) : make_uint4(0, 0, 0, 0);
        r[k] = on && w ? rstd_io[tok * heads + h0 + k] : 0.f;
      }
    }
    float c[8], s[8];
    load_f32x8(cs + tok * (D / 2) + li * 8, c);
    load_f32x8(sn + tok * (D / 2) + li * 8, s);
#pragma unroll
    for (int k = 0; k < HC; ++k) {
      const bool on = live && h0 + k < heads;
      float a[8], b[8], oa[8], ob[8];
      if (!BWD) {
        unpack8(xa[k], a); unpack8(xb[k], b);
        if (w) {
          float ss = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) ss += a[j] * a[j] + b[j] * b[j];
#pragma unroll
          for (int o = LPI / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          const float rr = rsqrtf(ss / D + eps);
          if (li == 0 && on && rstd_io) rstd_io[tok * heads + h0 + k] = rr;
#pragma unroll
          for (int j = 0; j < 8; ++j) { a[j] = a[j] * rr * wa[j]; b[j] = b[j] * rr * wb[j]; }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) { oa[j] = a[j] * c[j] - b[j] * s[j]; ob[j] = a[j] * s[j] + b[j] * c[j]; }
      } else {
        // dy -> d(normed) by the inverse rotation, then RMSNorm backward per head
        float ya[8], yb[8];
        unpack8(ga[k], ya); unpack8(gb[k], yb);
#pragma unroll
        for (int j = 0; j < 8; ++j) { oa[j] = ya[j] * c[j] + yb[j] * s[j]; ob[j] = yb[j] * c[j] - ya[j] * s[j]; }
        if (w) {
          unpack8(xa[k], a); unpack8(xb[k], b);
          float dot = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) dot += oa[j] * wa[j] * a[j] + ob[j] * wb[j] * b[j];
#pragma unroll
          for (int o = LPI / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
          const float cc = dot * r[k] * r[k] * r[k] / D;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            dwa[j] += oa[j] * a[j] * r[k];
            dwb[j] += ob[j] * b[j] * r[k];
            oa[j] = r[k] * wa[j] * oa[j] - a[j] * cc;
            ob[j] = r[k] * wb[j] * ob[j] - b[j] * cc;
          }
        }
      }
      if (on) {
        *reinterpret_cast<uint4*>(yp + k * D) = pack8(oa);
        *reinterpret_cast<uint4*>(yp + k * D + D / 2) = pack8(ob);
      }
    }
  }
  if (BWD && dw) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      // lanes of a warp that hold the same columns add up before the block does
#pragma unroll
      for (int o = LPI; o < 32; o <<= 1) {
        dwa[j] += __shfl_xor_sync(0xffffffffu, dwa[j], o);
        dwb[j] += __shfl_xor_sync(0xffffffffu, dwb[j], o);
      }
      if (sub == 0) { atomicAdd(&dw_part[li * 8 + j], dwa[j]); atomicAdd(&dw_part[D / 2 + li * 8 + j], dwb[j]); }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += blockDim.x) atomicAdd(&dw[i], dw_part[i]);
  }
}

// ---------------------------------------------------------------- gated activations
__device__ __forceinline__ float act_fwd(float g, int kind) {
  if (kind == ACT_SWISH) return __fdividef(g, 1.f + __expf(-g));
  if (kind == ACT_QUICK_GELU) return __fdividef(g, 1.f + __expf(-1.702f * g));
  if (kind == ACT_GELU_TANH) {
    const float u = 0.7978845608f * (g + 0.044715f * g * g * g);
    return 0.5f * g * (1.f + tanhf(u));
  }
  if (kind == ACT_RELU2) { const float r = fmaxf(g, 0.f); return r * r; }
  return g;
}
__device__ __forceinline__ float act_grad(float g, int kind) {
  if (kind == ACT_SWISH) { const float s = __fdividef(1.f, 1.f + __expf(-g)); return s * (1.f + g * (1.f - s)); }
  if (kind == ACT_QUICK_GELU) { const float s = __fdividef(1.f, 1.f + __expf(-1.702f * g)); return s * (1.f + 1.702f * g * (1.f - s)); }
  if (kind == ACT_GELU_TANH) {
    const float u = 0.7978845608f * (g + 0.044715f * g * g * g);
    const float t = tanhf(u);
    return 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * 0.7978845608f * (1.f + 3.f * 0.044715f * g * g);
  }
  if (kind == ACT_RELU2) return 2.f * fmaxf(g, 0.f);
  return 1.f;
}

// act(g) and act'(g) together: the sigmoid kinds share their one exponential and reciprocal.
__device__ __forceinline__ void act_both(float g, int kind, float& a, float& da) {
  if (kind == ACT_SWISH || kind == ACT_QUICK_GELU) {
    const float k = kind == ACT_SWISH ? 1.f : 1.702f;
    const float s = __fdividef(1.f, 1.f + __expf(-k * g));
    a = g * s;
    da = s * (1.f + k * g * (1.f - s));
    return;
  }
  a = act_fwd(g, kind);
  da = act_grad(g, kind);
}

// h: [rows, 2f] (gate columns [0,f), up columns [f,2f)); out: [rows, f].
// limit > 0 clamps gate from above and up to [-limit, limit] (gpt-oss); up_offset is
// added to up after the clamp. Optional row scale (router weight) multiplies the output.
__global__ void glu_fwd_kernel(const __nv_bfloat16* __restrict__ h, __nv_bfloat16* __restrict__ out,
                               const float* __restrict__ row_scale, long rows, int f, int kind,
                               float limit, float up_offset) {
  const long total = rows * (long)(f / 8);
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long row = i / (f / 8);
    const int c8 = (int)(i % (f / 8));
    const uint4 gv = *reinterpret_cast<const uint4*>(h + row * 2 * f + c8 * 8);
    const uint4 uv = *reinterpret_cast<const uint4*>(h + row * 2 * f + f + c8 * 8);
    const float rs = row_scale ? row_scale[row] : 1.f;
    uint4 o; uint32_t* ou = &o.x; const uint32_t* gu = &gv.x; const uint32_t* uu = &uv.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 g = unpack_bf16(gu[j]), u = unpack_bf16(uu[j]);
      if (limit > 0.f) {
        g.x = fminf(g.x, limit); g.y = fminf(g.y, limit);
        u.x = fminf(fmaxf(u.x, -limit), limit); u.y = fminf(fmaxf(u.y, -limit), limit);
      }
      ou[j] = pack_bf16(act_fwd(g.x, kind) * (u.x + up_offset) * rs, act_fwd(g.y, kind) * (u.y + up_offset) * rs);
    }
    *reinterpret_cast<uint4*>(out + row * f + c8 * 8) = o;
  }
}

// dh: [rows, 2f] from dout [rows, f], eight columns of both halves at a time. Returns this piece's
// share of d(row_scale) = sum_cols dout * act(g) * (u + off).
__device__ __forceinline__ float glu_bwd_piece(const uint4& gv, const uint4& uv, const uint4& dv, float rs, int kind,
                                               float limit, float up_offset, uint4& og, uint4& ou) {
  uint32_t* ogu = &og.x; uint32_t* ouu = &ou.x;
  const uint32_t* gu = &gv.x; const uint32_t* uu = &uv.x; const uint32_t* du = &dv.x;
  float ds = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 g = unpack_bf16(gu[j]), u = unpack_bf16(uu[j]), d = unpack_bf16(du[j]);
    float gx[2] = {g.x, g.y}, ux[2] = {u.x, u.y}, dx[2] = {d.x, d.y}, rg[2], ru[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      bool g_pass = true, u_pass = true;
      float gg = gx[e], uu_ = ux[e];
      if (limit > 0.f) {
        if (gg > limit) { gg = limit; g_pass = false; }
        if (uu_ > limit) { uu_ = limit; u_pass = false; }
        if (uu_ < -limit) { uu_ = -limit; u_pass = false; }
      }
      float a, da;
      act_both(gg, kind, a, da);
      ds += dx[e] * a * (uu_ + up_offset);
      const float dsc = dx[e] * rs;
      rg[e] = g_pass ? dsc * (uu_ + up_offset) * da : 0.f;
      ru[e] = u_pass ? dsc * a : 0.f;
    }
    ogu[j] = pack_bf16(rg[0], rg[1]);
    ouu[j] = pack_bf16(ru[0], ru[1]);
  }
  return ds;
}

__global__ void __launch_bounds__(256)
glu_bwd_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ dout,
               __nv_bfloat16* __restrict__ dh, const float* __restrict__ row_scale, long rows, int f, int kind,
               float limit, float up_offset) {
  const long total = rows * (long)(f / 8);
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long row = i / (f / 8);
    const int c8 = (int)(i % (f / 8));
    const uint4 gv = *reinterpret_cast<const uint4*>(h + row * 2 * f + c8 * 8);
    const uint4 uv = *reinterpret_cast<const uint4*>(h + row * 2 * f + f + c8 * 8);
    const uint4 dv = *reinterpret_cast<const uint4*>(dout + row * f + c8 * 8);
    uint4 og, ou;
    glu_bwd_piece(gv, uv, dv, row_scale ? row_scale[row] : 1.f, kind, limit, up_offset, og, ou);
    *reinterpret_cast<uint4*>(dh + row * 2 * f + c8 * 8) = og;
    *reinterpret_cast<uint4*>(dh + row * 2 * f + f + c8 * 8) = ou;
  }
}

// The same with the gradient of the row scale: TPR threads per row, so that the row's sum is a
// reduction and one store. (An atomic per eight columns queued f / 8 of them on one address:
// 7200 rows of 2880 took 129 us, a warp per row 51; 147456 rows of 768 312 and 182.)
template <int TPR>
__global__ void __launch_bounds__(256)
glu_bwd_rows_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ dout,
                    __nv_bfloat16* __restrict__ dh, const float* __restrict__ row_scale,
                    float* __restrict__ d_row_scale, long rows, int f, int kind, float limit, float up_offset) {
  constexpr int RPB = 256 / TPR;   // rows a block works on at once
  __shared__ float part[8];
  const int li = threadIdx.x % TPR, nvec = f / 8;
  // whole blocks iterate together: the reductions need every thread
  for (long first = (long)blockIdx.x * RPB; first < rows; first += (long)gridDim.x * RPB) {
    const long row = first + threadIdx.x / TPR;
    float ds = 0.f;
    if (row < rows) {
      const uint4* gp = reinterpret_cast<const uint4*>(h + row * 2 * f);
      const uint4* dp = reinterpret_cast<const uint4*>(dout + row * f);
      uint4* op = reinterpret_cast<uint4*>(dh + row * 2 * f);
      const float rs = row_scale ? row_scale[row] : 1.f;
#pragma unroll 3
      for (int c = li; c < nvec; c += TPR) {
        const uint4 gv = gp[c], uv = gp[nvec + c], dv = dp[c];
        uint4 og, ou;
        ds += glu_bwd_piece(gv, uv, dv, rs, kind, limit, up_offset, og, ou);
        op[c] = og;
        op[nvec + c] = ou;
      }
    }
#pragma unroll
    for (int o = (TPR < 32 ? TPR : 32) / 2; o > 0; o >>= 1) ds += __shfl_xor_sync(0xffffffffu, ds, o);
    if (TPR > 32) {
      if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ds;
      __syncthreads();
      ds = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) ds += part[w];
      __syncthreads();
    }
    if (li == 0 && row < rows) d_row_scale[row] = ds;
  }
}

// ---------------------------------------------------------------- MXFP8 quantiser
// Tile: 128 rows x 128 columns per block of 256 threads, staged once in shared memory as
// bf16 (see qtile_at for its layout). Each tile fills exactly one 512-byte scale tile of the row-wise output and one
// of the transposed output, written as whole tiles (padding scales included), and every
// byte of both quantised outputs inside the padded extents, so the caller allocates
// without clearing. Optional row gather (`row_index[r]` = source row of output row r,
// negative = zero row) fuses the MoE permute into the quantiser.
//   q_row [R, C] e4m3, sf_row tiles over (R, C/32);  q_col [C, R_pad] e4m3 (R_pad = ld_col),
//   sf_col tiles over (C, R_pad/32).
constexpr int QT = 128;
// The 128×128 bf16 tile sits in shared memory without padding, its 16-byte chunks (8 columns)
// XOR-swizzled so that three access patterns are all free of bank conflicts: eight consecutive
// chunks of a row (the load), chunk k of the four 32-column blocks of two adjacent rows (the
// row-wise pass), and one chunk of the rows 32a + b, a < 4, b < 2 (the transposing ldmatrix of the
// column pass).
__device__ __forceinline__ int qtile_at(int row, int chunk) {
  const int g = (((row >> 5) & 3) << 1) | (row & 1);
  return row * QT + (((chunk & 8) | ((chunk ^ g ^ ((chunk >> 3) << 1)) & 7)) << 3);
}
// The largest magnitude of 32 bf16 values in 16 words, two at a time (a NaN never wins: 0 where all are).
__device__ __forceinline__ float amax32(const uint32_t (&w)[16]) {
  uint32_t m = w[0] & 0x7fff7fffu;
#pragma unroll
  for (int j = 1; j < 16; ++j) asm("max.bf16x2 %0, %1, %2;" : "=r"(m) : "r"(m), "r"(w[j] & 0x7fff7fffu));
  const float2 t = unpack_bf16(m);
  return fmaxf(fmaxf(t.x, t.y), 0.f);
}
// 1 / 2^(e - 127) as bf16 (exact; e = 254 gives bf16's 2^-127).
__device__ __forceinline__ unsigned short e8m0_inv_bf16(uint8_t e) {
  return e < 254 ? (unsigned short)((254 - e) << 7) : (unsigned short)0x0040;
}
// Both values of a bf16 pair times a bf16 power of two, exactly, in fp32: one mixed-precision
// multiply-add each (adding -0 keeps the sign of zeros) instead of a conversion and a product.
__device__ __forceinline__ float2 scaled_bf16(uint32_t w, unsigned short inv) {
  float2 t;
  asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(t.x) : "h"((unsigned short)w), "h"(inv), "f"(-0.f));
  asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(t.y) : "h"((unsigned short)(w >> 16)), "h"(inv), "f"(-0.f));
  return t;
}
// 32 values times `inv` as e4m3 to 32 consecutive bytes: one 32-byte store where the address allows.
__device__ __forceinline__ void store_e4m3x32(uint8_t* dst, const uint32_t (&w)[16], unsigned short inv, bool wide) {
  uint32_t q[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 a = scaled_bf16(w[2 * j], inv), b = scaled_bf16(w[2 * j + 1], inv);
    q[j] = cvt_e4m3x4(a.x, a.y, b.x, b.y);
  }
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(q[0]), "r"(q[1]), "r"(q[2]),
                 "r"(q[3]), "r"(q[4]), "r"(q[5]), "r"(q[6]), "r"(q[7]) : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) reinterpret_cast<uint2*>(dst)[j] = make_uint2(q[2 * j], q[2 * j + 1]);
  }
}

// What the quantiser reads its 128×128 tile from: the matrix itself, or a gated activation
// computed on the way in (the activation, or its gradient, is then never written as bf16).
constexpr int QUANT_CTAS = 5, QUANT_GLU_CTAS = 4;   // blocks per SM: 48 and 64 registers a thread
enum { QSRC_PLAIN = 0, QSRC_GLU_FWD = 1, QSRC_GLU_BWD = 2, QSRC_MX = 3 };
struct QuantGlu {
  const float* row_scale;     // PLAIN: output row r is its source row times row_scale[r] (rounded to bf16);
                              // GLU_FWD: the activation of row r times row_scale[r] (as glu_fwd_kernel)
  const __nv_bfloat16* dout;  // GLU_BWD: gradient of the activation's output [rows, f]
  int f;                      // h is [rows, 2f]: gate columns, then up columns
  int kind;
  float limit, up_offset;
  const uint8_t* src_sf;      // MX: the source is e4m3 bytes [rows, cols] with these scale tiles (along cols)
};

// Eight bf16 values of eight e4m3 bytes times their block's scale 2^(e - 127) (exact in bf16).
__device__ __forceinline__ uint4 dequant_e4m3x8(uint2 q, uint8_t e) {
  const float sc = e > 0 ? __uint_as_float((uint32_t)e << 23) : __uint_as_float(0x00400000u);
  uint4 o; uint32_t* ou = &o.x;
  const uint32_t w[2] = {q.x, q.y};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_fp8x2_storage_t pair = (__nv_fp8x2_storage_t)((w[j >> 1] >> (16 * (j & 1))) & 0xffffu);
    const float2 f = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(pair, __NV_E4M3)));
    ou[j] = pack_bf16(f.x * sc, f.y * sc);
  }
  return o;
}

// Eight gated activations from eight gates and ups (same rounding as glu_fwd_kernel).
__device__ __forceinline__ uint4 glu_fwd8(const uint4& gv, const uint4& uv, const QuantGlu& gp, float rs) {
  uint4 o; uint32_t* ou = &o.x; const uint32_t* gu = &gv.x; const uint32_t* uu = &uv.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 g = unpack_bf16(gu[j]), u = unpack_bf16(uu[j]);
    if (gp.limit > 0.f) {
      g.x = fminf(g.x, gp.limit); g.y = fminf(g.y, gp.limit);
      u.x = fminf(fmaxf(u.x, -gp.limit), gp.limit); u.y = fminf(fmaxf(u.y, -gp.limit), gp.limit);
    }
    ou[j] = pack_bf16(act_fwd(g.x, gp.kind) * (u.x + gp.up_offset) * rs,
                      act_fwd(g.y, gp.kind) * (u.y + gp.up_offset) * rs);
  }
  return o;
}
// Eight gradients of the gate (up_half false) or of the up (true) columns (as glu_bwd_kernel).
__device__ __forceinline__ uint4 glu_bwd8(const uint4& gv, const uint4& uv, const uint4& dv, bool up_half,
                                          const QuantGlu& gp) {
  uint4 o; uint32_t* ou = &o.x;
  const uint32_t* gu = &gv.x; const uint32_t* uu = &uv.x; const uint32_t* du = &dv.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 g = unpack_bf16(gu[j]), u = unpack_bf16(uu[j]), d = unpack_bf16(du[j]);
    const float gx[2] = {g.x, g.y}, ux[2] = {u.x, u.y}, dx[2] = {d.x, d.y};
    float r[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      bool g_pass = true, u_pass = true;
      float gg = gx[e], uu_ = ux[e];
      if (gp.limit > 0.f) {
        if (gg > gp.limit) { gg = gp.limit; g_pass = false; }
        if (uu_ > gp.limit) { uu_ = gp.limit; u_pass = false; }
        if (uu_ < -gp.limit) { uu_ = -gp.limit; u_pass = false; }
      }
      float a, da;
      act_both(gg, gp.kind, a, da);
      if (up_half) r[e] = u_pass ? dx[e] * a : 0.f;
      else r[e] = g_pass ? dx[e] * (uu_ + gp.up_offset) * da : 0.f;
    }
    ou[j] = pack_bf16(r[0], r[1]);
  }
  return o;
}

template <int SRC>
__global__ void __launch_bounds__(256, SRC == QSRC_GLU_FWD || SRC == QSRC_GLU_BWD ? QUANT_GLU_CTAS : QUANT_CTAS)
quant_mxfp8_kernel(const __nv_bfloat16* __restrict__ x, long ld_x,
                   const int* __restrict__ row_index,
                   uint8_t* __restrict__ q_row, uint8_t* __restrict__ sf_row,
                   uint8_t* __restrict__ q_col, uint8_t* __restrict__ sf_col,
                   long rows, int cols, long ld_col, long x_batch_stride, QuantGlu gp) {
  // What bounds it is the load / store unit: stores of 8 or 16 bytes per row of the output took a
  // cycle each (65536 x 2048 both ways: 132 us at 75 % of its cycles, 24 instructions per element);
  // with 32-byte stores and a whole block per thread 94 us (copying the bytes would take 83).
  // outputs start on 32-byte boundaries (block offsets are multiples of 32)
  const bool wide = ((reinterpret_cast<uintptr_t>(q_row) | reinterpret_cast<uintptr_t>(q_col)) & 31) == 0;
  __shared__ __align__(128) __nv_bfloat16 tile[QT * QT];
  __shared__ __align__(16) uint8_t sfr[512];
  __shared__ __align__(16) uint8_t sfc[512];
  const int sf_cols_row = ((cols / 32) + 3) & ~3;
  const int sf_cols_col = (int)(((ld_col / 32) + 3) & ~3L);
  if (blockIdx.z > 0) {
    // batched: matrix z of a stack, every output advanced by its own size
    const long z = blockIdx.z;
    x += z * x_batch_stride;
    if (q_row) { q_row += z * rows * cols; sf_row += z * ((rows + 127) / 128) * (sf_cols_row / 4) * 512; }
    if (q_col) { q_col += z * (long)cols * ld_col; sf_col += z * ((cols + 127) / 128) * (sf_cols_col / 4) * 512; }
  }
  const int tid = threadIdx.x;
  const long r0 = (long)blockIdx.y * QT;
  const int c0 = blockIdx.x * QT;
  const int cc = (tid & 15) * 8;  // load: 16 threads per row (8 elements each), 16 rows per pass
  // the place of this thread's piece of row 16 * base + tid / 16: bits 5-6 of the row are base / 2
  const int place0 = qtile_at(tid >> 4, tid & 15);
  auto place = [&](int base) { return (place0 ^ (((base >> 1) << 1) << 3)) + base * 16 * QT; };
  if (SRC == QSRC_MX) {
    // the source is already MXFP8 along its columns (what a peer pushed): dequantise into the
    // tile; the column pass below then quantises along the rows
    const uint8_t* x8 = reinterpret_cast<const uint8_t*>(x);
    const int src_sf_cols = ((cols / 32) + 3) & ~3;
#pragma unroll
    for (int base = 0; base < 8; ++base) {
      const long r = r0 + base * 16 + (tid >> 4);
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r < rows && c0 + cc < cols) {
        const uint2 q = *reinterpret_cast<const uint2*>(x8 + r * ld_x + c0 + cc);
        v = dequant_e4m3x8(q, gp.src_sf[sf_offset(r, (c0 + cc) >> 5, src_sf_cols)]);
      }
      *reinterpret_cast<uint4*>(&tile[place(base)]) = v;
    }
  } else if (SRC == QSRC_PLAIN && gp.row_scale == nullptr) {
    // straight into the tile, all eight pieces of a thread in flight without registers; rows that
    // do not exist are zeros. The gathered rows' numbers are read before the first copy is issued
    // (between the copies each would wait for the one before:
    // 139264 gathered rows of 2048 203 us, so 190; 173 since scaling takes one instruction).
    long src[8];
#pragma unroll
    for (int base = 0; base < 8; ++base) {
      const long r = r0 + base * 16 + (tid >> 4);
      src[base] = r < rows ? (row_index ? (long)row_index[r] : r) : -1;
    }
#pragma unroll
    for (int base = 0; base < 8; ++base) {
      const bool live = src[base] >= 0 && c0 + cc < cols;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&tile[place(base)]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(live ? x + src[base] * ld_x + c0 + cc : x),
                   "r"(live ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (SRC == QSRC_PLAIN) {
#pragma unroll
    for (int base = 0; base < 8; base += 4) {
      uint4 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const long r = r0 + (base + i) * 16 + (tid >> 4);
        long src = r;
        if (row_index && r < rows) src = row_index[r];
        v[i] = make_uint4(0, 0, 0, 0);
        if (r < rows && src >= 0 && c0 + cc < cols) {
          v[i] = *reinterpret_cast<const uint4*>(x + src * ld_x + c0 + cc);
          const float rs = gp.row_scale[r];
          uint32_t* u = &v[i].x;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 t = unpack_bf16(u[j]);
            u[j] = pack_bf16(t.x * rs, t.y * rs);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(&tile[place(base + i)]) = v[i];
    }
  } else {
    // the tile is computed from h (and dout), two rows' loads in flight per thread.
    // GLU_FWD: cols == f, column c pairs h[:, c] with h[:, f + c]. GLU_BWD: cols == 2f and
    // a tile lies in one half (f % 128 == 0): gate gradients, then up gradients.
    const bool up_half = SRC == QSRC_GLU_BWD && c0 >= gp.f;
    const int hc = (up_half ? c0 - gp.f : c0) + cc;  // gate column in h
#pragma unroll 1
    for (int base = 0; base < 8; base += 2) {
      uint4 g[2], u[2], d[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const long r = r0 + (base + i) * 16 + (tid >> 4);
        g[i] = u[i] = d[i] = make_uint4(0, 0, 0, 0);
        if (r < rows && c0 + cc < cols) {
          g[i] = *reinterpret_cast<const uint4*>(x + r * ld_x + hc);
          u[i] = *reinterpret_cast<const uint4*>(x + r * ld_x + gp.f + hc);
          if (SRC == QSRC_GLU_BWD) d[i] = *reinterpret_cast<const uint4*>(gp.dout + r * (long)gp.f + hc);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const long r = r0 + (base + i) * 16 + (tid >> 4);
        uint4 o = make_uint4(0, 0, 0, 0);
        if (r < rows && c0 + cc < cols)
          o = SRC == QSRC_GLU_FWD ? glu_fwd8(g[i], u[i], gp, gp.row_scale ? gp.row_scale[r] : 1.f)
                                  : glu_bwd8(g[i], u[i], d[i], up_half, gp);
        *reinterpret_cast<uint4*>(&tile[place(base + i)]) = o;
      }
    }
  }
  __syncthreads();
  // Both passes give a thread one whole 32-element block: its maximum needs no exchange, the scale is
  // formed once, and it leaves as 32 bytes, four neighbours filling a 128-byte line.
  const int lane = tid & 31, warp = tid >> 5;
  if (q_row) {
    const int cb = lane & 3;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      const int rr = i * 64 + warp * 8 + (lane >> 2);
      const long r = r0 + rr;
      // chunk cb * 4 + k differs from cb * 4 in its two low bits alone, and so does its place
      const int first = qtile_at(rr, cb * 4);
      uint32_t w[16];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 v = *reinterpret_cast<const uint4*>(&tile[first ^ (k << 3)]);
        w[4 * k] = v.x; w[4 * k + 1] = v.y; w[4 * k + 2] = v.z; w[4 * k + 3] = v.w;
      }
      const bool live = r < rows && c0 + cb * 32 < cols;
      const uint8_t e = e8m0_of(amax32(w));
      sfr[(rr & 31) * 16 + (rr >> 5) * 4 + cb] = live ? e : (uint8_t)127;
      if (live) store_e4m3x32(q_row + r * cols + c0 + cb * 32, w, e8m0_inv_bf16(e), wide);
    }
  }
  if (q_col) {
    // A warp takes 8 columns at a time. A transposing ldmatrix hands thread (column t / 4, q = t % 4)
    // rows 2q and 2q + 1 of each 8x8 matrix; matrix m of load j holds the rows 32a + 8j + 2m + b, so
    // after four loads of four the thread has rows 32q .. 32q + 31 of its column, in order.
    const int m = lane >> 3, i = lane & 7;  // this lane addresses row i of matrix m
    const int col = lane >> 2, q = lane & 3;
#pragma unroll 1
    for (int task = 0; task < 2; ++task) {
      const int cg = warp * 2 + task;
      // the swizzle looks at bits 0 and 5-6 of the row: 8 rows further the chunk stays in its place
      const uint32_t first = (uint32_t)__cvta_generic_to_shared(&tile[qtile_at(32 * (i >> 1) + 2 * m + (i & 1), cg)]);
      uint32_t w[16];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t addr = first + j * 8 * QT * 2;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[4 * j]), "=r"(w[4 * j + 1]), "=r"(w[4 * j + 2]), "=r"(w[4 * j + 3]) : "r"(addr));
      }
      const int ccol = cg * 8 + col;
      const bool live = c0 + ccol < cols;
      const uint8_t e = e8m0_of(amax32(w));
      sfc[(ccol & 31) * 16 + (ccol >> 5) * 4 + q] = live ? e : (uint8_t)127;
      if (live && r0 + 32 * q < ld_col)
        store_e4m3x32(q_col + (size_t)(c0 + ccol) * ld_col + r0 + 32 * q, w, e8m0_inv_bf16(e), wide);
    }
  }
  __syncthreads();
  // one whole 512-byte scale tile per output
  if (q_row && tid < 32) {
    uint8_t* dst = sf_row + ((size_t)blockIdx.y * (sf_cols_row >> 2) + blockIdx.x) * 512;
    reinterpret_cast<uint4*>(dst)[tid] = reinterpret_cast<const uint4*>(sfr)[tid];
  }
  if (q_col && tid >= 32 && tid < 64) {
    uint8_t* dst = sf_col + ((size_t)blockIdx.x * (sf_cols_col >> 2) + blockIdx.y) * 512;
    reinterpret_cast<uint4*>(dst)[tid - 32] = reinterpret_cast<const uint4*>(sfc)[tid - 32];
  }
}

// ---------------------------------------------------------------- NVFP4 quantiser
// x [rows, cols] bf16 -> E2M1 codes, two per byte (low nibble first), in blocks of 16 along a
// row with one E4M3 scale each, under one fp32 scale for the tensor (*tensor_scale =
// amax / (6 * 448), taken by the caller's reduction). One thread per block: two 16-byte loads,
// the block's largest magnitude, its scale rounded to E4M3, sixteen values rounded to nearest
// by the hardware's E2M1 conversion, one 8-byte store.
__global__ void quant_nvfp4_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ tensor_scale,
                                   uint8_t* __restrict__ packed, uint8_t* __restrict__ scales, long blocks) {
  const float ts = *tensor_scale;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < blocks; i += (long)gridDim.x * blockDim.x) {
    const uint4 a = *reinterpret_cast<const uint4*>(x + i * 16);
    const uint4 b = *reinterpret_cast<const uint4*>(x + i * 16 + 8);
    float v[16];
    const uint32_t* au = &a.x; const uint32_t* bu = &b.x;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 f = unpack_bf16(au[q]), g = unpack_bf16(bu[q]);
      v[2 * q] = f.x; v[2 * q + 1] = f.y; v[8 + 2 * q] = g.x; v[8 + 2 * q + 1] = g.y;
    }
    float amax = 0.f;
#pragma unroll
    for (int q = 0; q < 16; ++q) amax = fmaxf(amax, fabsf(v[q]));
    const __nv_fp8_storage_t sbyte = __nv_cvt_float_to_fp8(fminf(__fdiv_rn(amax, 6.f * ts), 448.f), __NV_SATFINITE, __NV_E4M3);
    const float scale = __half2float(__half(__nv_cvt_fp8_to_halfraw(sbyte, __NV_E4M3)));
    const float denom = scale * ts;
    uint32_t w[2] = {0u, 0u};
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float lo = denom > 0.f ? __fdiv_rn(v[2 * q], denom) : 0.f;
      const float hi = denom > 0.f ? __fdiv_rn(v[2 * q + 1], denom) : 0.f;
      const uint32_t byte = (uint32_t)__nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
      w[q >> 2] |= (byte & 0xffu) << (8 * (q & 3));
    }
    *reinterpret_cast<uint2*>(packed + i * 8) = make_uint2(w[0], w[1]);
    scales[i] = sbyte;
  }
}

// ---------------------------------------------------------------- cross-entropy
// One block per row of a logits chunk [rows, vocab] (bf16). Writes per-row loss and
// logZ (fp32) and overwrites the logits with dlogits = (softmax - onehot) * grad_scale
// * mask (+ z-loss term), ready for the dX / dW GEMMs.
// A row is walked twice: the running maximum and the sum relative to it in one pass (a lane's sum
// is rescaled only when its maximum moves), then the gradient; the second walk finds most of the row
// in L2. Four 16-byte loads per thread in flight and three blocks per SM: 4096 x 151936 took 840 us
// with separate walks for the maximum and the sum, 576 now (597 at two blocks; one read and one
// write of device memory would take 381). Rows that do not give 512 threads a load each take 128, and many
// rows of up to 4096 entries 256 (2048 x 128: 4.3 us, 10.1 with 512; 2048 x 4096: 12.5 and 16.7).
constexpr int CE_UNROLL = 4;
__device__ __forceinline__ void ce_load8(const uint4& v, float softcap, float (&t)[8]) {
  unpack8(v, t);
  if (softcap > 0.f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) t[j] = softcap * tanhf(t[j] / softcap);
  }
}
template <int CE_THREADS>
__global__ void __launch_bounds__(CE_THREADS, 1536 / CE_THREADS)
ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const int* __restrict__ targets,
                  const float* __restrict__ mask, float* __restrict__ loss,
                  float* __restrict__ logz_out, int vocab, long ld, float grad_scale,
                  float z_weight, float softcap) {
  const long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  uint4* lv = reinterpret_cast<uint4*>(lr);
  const int nvec = vocab / 8;
  __shared__ float red[2][CE_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float mx = -INFINITY, sum = 0.f;
  auto add8 = [&](const uint4& v) {
    float t[8];
    ce_load8(v, softcap, t);
    float top = t[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) top = fmaxf(top, t[j]);
    if (top > mx) {
      sum *= __expf(mx - top);      // 0 the first time: mx is -inf
      mx = top;
    }
    const float ref = mx == -INFINITY ? 0.f : mx;   // only -inf (or NaN) so far: they count 0 (NaN)
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += __expf(t[j] - ref);
  };
  int i = threadIdx.x;
  for (; i + (CE_UNROLL - 1) * CE_THREADS < nvec; i += CE_UNROLL * CE_THREADS) {
    uint4 v[CE_UNROLL];
#pragma unroll
    for (int k = 0; k < CE_UNROLL; ++k) v[k] = lv[i + k * CE_THREADS];
#pragma unroll
    for (int k = 0; k < CE_UNROLL; ++k) add8(v[k]);
  }
  for (; i < nvec; i += CE_THREADS) add8(lv[i]);
  const float wmx = warp_max(mx);
  sum = warp_sum(wmx == mx ? sum : sum * __expf(mx - wmx));
  if (lane == 0) { red[0][warp] = wmx; red[1][warp] = sum; }
  __syncthreads();
  mx = red[0][lane & (CE_THREADS / 32 - 1)];
  const float wsum = red[1][lane & (CE_THREADS / 32 - 1)];
  const float all = warp_max(mx);
  sum = warp_sum(lane < CE_THREADS / 32 ? wsum * __expf(mx - all) : 0.f);
  mx = all;
  const float logz = mx + logf(sum);
  const int tgt = targets[row];
  const float m = mask ? mask[row] : 1.f;
  if (threadIdx.x == 0) {
    float t = __bfloat162float(lr[tgt]);
    if (softcap > 0.f) t = softcap * tanhf(t / softcap);
    loss[row] = (logz - t + z_weight * logz * logz) * m;
    if (logz_out) logz_out[row] = logz;
  }
  __syncthreads();  // the target logit is read before it is overwritten below
  const float gs = grad_scale * m;
  const float zfac = 1.f + 2.f * z_weight * logz;
  const float inv = 1.f / sum;
  auto grad8 = [&](int at, uint4& v) {
    float t[8], cap[8];
    unpack8(v, t);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      cap[j] = 1.f;
      if (softcap > 0.f) {
        const float a = tanhf(t[j] / softcap);
        t[j] = softcap * a;
        cap[j] = 1.f - a * a;
      }
      float p = __expf(t[j] - mx) * inv * zfac;
      if (at * 8 + j == tgt) p -= 1.f;
      t[j] = p * gs * cap[j];
    }
    v = pack8(t);
  };
  i = threadIdx.x;
  for (; i + (CE_UNROLL - 1) * CE_THREADS < nvec; i += CE_UNROLL * CE_THREADS) {
    uint4 v[CE_UNROLL];
#pragma unroll
    for (int k = 0; k < CE_UNROLL; ++k) v[k] = lv[i + k * CE_THREADS];
#pragma unroll
    for (int k = 0; k < CE_UNROLL; ++k) {
      grad8(i + k * CE_THREADS, v[k]);
      lv[i + k * CE_THREADS] = v[k];
    }
  }
  for (; i < nvec; i += CE_THREADS) {
    uint4 v = lv[i];
    grad8(i, v);
    lv[i] = v;
  }
}

// Eight consecutive values as fp32, 16-byte accesses.
template <typename TT> struct Vec8;
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&f)[8]) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&f)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
};
template <> struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    float2 t;
    t = unpack_bf16(v.x); f[0] = t.x; f[1] = t.y;
    t = unpack_bf16(v.y); f[2] = t.x; f[3] = t.y;
    t = unpack_bf16(v.z); f[4] = t.x; f[5] = t.y;
    t = unpack_bf16(v.w); f[6] = t.x; f[7] = t.y;
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&f)[8]) {
    uint4 v;
    v.x = pack_bf16(f[0], f[1]); v.y = pack_bf16(f[2], f[3]);
    v.z = pack_bf16(f[4], f[5]); v.w = pack_bf16(f[6], f[7]);
    *reinterpret_cast<uint4*>(p) = v;
  }
};

// out = bf16(src * *scale), src fp32 or bf16: the head's kept gradients times the incoming one, one
// pass instead of a product and a conversion.
template <typename ST>
__global__ void __launch_bounds__(256)
scale_to_bf16_kernel(const ST* __restrict__ src, const float* __restrict__ scale, __nv_bfloat16* __restrict__ out, long n) {
  const float sc = *scale;
  const long groups = n / 8, stride = (long)gridDim.x * blockDim.x;
  const long first = (long)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll 4
  for (long i = first; i < groups; i += stride) {
    float f[8];
    Vec8<ST>::load(src + i * 8, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] *= sc;
    *reinterpret_cast<uint4*>(out + i * 8) = pack8(f);
  }
  const long tail = groups * 8 + first;
  if (tail < n) out[tail] = __float2bfloat16((float)src[tail] * sc);
}

// ---------------------------------------------------------------- AdamW over flat buffers
// p: fp32 master (or bf16 master when MASTER_BF16), g: bf16 or fp32 grads, optional
// bf16 shadow copy of the updated weights. Moments: fp32, bf16, or 8-bit block-scaled
// (e4m3 values with one E8M0 scale per 32 elements; the second moment is stored as its
// square root so that its dynamic range fits).
// Each lane owns 8 consecutive elements (one 128-bit access of bf16); four adjacent
// lanes form one 32-element scale block of the 8-bit moments and share its amax by
// two shuffles. The buffer length may be ragged: tail elements take scalar paths.
template <typename PT, typename GT, int MOM>
__global__ void adamw_kernel(PT* __restrict__ p, const GT* __restrict__ g, void* __restrict__ m_,
                             void* __restrict__ v_, uint8_t* __restrict__ m_sf, uint8_t* __restrict__ v_sf,
                             __nv_bfloat16* __restrict__ shadow, long n, float lr, float b1, float b2,
                             float eps, float wd, float bc1, float bc2, const float* __restrict__ grad_scale_ptr,
                             float grad_scale_const) {
  const float gscale = grad_scale_ptr ? *grad_scale_ptr * grad_scale_const : grad_scale_const;
  const long groups = (n + 7) / 8;
  // whole warps iterate together so that the 4-lane shuffles below are always converged
  const long warp_groups = (groups + 31) / 32 * 32;
  for (long gi = (long)blockIdx.x * blockDim.x + threadIdx.x; gi < warp_groups; gi += (long)gridDim.x * blockDim.x) {
    const long i0 = gi * 8;
    const bool active = i0 < n;
    const bool full = i0 + 8 <= n;
    const int cnt = active ? (int)min(8L, n - i0) : 0;
    float pw[8], gr[8], pm[8], pv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { pw[j] = 0.f; gr[j] = 0.f; pm[j] = 0.f; pv[j] = 0.f; }
    if (full) {
      Vec8<PT>::load(p + i0, pw);
      Vec8<GT>::load(g + i0, gr);
    } else {
      _Pragma("unroll") for (int j = 0; j < 8; ++j) if (j < cnt) { pw[j] = (float)p[i0 + j]; gr[j] = (float)g[i0 + j]; }
    }
    const long blk = i0 >> 5;
    if (MOM == MOM_F32) {
      if (full) { Vec8<float>::load(reinterpret_cast<float*>(m_) + i0, pm); Vec8<float>::load(reinterpret_cast<float*>(v_) + i0, pv); }
      else _Pragma("unroll") for (int j = 0; j < 8; ++j) if (j < cnt) { pm[j] = reinterpret_cast<float*>(m_)[i0 + j]; pv[j] = reinterpret_cast<float*>(v_)[i0 + j]; }
    } else if (MOM == MOM_BF16) {
      if (full) { Vec8<__nv_bfloat16>::load(reinterpret_cast<__nv_bfloat16*>(m_) + i0, pm); Vec8<__nv_bfloat16>::load(reinterpret_cast<__nv_bfloat16*>(v_) + i0, pv); }
      else _Pragma("unroll") for (int j = 0; j < 8; ++j) if (j < cnt) {
        pm[j] = __bfloat162float(reinterpret_cast<__nv_bfloat16*>(m_)[i0 + j]);
        pv[j] = __bfloat162float(reinterpret_cast<__nv_bfloat16*>(v_)[i0 + j]);
      }
    } else if (active) {
      const float sm = __uint_as_float((uint32_t)max((int)m_sf[blk], 1) << 23);
      const float sv = __uint_as_float((uint32_t)max((int)v_sf[blk], 1) << 23);
      // the eight moment bytes of m and of v travel as two 32-bit words each (no byte arrays:
      // those would live in local memory)
      uint2 mw = make_uint2(0, 0), vw = make_uint2(0, 0);
      if (full) {
        mw = *reinterpret_cast<const uint2*>(reinterpret_cast<uint8_t*>(m_) + i0);
        vw = *reinterpret_cast<const uint2*>(reinterpret_cast<uint8_t*>(v_) + i0);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < cnt) {
            const uint32_t bm = reinterpret_cast<uint8_t*>(m_)[i0 + j], bv = reinterpret_cast<uint8_t*>(v_)[i0 + j];
            if (j < 4) { mw.x |= bm << (8 * j); vw.x |= bv << (8 * j); }
            else { mw.y |= bm << (8 * (j - 4)); vw.y |= bv << (8 * (j - 4)); }
          }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // two values per conversion
        const __nv_fp8x2_storage_t m2 = (__nv_fp8x2_storage_t)(((j < 2 ? mw.x : mw.y) >> (16 * (j & 1))) & 0xffffu);
        const __nv_fp8x2_storage_t v2 = (__nv_fp8x2_storage_t)(((j < 2 ? vw.x : vw.y) >> (16 * (j & 1))) & 0xffffu);
        const float2 fm = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(m2, __NV_E4M3)));
        const float2 fv = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(v2, __NV_E4M3)));
        pm[2 * j] = fm.x * sm; pm[2 * j + 1] = fm.y * sm;
        const float r0 = fv.x * sv, r1 = fv.y * sv;
        pv[2 * j] = r0 * r0; pv[2 * j + 1] = r1 * r1;
      }
    }
    // one approximate square root and one approximate reciprocal per element (the special
    // function unit): the exact forms cost more instructions than the memory traffic hides
    float am = 0.f, av = 0.f;
    float sq[8];
    const float ibc1 = 1.f / bc1, isb2 = rsqrtf(bc2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gg = gr[j] * gscale;
      pm[j] = b1 * pm[j] + (1.f - b1) * gg;
      pv[j] = b2 * pv[j] + (1.f - b2) * gg * gg;
      asm("sqrt.approx.f32 %0, %1;" : "=f"(sq[j]) : "f"(pv[j]));
      const float upd = __fdividef(pm[j] * ibc1, fmaf(sq[j], isb2, eps)) + wd * pw[j];
      pw[j] -= lr * upd;
      if (j < cnt) { am = fmaxf(am, fabsf(pm[j])); av = fmaxf(av, sq[j]); }
    }
    if (full) {
      Vec8<PT>::store(p + i0, pw);
      if (shadow) Vec8<__nv_bfloat16>::store(shadow + i0, pw);
    } else {
      _Pragma("unroll") for (int j = 0; j < 8; ++j) if (j < cnt) { p[i0 + j] = (PT)pw[j]; if (shadow) shadow[i0 + j] = __float2bfloat16(pw[j]); }
    }
    if (MOM == MOM_F32) {
      if (full) { Vec8<float>::store(reinterpret_cast<float*>(m_) + i0, pm); Vec8<float>::store(reinterpret_cast<float*>(v_) + i0, pv); }
      else _Pragma("unroll") for (int j = 0; j < 8; ++j) if (j < cnt) { reinterpret_cast<float*>(m_)[i0 + j] = pm[j]; reinterpret_cast<float*>(v_)[i0 + j] = pv[j]; }
    } else if (MOM == MOM_BF16) {
      if (full) { Vec8<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(m_) + i0, pm); Vec8<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(v_) + i0, pv); }
      else _Pragma("unroll") for (int j = 0; j < 8; ++j) if (j < cnt) {
        reinterpret_cast<__nv_bfloat16*>(m_)[i0 + j] = __float2bfloat16(pm[j]);
        reinterpret_cast<__nv_bfloat16*>(v_)[i0 + j] = __float2bfloat16(pv[j]);
      }
    } else {
      // amax over the 4 lanes of the scale block
      am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1)); am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
      av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 1)); av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 2));
      if (active) {
        const uint8_t em = (uint8_t)max((int)e8m0_of(am), 1), ev = (uint8_t)max((int)e8m0_of(av), 1);
        const float im = e8m0_inv(em), iv = e8m0_inv(ev);
        if ((threadIdx.x & 3) == 0) { m_sf[blk] = em; v_sf[blk] = ev; }
        uint2 mo = make_uint2(0, 0), vo = make_uint2(0, 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t m2 = __nv_cvt_float2_to_fp8x2(make_float2(pm[2 * j] * im, pm[2 * j + 1] * im), __NV_SATFINITE, __NV_E4M3);
          const uint32_t v2 = __nv_cvt_float2_to_fp8x2(make_float2(sq[2 * j] * iv, sq[2 * j + 1] * iv), __NV_SATFINITE, __NV_E4M3);
          if (j < 2) { mo.x |= m2 << (16 * j); vo.x |= v2 << (16 * j); }
          else { mo.y |= m2 << (16 * (j - 2)); vo.y |= v2 << (16 * (j - 2)); }
        }
        if (full) {
          *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(m_) + i0) = mo;
          *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(v_) + i0) = vo;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < cnt) {
              reinterpret_cast<uint8_t*>(m_)[i0 + j] = (uint8_t)(((j < 4 ? mo.x : mo.y) >> (8 * (j & 3))) & 0xff);
              reinterpret_cast<uint8_t*>(v_)[i0 + j] = (uint8_t)(((j < 4 ? vo.x : vo.y) >> (8 * (j & 3))) & 0xff);
            }
        }
      }
    }
  }
}

// sum of squares of a flat buffer into out[0] (fp32 atomics), for the global grad norm
template <typename GT>
__global__ void sumsq_kernel(const GT* __restrict__ g, long n, float* __restrict__ out) {
  float s = 0.f;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float v = (float)g[i];
    s += v * v;
  }
  s = warp_sum(s);
  __shared__ float red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (warp == 0) {
    float v = lane < (blockDim.x >> 5) ? red[lane] : 0.f;
    v = warp_sum(v);
    if (lane == 0) atomicAdd(out, v);
  }
}

// ---------------------------------------------------------------- router top-k
// The k largest of each row of scores [rows, n] (fp32), indices in descending order of value
// (ties: the lower index first). One warp per row; lane l holds columns l, l + 32, ... in
// registers and the warp picks one winner per round by shuffles.
template <int NV>
__global__ void topk_rows_kernel(const float* __restrict__ scores, long* __restrict__ idx, long rows, int n, int k) {
  const int lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const float* sr = scores + row * n;
  float v[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int c = j * 32 + lane;
    v[j] = c < n ? sr[c] : -INFINITY;
    if (v[j] != v[j]) v[j] = -INFINITY;  // a NaN never wins
  }
  for (int round = 0; round < k; ++round) {
    float best = -INFINITY;
    int at = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int c = j * 32 + lane;
      if (c < n && (v[j] > best || (v[j] == best && c < at))) { best = v[j]; at = c; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
    if (lane == 0) idx[row * k + round] = at;
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (j * 32 + lane == at) v[j] = -INFINITY;  // taken: out of the next rounds
  }
}

// ---------------------------------------------------------------- MoE routing
// The picks [n] (expert of each) in expert order, every expert's rows padded to `align`: a stable
// counting sort in three launches that never wait for the host. Each block owns one contiguous
// range of picks; (1) counts per block, (2) one block turns them into each block's first row of
// each expert and the padded offsets, (3) each block places its picks: its eight warps own
// consecutive ranges and walk them 32 picks at a time, ranked by __match_any_sync, so picks of an
// expert stay in order. It replaces a radix sort, a histogram with two host synchronisations and
// some forty small launches: about 300 us with the waits for 131072 picks of 128 experts, now 20.
// A pick outside [0, experts) is reported in the status word (its count is then picks, not waits; the
// host's text for this kernel's number says so); its pos is -2 (see combine_rows).
constexpr int KID_PICKS = 12;
constexpr int PICK_THREADS = 256;
__global__ void __launch_bounds__(PICK_THREADS)
pick_count_kernel(const long long* __restrict__ experts, long n, long per_block, int E, int* __restrict__ counts, Status* st) {
  extern __shared__ int hist[];
  for (int e = threadIdx.x; e < E; e += PICK_THREADS) hist[e] = 0;
  __syncthreads();
  const long lo = blockIdx.x * per_block, hi = min(n, lo + per_block);
  for (long i = lo + threadIdx.x; i < hi; i += PICK_THREADS) {
    const long long e = experts[i];
    if (e >= 0 && e < E) atomicAdd(&hist[e], 1);
    else report_failure(st, KID_PICKS, 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += PICK_THREADS) counts[(long)blockIdx.x * E + e] = hist[e];
}
// counts [blocks, E] become each block's first row; totals [E]; offsets [E + 1]. One block, E <= 1024.
__global__ void __launch_bounds__(1024)
pick_scan_kernel(int* __restrict__ counts, int blocks, int E, int align, int* __restrict__ totals, int* __restrict__ offsets) {
  __shared__ int warp_sums[32];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  int total = 0;
  if (e < E) {
#pragma unroll 8
    for (int b = 0; b < blocks; ++b) total += counts[(long)b * E + e];
    totals[e] = total;
  }
  const int padded = (total + align - 1) / align * align;
  int incl = padded;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += warp_sums[w];
  int at = before + incl - padded;
  if (e >= E) return;
  offsets[e] = at;
  if (e == E - 1) offsets[E] = at + padded;
#pragma unroll 8
  for (int b = 0; b < blocks; ++b) {
    const int c = counts[(long)b * E + e];
    counts[(long)b * E + e] = at;
    at += c;
  }
}
__global__ void __launch_bounds__(PICK_THREADS)
pick_place_kernel(const long long* __restrict__ experts, const float* __restrict__ weights, long n, long per_block, int k,
                  int E, const int* __restrict__ first, const int* __restrict__ totals, const int* __restrict__ offsets,
                  int* __restrict__ row_index, int* __restrict__ pos, float* __restrict__ w_row, long rows) {
  extern __shared__ int seen[];   // [8 warps][E]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = PICK_THREADS / 32;
  for (int e = threadIdx.x; e < NW * E; e += PICK_THREADS) seen[e] = 0;
  __syncthreads();
  int* mine = seen + warp * E;
  const long per_warp = per_block / NW;   // the caller makes per_block a multiple of 32 * NW
  const long lo = blockIdx.x * per_block + warp * per_warp, hi = min(n, lo + per_warp);
  for (long i0 = lo; i0 < hi; i0 += 32) {
    const long i = i0 + lane;
    const long long e = i < hi ? experts[i] : -1;
    const int key = e >= 0 && e < E ? (int)e : -1;
    const unsigned same = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && lane == __ffs(same) - 1) mine[key] += __popc(same);
    __syncwarp();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += PICK_THREADS) {
    int at = first[(long)blockIdx.x * E + e];
#pragma unroll
    for (int w = 0; w < NW; ++w) { const int c = seen[w * E + e]; seen[w * E + e] = at; at += c; }
  }
  __syncthreads();
  for (long i0 = lo; i0 < hi; i0 += 32) {
    const long i = i0 + lane;
    const long long e = i < hi ? experts[i] : -1;
    const int key = e >= 0 && e < E ? (int)e : -1;
    const unsigned same = __match_any_sync(0xffffffffu, key);
    const int dest = key >= 0 ? mine[key] + __popc(same & ((1u << lane) - 1u)) : -2;
    __syncwarp();
    if (key >= 0 && lane == __ffs(same) - 1) mine[key] += __popc(same);
    __syncwarp();
    if (i < hi) {
      pos[i] = dest;
      if (key >= 0) {
        row_index[dest] = (int)(i / k);
        if (w_row) w_row[dest] = weights[i];
      }
    }
  }
  // the rows that no pick fills: every expert's padding and what follows the last expert
  auto clear = [&](long r) { row_index[r] = -1; if (w_row) w_row[r] = 0.f; };
  for (int e = blockIdx.x; e < E; e += gridDim.x)
    for (long r = offsets[e] + totals[e] + threadIdx.x; r < offsets[e + 1]; r += PICK_THREADS) clear(r);
  for (long r = offsets[E] + (long)blockIdx.x * PICK_THREADS + threadIdx.x; r < rows; r += (long)gridDim.x * PICK_THREADS) clear(r);
}

// ---------------------------------------------------------------- MoE gather / combine
// out[r] = x[index[r]] (zero row when index[r] < 0); rows of d bf16, d % 8 == 0.
__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ index,
                                   __nv_bfloat16* __restrict__ out, long rows, int d) {
  const int vec = d / 8;
  const long total = rows * vec;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long r = i / vec; const int c = (int)(i % vec);
    const int src = index[r];
    uint4 v = make_uint4(0, 0, 0, 0);
    if (src >= 0) v = reinterpret_cast<const uint4*>(x + (long)src * d)[c];
    reinterpret_cast<uint4*>(out + r * d)[c] = v;
  }
}
// out[i] = v[pos[i]]; NaN for a pick of no expert (pos < 0).
__global__ void pick_values_kernel(const float* __restrict__ v, const int* __restrict__ pos, float* __restrict__ out, long picks) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < picks; i += (long)gridDim.x * blockDim.x) {
    const int r = pos[i];
    out[i] = r < 0 ? __int_as_float(0x7fffffff) : v[r];
  }
}
// out[t] = sum_k w[t,k] * y[pos[t,k]]  (pos < 0 = dropped pick; -2 = a pick of no expert, which
// makes the row NaN); w may be null (= 1).
__global__ void combine_rows_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ pos,
                                    const float* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                    long tokens, int k, int d) {
  const int vec = d / 8;
  const long total = tokens * vec;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long t = i / vec; const int c = (int)(i % vec);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = 0; j < k; ++j) {
      const int r = pos[t * k + j];
      if (r < 0) {
        if (r == -2) acc[0] = acc[1] = acc[2] = acc[3] = acc[4] = acc[5] = acc[6] = acc[7] = __int_as_float(0x7fffffff);
        continue;
      }
      const float ww = w ? w[t * k + j] : 1.f;
      const uint4 v = reinterpret_cast<const uint4*>(y + (long)r * d)[c];
      const uint32_t* u = &v.x;
#pragma unroll
      for (int q = 0; q < 4; ++q) { const float2 f = unpack_bf16(u[q]); acc[2 * q] += ww * f.x; acc[2 * q + 1] += ww * f.y; }
    }
    uint4 o;
    o.x = pack_bf16(acc[0], acc[1]); o.y = pack_bf16(acc[2], acc[3]);
    o.z = pack_bf16(acc[4], acc[5]); o.w = pack_bf16(acc[6], acc[7]);
    reinterpret_cast<uint4*>(out + t * d)[c] = o;
  }
}

// Backward of the weighted combine, one warp per pick (t, j) with r = pos[t,j]:
//   dy[r] = w[t,j] * dout[t]     dw[t,j] = <y[r], dout[t]>     (dropped picks: dw = 0)
__global__ void combine_bwd_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ dout,
                                   const int* __restrict__ pos, const float* __restrict__ w,
                                   __nv_bfloat16* __restrict__ dy, float* __restrict__ dw,
                                   long picks, int k, int d) {
  const int lane = threadIdx.x & 31;
  const int vec = d / 8;
  for (long i = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < picks;
       i += (long)gridDim.x * (blockDim.x >> 5)) {
    const int r = pos[i];
    if (r < 0) { if (lane == 0 && dw) dw[i] = 0.f; continue; }
    const long t = i / k;
    const float ww = w ? w[i] : 1.f;
    float dot = 0.f;
    for (int c = lane; c < vec; c += 32) {
      const uint4 g = reinterpret_cast<const uint4*>(dout + t * d)[c];
      const uint32_t* gu = &g.x;
      uint4 o; uint32_t* ou = &o.x;
      uint4 yv = make_uint4(0, 0, 0, 0);
      if (dw) yv = reinterpret_cast<const uint4*>(y + (long)r * d)[c];
      const uint32_t* yu = &yv.x;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 gf = unpack_bf16(gu[q]);
        const float2 yf = unpack_bf16(yu[q]);
        dot += gf.x * yf.x + gf.y * yf.y;
        ou[q] = pack_bf16(gf.x * ww, gf.y * ww);
      }
      if (dy) reinterpret_cast<uint4*>(dy + (long)r * d)[c] = o;
    }
    if (dw) {
      dot = warp_sum(dot);
      if (lane == 0) dw[i] = dot;
    }
  }
}

// ---------------------------------------------------------------- launchers
static inline int grid_for(long work, int per_block, int cap = 148 * 16) {
  long g = (work + per_block - 1) / per_block;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

void rmsnorm_fwd(const void* x, const float* w, void* y, float* rstd, long rows, int d, float eps, cudaStream_t s) {
  const int wpb = 8, grid = (int)((rows + wpb - 1) / wpb);
  const bool w16 = reinterpret_cast<uintptr_t>(w) % 16 == 0;
  const int threads = (d / 8 + 31) / 32 * 32;
  const int nv = threads / 32;   // 16-byte pieces of a row per lane; 8 of them are the most held
#define RN_CASE(NV_, COND) \
  if (COND) { rmsnorm_fwd_kernel<NV_><<<grid, wpb * 32, 0, s>>>((const __nv_bfloat16*)x, w, w16, (__nv_bfloat16*)y, rstd, (int)rows, d, eps); return; }
#define RC_CASE(PIECES_, ROWS_, COND) \
  if (COND) { \
    rmsnorm_fwd_columns_kernel<PIECES_, ROWS_><<<(int)((rows + ROWS_ - 1) / ROWS_), PIECES_ == 1 ? threads : (threads / 2 + 31) / 32 * 32, 0, s>>>( \
        (const __nv_bfloat16*)x, w, w16, (__nv_bfloat16*)y, rstd, (int)rows, d, eps); \
    return; }
  // few rows: a block each, so that a lane waits for one load and not for eight (300 x 2048 2.3 us, a warp
  // per row 4.2; at 1000 rows 4.4 either way)
  RC_CASE(1, 1, rows <= 592 && nv > 2 && nv <= 8)
  RN_CASE(1, nv <= 1) RN_CASE(2, nv <= 2) RN_CASE(4, nv <= 4) RN_CASE(8, nv <= 8)
  RC_CASE(1, 2, threads <= 512) RC_CASE(2, 2, threads <= 1024)
#undef RC_CASE
  RN_CASE(0, true)
#undef RN_CASE
}
// Rows of partial sums that the backward leaves for dw (one per block); 0: it adds into dw with atomics.
// 512 threads per SM, as many as are resident with 128 registers. (Atomics of every block into dw
// cost more than the pass itself: 16384 x 2048 took 66 us with them.)
int rmsnorm_bwd_partials(long rows, int d) {
  if (d < 512 || d > 8192 || d % 8 != 0) return 0;
  const int threads = (d / 8 + 31) / 32 * 32, per = threads <= 512 ? 4 : 2;
  return (int)max(1L, min((rows + per - 1) / per, 148L * max(1, 512 / threads)));
}
void rmsnorm_bwd(const void* x, const float* w, const void* dy, const float* rstd, void* dx, float* dw, float* dw_part,
                 long rows, int d, cudaStream_t s) {
  const int blocks = rmsnorm_bwd_partials(rows, d);
  const bool w16 = reinterpret_cast<uintptr_t>(w) % 16 == 0;
  if (blocks > 0) {
    const int threads = (d / 8 + 31) / 32 * 32;
    float* part = dw ? dw_part : nullptr;
#define RB_CASE(THREADS_, ROWS_) \
    rmsnorm_bwd_columns_kernel<THREADS_, ROWS_><<<blocks, threads, 0, s>>>((const __nv_bfloat16*)x, w, w16, \
        (const __nv_bfloat16*)dy, rstd, (__nv_bfloat16*)dx, part, (int)rows, d)
    if (threads <= 256) RB_CASE(256, 4);
    else if (threads <= 512) RB_CASE(512, 4);
    else RB_CASE(1024, 2);
#undef RB_CASE
    if (part) sum_rows_kernel<<<(d + 31) / 32, 1024, 0, s>>>(part, dw, blocks, d);
    return;
  }
  const int wpb = 8;
  int grid = (int)min((rows + wpb - 1) / wpb, 148L * 4);
  if (d % 8 == 0 && d < 512 && w16) {   // gains between 16-byte boundaries: the kernel below
    rmsnorm_bwd_slab_kernel<<<grid, wpb * 32, (size_t)wpb * d * sizeof(float), s>>>((const __nv_bfloat16*)x, w, (const __nv_bfloat16*)dy, rstd, (__nv_bfloat16*)dx, dw, (int)rows, d);
    return;
  }
  rmsnorm_bwd_kernel<<<grid, wpb * 32, d * sizeof(float), s>>>(
      (const __nv_bfloat16*)x, w, (const __nv_bfloat16*)dy, rstd, (__nv_bfloat16*)dx, dw, (int)rows, d);
}
const char* norm_rope(bool bwd, const void* x, const float* w, const float* cs, const float* sn, void* y,
                      float* rstd, const void* dy, float* dw, long tokens, int heads, int D,
                      long stride_x, long stride_y, float eps, cudaStream_t s) {
  const int wpb = 8;
  // heads a lane group takes at once: one where there is one (32768 x 1 x 128: 9.4 us four at a time, 5.7), or
  // where all of them are 256 lanes per SM or less (16 x 32 x 128 2.8 us, 2.2; 509 x 32 x 128 3.1, 3.9)
  const bool single = heads == 1 || tokens * heads * (D / 16) <= 148L * 256;
  const int hc = single ? 1 : bwd ? 2 : 4;
  const long items = tokens * ((heads + hc - 1) / hc), steps = (items + 512 / D - 1) / (512 / D);  // 512 / D items per warp
  const int grid = (int)min((steps + wpb - 1) / wpb, 148L * (bwd ? 2 : 8));
  const bool w16 = reinterpret_cast<uintptr_t>(w) % 16 == 0;
#define NR_LAUNCH(D_, BWD_, HC_) norm_rope_kernel<D_, BWD_, HC_><<<grid, wpb * 32, 0, s>>>((const __nv_bfloat16*)x, w, w16, cs, sn, (__nv_bfloat16*)y, rstd, \
      BWD_ ? (const __nv_bfloat16*)dy : nullptr, BWD_ ? dw : nullptr, tokens, heads, stride_x, stride_y, eps)
#define NR_CASE(D_) \
  if (D == D_) { \
    if (bwd) { if (single) NR_LAUNCH(D_, true, 1); else NR_LAUNCH(D_, true, 2); } \
    else     { if (single) NR_LAUNCH(D_, false, 1); else NR_LAUNCH(D_, false, 4); } \
    return nullptr; }
  NR_CASE(64) NR_CASE(128) NR_CASE(256)
#undef NR_CASE
#undef NR_LAUNCH
  return "norm_rope: head_dim must be 64, 128 or 256";
}
void glu_fwd(const void* h, void* out, const float* row_scale, long rows, int f, int kind, float limit, float up_offset, cudaStream_t s) {
  glu_fwd_kernel<<<grid_for(rows * (f / 8), 256), 256, 0, s>>>((const __nv_bfloat16*)h, (__nv_bfloat16*)out, row_scale, rows, f, kind, limit, up_offset);
}
void glu_bwd(const void* h, const void* dout, void* dh, const float* row_scale, float* d_row_scale, long rows, int f, int kind, float limit, float up_offset, cudaStream_t s) {
  if (d_row_scale) {
#define GR_CASE(TPR_) glu_bwd_rows_kernel<TPR_><<<grid_for(rows, 256 / TPR_, 148 * 16), 256, 0, s>>>((const __nv_bfloat16*)h, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dh, row_scale, d_row_scale, rows, f, kind, limit, up_offset)
    // A warp per row, but for rows that leave most of its lanes idle (65536 x 64: atomics 14.3 us, a warp
    // 34.0, eight threads 16.4; 147456 x 8: 9.6, 64.6, 22.5 with eight) and for rows too few for their warps to fill
    // the GPU (1 x 14336: 8.7, 52.9, a block per row 12.3; 1000 x 2880 73.9, 22.3, 14.3; from 4096 rows on
    // a warp is no slower, and so at 2368 x 768).
    if (rows <= 148 * 8) { if (f >= 768) GR_CASE(256); else GR_CASE(32); }
    else if (f < 64) GR_CASE(1);
    else if (f <= 128) GR_CASE(8);
    else GR_CASE(32);
#undef GR_CASE
  }
  else
    glu_bwd_kernel<<<grid_for(rows * (f / 8), 256), 256, 0, s>>>((const __nv_bfloat16*)h, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dh, row_scale, rows, f, kind, limit, up_offset);
}
void quant_mxfp8(const void* x, long ld_x, const int* row_index, const float* row_scale, uint8_t* q_row, uint8_t* sf_row, uint8_t* q_col, uint8_t* sf_col, long rows, int cols, long ld_col, int batch, long x_batch_stride, cudaStream_t s) {
  const long extent = q_col ? (ld_col > rows ? ld_col : rows) : rows;  // the transposed copy is padded to ld_col
  dim3 grid((cols + 127) / 128, (unsigned)((extent + 127) / 128), batch);
  quant_mxfp8_kernel<QSRC_PLAIN><<<grid, 256, 0, s>>>((const __nv_bfloat16*)x, ld_x, row_index, q_row, sf_row, q_col, sf_col, rows, cols, ld_col, x_batch_stride, QuantGlu{row_scale, nullptr, 0, 0, 0.f, 0.f, nullptr});
}
void requant_mxfp8_cols(const uint8_t* q, const uint8_t* sf, uint8_t* q_col, uint8_t* sf_col, long rows, int cols,
                        long ld_col, cudaStream_t s) {
  const long extent = ld_col > rows ? ld_col : rows;
  dim3 grid((cols + 127) / 128, (unsigned)((extent + 127) / 128), 1);
  quant_mxfp8_kernel<QSRC_MX><<<grid, 256, 0, s>>>((const __nv_bfloat16*)q, cols, nullptr, nullptr, nullptr, q_col, sf_col,
                                                   rows, cols, ld_col, 0, QuantGlu{nullptr, nullptr, 0, 0, 0.f, 0.f, sf});
}
void quant_mxfp8_glu(const void* h, const void* dout, const float* row_scale, uint8_t* q_row, uint8_t* sf_row,
                     uint8_t* q_col, uint8_t* sf_col, long rows, int f, long ld_col, int kind, float limit,
                     float up_offset, cudaStream_t s) {
  const int cols = dout ? 2 * f : f;
  const long extent = q_col ? (ld_col > rows ? ld_col : rows) : rows;
  dim3 grid((cols + 127) / 128, (unsigned)((extent + 127) / 128), 1);
  QuantGlu gp{dout ? nullptr : row_scale, (const __nv_bfloat16*)dout, f, kind, limit, up_offset, nullptr};
  if (dout) quant_mxfp8_kernel<QSRC_GLU_BWD><<<grid, 256, 0, s>>>((const __nv_bfloat16*)h, 2L * f, nullptr, q_row, sf_row, q_col, sf_col, rows, cols, ld_col, 0, gp);
  else quant_mxfp8_kernel<QSRC_GLU_FWD><<<grid, 256, 0, s>>>((const __nv_bfloat16*)h, 2L * f, nullptr, q_row, sf_row, q_col, sf_col, rows, cols, ld_col, 0, gp);
}
void quant_nvfp4(const void* x, const float* tensor_scale, uint8_t* packed, uint8_t* scales, long rows, int cols,
                 cudaStream_t s) {
  const long blocks = rows * (cols / 16);
  quant_nvfp4_kernel<<<grid_for(blocks, 256), 256, 0, s>>>((const __nv_bfloat16*)x, tensor_scale, packed, scales, blocks);
}
void ce_fwd_bwd(void* logits, const int* targets, const float* mask, float* loss, float* logz, long rows, int vocab, long ld, float grad_scale, float z_weight, float softcap, cudaStream_t s) {
#define CE_CASE(THREADS_) ce_fwd_bwd_kernel<THREADS_><<<(unsigned)rows, THREADS_, 0, s>>>((__nv_bfloat16*)logits, targets, mask, loss, logz, vocab, ld, grad_scale, z_weight, softcap)
  if (vocab <= 8 * 128) CE_CASE(128); else if (vocab <= 8 * 512 && rows > 148 * 4) CE_CASE(256); else CE_CASE(512);
#undef CE_CASE
}
void scale_to_bf16(const void* src, bool src_bf16, const float* scale, void* out, long n, cudaStream_t s) {
  const int grid = grid_for(n / 8, 256 * 4, 148 * 8);
  if (src_bf16) scale_to_bf16_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)src, scale, (__nv_bfloat16*)out, n);
  else scale_to_bf16_kernel<float><<<grid, 256, 0, s>>>((const float*)src, scale, (__nv_bfloat16*)out, n);
}
const char* adamw(void* p, bool p_bf16, const void* g, bool g_bf16, void* m, void* v, uint8_t* m_sf, uint8_t* v_sf, int mom,
                  void* shadow, long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2,
                  const float* gscale_ptr, float gscale, cudaStream_t s) {
  const int grid = grid_for((n + 7) / 8, 256, 148 * 32);
#define AW(PT, GT, MOM_) adamw_kernel<PT, GT, MOM_><<<grid, 256, 0, s>>>((PT*)p, (const GT*)g, m, v, m_sf, v_sf, (__nv_bfloat16*)shadow, n, lr, b1, b2, eps, wd, bc1, bc2, gscale_ptr, gscale)
#define AW_MOM(PT, GT) { if (mom == MOM_F32) AW(PT, GT, MOM_F32); else if (mom == MOM_BF16) AW(PT, GT, MOM_BF16); else AW(PT, GT, MOM_FP8); return nullptr; }
  if (!p_bf16 && g_bf16) AW_MOM(float, __nv_bfloat16)
  if (!p_bf16 && !g_bf16) AW_MOM(float, float)
  if (p_bf16 && g_bf16) AW_MOM(__nv_bfloat16, __nv_bfloat16)
  if (p_bf16 && !g_bf16) AW_MOM(__nv_bfloat16, float)
#undef AW_MOM
#undef AW
  return "adamw: unsupported dtypes";
}
void sumsq(const void* g, bool bf16, long n, float* out, cudaStream_t s) {
  const int grid = grid_for(n, 256 * 8, 148 * 8);
  if (bf16) sumsq_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)g, n, out);
  else sumsq_kernel<float><<<grid, 256, 0, s>>>((const float*)g, n, out);
}
const char* topk_rows(const float* scores, long* idx, long rows, int n, int k, cudaStream_t s) {
  const int wpb = 8;
  const unsigned grid = (unsigned)((rows + wpb - 1) / wpb);
#define TK_CASE(NV_) if (n <= NV_ * 32) { topk_rows_kernel<NV_><<<grid, wpb * 32, 0, s>>>(scores, idx, rows, n, k); return nullptr; }
  TK_CASE(1) TK_CASE(2) TK_CASE(4) TK_CASE(8) TK_CASE(16)
#undef TK_CASE
  return "topk_rows: at most 512 columns";
}
int pick_blocks(long n) { return (int)min(128L, (n + 1023) / 1024); }
void sort_picks(const long long* experts, const float* weights, long n, int k, int E, int align, int* row_index, int* pos,
                int* offsets, float* w_row, long rows, int* work, Status* st, cudaStream_t s) {
  const int blocks = pick_blocks(n);
  const long per_block = ((n + blocks - 1) / blocks + 255) / 256 * 256;
  int* totals = work + (long)blocks * E;
  pick_count_kernel<<<blocks, PICK_THREADS, E * sizeof(int), s>>>(experts, n, per_block, E, work, st);
  pick_scan_kernel<<<1, 1024, 0, s>>>(work, blocks, E, align, totals, offsets);
  pick_place_kernel<<<blocks, PICK_THREADS, 8 * E * sizeof(int), s>>>(experts, weights, n, per_block, k, E, work, totals, offsets,
                                                                      row_index, pos, w_row, rows);
}
void pick_values(const float* v, const int* pos, float* out, long picks, cudaStream_t s) {
  pick_values_kernel<<<grid_for(picks, 256), 256, 0, s>>>(v, pos, out, picks);
}
void gather_rows(const void* x, const int* index, void* out, long rows, int d, cudaStream_t s) {
  gather_rows_kernel<<<grid_for(rows * (d / 8), 256), 256, 0, s>>>((const __nv_bfloat16*)x, index, (__nv_bfloat16*)out, rows, d);
}
void combine_bwd(const void* y, const void* dout, const int* pos, const float* w, void* dy, float* dw, long picks, int k, int d, cudaStream_t s) {
  combine_bwd_kernel<<<grid_for(picks, 8), 256, 0, s>>>((const __nv_bfloat16*)y, (const __nv_bfloat16*)dout, pos, w, (__nv_bfloat16*)dy, dw, picks, k, d);
}
void combine_rows(const void* y, const int* pos, const float* w, void* out, long tokens, int k, int d, cudaStream_t s) {
  combine_rows_kernel<<<grid_for(tokens * (d / 8), 256), 256, 0, s>>>((const __nv_bfloat16*)y, pos, w, (__nv_bfloat16*)out, tokens, k, d);
}

}  // namespace bux
