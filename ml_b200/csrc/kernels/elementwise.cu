// Bandwidth-bound kernels of the training step: embedding, RMSNorm (fwd, fused residual-add fwd, bwd), RoPE,
// SwiGLU, fused cross-entropy, AdamW, vision helpers and casts.  All are written for HBM3e streaming:
// 16-byte vector accesses, one pass over DRAM per tensor (second passes over a row hit L1/L2), fp32 math,
// one rounding to bf16 on store.  Formulas follow the reference kernels they replace
// (train/gpt_kernels.cuh: encoder :225-243, rmsnorm :275-458, rope :645-713, swiglu :589-640, CE :1169-1210,
// adamw :1357-1400) but none of the code is shared with them.
#include "../common.cuh"
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include "../no_alloc.h"

#include <algorithm>
#include <cstdio>

MLB_DEFINE_ERROR_WORD(elementwise)

namespace {

__device__ __forceinline__ void load8(const bf16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const bf162* h = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {     // 8 bf16 held packed in four registers
  f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
  f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
  f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
  f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]); u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}
// 8 floats * scale -> 8 E4M3 bytes (round to nearest even, saturating at +-448), one 8-byte store
__device__ __forceinline__ void store8_e4m3(uint8_t* p, const float (&f)[8], float scale) {
  uint2 u;
  u.x = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[0] * scale, f[1] * scale), __NV_SATFINITE, __NV_E4M3) |
        ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[2] * scale, f[3] * scale), __NV_SATFINITE, __NV_E4M3) << 16);
  u.y = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[4] * scale, f[5] * scale), __NV_SATFINITE, __NV_E4M3) |
        ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[6] * scale, f[7] * scale), __NV_SATFINITE, __NV_E4M3) << 16);
  *reinterpret_cast<uint2*>(p) = u;
}

// ------------------------------------------------------------------ embedding
// A token id outside [0, V) (a token file made with a larger vocabulary, a damaged file) would index past the table:
// such a row gets zeros / no gradient, and the error word says so (MLB_ERR_BOUNDS, detail 0xE1 forward, 0xE2 backward,
// 0xCE for a cross-entropy target), so the step that read it fails on the host instead of corrupting memory.
// PER threads a row: a warp, four rows to a block, because with a block per row the rate at which blocks start is the bound (16384 of them take 17 us,
// whatever they do); a block of 128 where few rows leave that rate to spare and a warp would have to go round (the rules stand at the entry points).
// Then the dependent trips of a row are what is left, its id, the table, so four items of each thread are in flight at a time; an unrolled loop is not
// enough, its remainder goes one by one (768 columns are three vectors a lane).  us with the rows in L2: a block per row (96 and 256 threads, single
// additions), a warp in an unrolled loop, this.  Forward 64 x 768 1.11, 1.68, 1.17; 64 x 2048 1.65, 1.69, 1.20; 1003 x 768 1.43, 1.70, 1.54; 16384 x 768
// 17.6, 5.7, 5.6.  Backward, four neighbouring elements an atomic addition where the rows allow it: 64 x 768 1.67, 2.31, 1.27; 64 x 2048 2.54, 4.18, 1.39;
// 1003 x 768 2.34, 2.52, 1.81; 1003 x 1001 2.70, 9.54, 2.40; 16384 x 768 19.1, 10.7, 10.5.  Slower than the block per row: up to 0.1 us forward at 768 columns
// and less than 1184 rows, up to 0.4 backward at some 513 odd columns.
template <int PER, typename T, typename Load, typename Store>
__device__ __forceinline__ void by_fours(int lane, int items, Load load, Store store) {
  for (int i = lane; i < items; i += 4 * PER) {
    T v[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (i + k * PER < items) v[k] = load(i + k * PER);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (i + k * PER < items) store(i + k * PER, v[k]);
  }
}
template <int PER>
__global__ void __launch_bounds__(128) embed_fwd_k(bf16* __restrict__ out, const bf16* __restrict__ wte, const int* __restrict__ ids, long rows, int C, int V) {
  mlb_pdl_sync();
  const int lane = threadIdx.x % PER;
  const long row = (long)blockIdx.x * (128 / PER) + threadIdx.x / PER;
  if (row >= rows) return;
  const int id = ids[row];
  bf16* dst = out + row * C;
  if ((unsigned)id >= (unsigned)V) {
    if (lane == 0) mlb_set_error(MLB_ERR_BOUNDS, 0xE1);
    for (int i = lane; i < C; i += PER) dst[i] = __float2bfloat16(0.f);
    return;
  }
  const bf16* src = wte + (long)id * C;
  if ((C & 7) == 0) {
    by_fours<PER, uint4>(lane, C >> 3, [&](int i) { return reinterpret_cast<const uint4*>(src)[i]; }, [&](int i, uint4 v) { reinterpret_cast<uint4*>(dst)[i] = v; });
  } else if (C <= 4 * PER) {
    by_fours<PER, bf16>(lane, C, [&](int i) { return src[i]; }, [&](int i, bf16 v) { dst[i] = v; });
  } else {      // (several trips by fours: 16384 x 513 9.1 us, so 6.2)
    for (int i = lane; i < C; i += PER) dst[i] = src[i];
  }
}
template <int PER>
__global__ void __launch_bounds__(128) embed_bwd_k(float* __restrict__ dwte, const bf16* __restrict__ dout, const int* __restrict__ ids, long rows, int C,
                                                   int V, int T, int n_pre, bool vec) {
  mlb_pdl_sync();
  const int lane = threadIdx.x % PER;
  const long row = (long)blockIdx.x * (128 / PER) + threadIdx.x / PER;
  if (row >= rows || (n_pre > 0 && (int)(row % T) < n_pre)) return;
  const int id = ids[row];
  if ((unsigned)id >= (unsigned)V) {
    if (lane == 0) mlb_set_error(MLB_ERR_BOUNDS, 0xE2);
    return;
  }
  float* dst = dwte + (long)id * C;
  const bf16* src = dout + row * C;
  if (vec)
    by_fours<PER, uint2>(lane, C >> 2, [&](int i) { return reinterpret_cast<const uint2*>(src)[i]; }, [&](int i, uint2 u) {
      asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + i * 4), "f"(__uint_as_float(u.x << 16)),
                   "f"(__uint_as_float(u.x & 0xffff0000u)), "f"(__uint_as_float(u.y << 16)), "f"(__uint_as_float(u.y & 0xffff0000u)) : "memory");
    });
  else
    by_fours<PER, bf16>(lane, C, [&](int i) { return src[i]; }, [&](int i, bf16 v) { atomicAdd(dst + i, __bfloat162float(v)); });
}
__global__ void set_prefix_k(bf16* __restrict__ x, const bf16* __restrict__ prefix, int B, int T, int n_pre, int C) {
  mlb_pdl_sync();
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long n = (long)B * n_pre * C;
  if (i >= n) return;
  int c = i % C;
  long r = i / C;
  int b = r / n_pre, p = r % n_pre;
  x[((long)b * T + p) * C + c] = prefix[i];
}
__global__ void gather_prefix_k(bf16* __restrict__ dprefix, const bf16* __restrict__ dresid, int B, int T, int n_pre, int C) {
  mlb_pdl_sync();
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long n = (long)B * n_pre * C;
  if (i >= n) return;
  int c = i % C;
  long r = i / C;
  int b = r / n_pre, p = r % n_pre;
  dprefix[i] = dresid[((long)b * T + p) * C + c];
}

// ------------------------------------------------------------------ RMSNorm forward (one warp per row)
// ADD: resid = a + b is stored (bf16) and the norm is taken over the un-rounded fp32 sum.
// NV > 0: C = NV * 256; the whole row (and the weight vector's slice) is fetched with all loads in flight at once and
// stays in registers between the sum of squares and the scaling - one read of the inputs instead of two.
template <bool ADD, bool F8 = false, int NV = 0>
__global__ void __launch_bounds__(256) rmsnorm_fwd_k(bf16* __restrict__ out, float* __restrict__ rstd, bf16* __restrict__ resid,
                                                     const bf16* __restrict__ a, const bf16* __restrict__ b,
                                                     const bf16* __restrict__ w, long rows, int C, float eps,
                                                     uint8_t* __restrict__ out8 = nullptr, float s8 = 1.f) {
  mlb_pdl_sync();
  const int lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const bf16* pa = a + row * C;
  const bf16* pb = ADD ? b + row * C : nullptr;
  float ss = 0.f;
  if constexpr (NV > 0) {
    uint4 ra[NV], rb[NV], rw[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const int i = (v * 32 + lane) * 8;
      ra[v] = *reinterpret_cast<const uint4*>(pa + i);
      if (ADD) rb[v] = *reinterpret_cast<const uint4*>(pb + i);
      rw[v] = __ldg(reinterpret_cast<const uint4*>(w + i));
    }
    float x[NV][8];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      unpack8(ra[v], x[v]);
      if (ADD) {
        float y[8];
        unpack8(rb[v], y);
#pragma unroll
        for (int j = 0; j < 8; j++) x[v][j] += y[j];
        store8(resid + row * C + (v * 32 + lane) * 8, x[v]);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) ss += x[v][j] * x[v][j];
    }
    ss = warp_sum(ss);
    const float r = rsqrtf(ss / (float)C + eps);
    if (lane == 0) rstd[row] = r;
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const int i = (v * 32 + lane) * 8;
      float ww[8];
      unpack8(rw[v], ww);
#pragma unroll
      for (int j = 0; j < 8; j++) x[v][j] = x[v][j] * r * ww[j];
      store8(out + row * C + i, x[v]);
      if (F8) store8_e4m3(out8 + row * C + i, x[v], s8);
    }
    return;
  }
  if ((C & 7) == 0) {
    for (int i = lane * 8; i < C; i += 256) {
      float x[8];
      load8(pa + i, x);
      if (ADD) {
        float y[8];
        load8(pb + i, y);
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] += y[j];
        store8(resid + row * C + i, x);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) ss += x[j] * x[j];
    }
    ss = warp_sum(ss);
    const float r = rsqrtf(ss / (float)C + eps);
    if (lane == 0) rstd[row] = r;
    for (int i = lane * 8; i < C; i += 256) {
      float x[8], ww[8];
      load8(pa + i, x);
      if (ADD) {
        float y[8];
        load8(pb + i, y);
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] += y[j];
      }
      load8(w + i, ww);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] = x[j] * r * ww[j];
      store8(out + row * C + i, x);
      if (F8) store8_e4m3(out8 + row * C + i, x, s8);     // E4M3 copy of the fp32 values for the 8-bit forward GEMM
    }
  } else {
    for (int i = lane; i < C; i += 32) {
      float x = __bfloat162float(pa[i]);
      if (ADD) { x += __bfloat162float(pb[i]); resid[row * C + i] = __float2bfloat16(x); }
      ss += x * x;
    }
    ss = warp_sum(ss);
    const float r = rsqrtf(ss / (float)C + eps);
    if (lane == 0) rstd[row] = r;
    for (int i = lane; i < C; i += 32) {
      float x = __bfloat162float(pa[i]);
      if (ADD) x += __bfloat162float(pb[i]);
      const float y = x * r * __bfloat162float(w[i]);
      out[row * C + i] = __float2bfloat16(y);
      if (F8) out8[row * C + i] = (uint8_t)__nv_cvt_float_to_fp8(y * s8, __NV_SATFINITE, __NV_E4M3);
    }
  }
}

// ------------------------------------------------------------------ LayerNorm (the prototype's norm: csrc/kernels/layer_norm_kernel.cu:12-87)
// y = (x - mean) * rstd * w + b over the last dimension; one warp per row, statistics in fp32, mean / rstd saved for backward.
// NV > 0: C = NV * 256, the row (and the slices of w and b) fetched once, 16 bytes a load; else any C, element by element.  Both add a row up in the
// same order, every 32nd element by a lane and then the lanes: the row turns through shared memory for it.  The bits are
// those of the element-wise form then, whatever the alignment.  3152 x 768 4.9 -> 4.1 us, 16384 x 768 14.5 -> 9.5, 16384 x 2048 45.6 -> 30.0 (a
// lane that adds the eight neighbours it has loaded takes 2.8, 7.5 and 35.4, in another order: its bf16 roundings go other ways, which a
// block of the image encoder makes 2.5e-3 of its outputs).
template <int NV>
__global__ void __launch_bounds__(256) layernorm_fwd_k(bf16* __restrict__ out, float* __restrict__ mean, float* __restrict__ rstd,
                                                       const bf16* __restrict__ x, const bf16* __restrict__ w, const bf16* __restrict__ b,
                                                       long rows, int C, float eps) {
  mlb_pdl_sync();
  const int lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const bf16* px = x + row * C;
  if constexpr (NV > 0) {
    __shared__ __align__(16) bf16 turn[8][NV * 256];
    bf16* mine = turn[threadIdx.x >> 5];
    uint4 rx[NV], rw[NV], rb[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const int i = (v * 32 + lane) * 8;
      rx[v] = *reinterpret_cast<const uint4*>(px + i);
      rw[v] = __ldg(reinterpret_cast<const uint4*>(w + i));
      rb[v] = b ? __ldg(reinterpret_cast<const uint4*>(b + i)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int v = 0; v < NV; v++) *reinterpret_cast<uint4*>(mine + (v * 32 + lane) * 8) = rx[v];
    __syncwarp();
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV * 8; i++) s += __bfloat162float(mine[i * 32 + lane]);
    const float mu = warp_sum(s) / (float)C;
#pragma unroll
    for (int i = 0; i < NV * 8; i++) { const float d = __bfloat162float(mine[i * 32 + lane]) - mu; ss += d * d; }
    const float r = rsqrtf(warp_sum(ss) / (float)C + eps);
    if (lane == 0) { mean[row] = mu; rstd[row] = r; }
#pragma unroll
    for (int v = 0; v < NV; v++) {
      float f[8], ww[8], bb[8];
      unpack8(rx[v], f);
      unpack8(rw[v], ww);
      unpack8(rb[v], bb);
#pragma unroll
      for (int j = 0; j < 8; j++) f[j] = (f[j] - mu) * r * ww[j] + bb[j];
      store8(out + row * C + (v * 32 + lane) * 8, f);
    }
    return;
  }
  float s = 0.f;
  for (int i = lane; i < C; i += 32) s += __bfloat162float(px[i]);
  const float mu = warp_sum(s) / (float)C;
  float ss = 0.f;
  for (int i = lane; i < C; i += 32) { const float d = __bfloat162float(px[i]) - mu; ss += d * d; }
  const float r = rsqrtf(warp_sum(ss) / (float)C + eps);
  if (lane == 0) { mean[row] = mu; rstd[row] = r; }
  for (int i = lane; i < C; i += 32) {
    const float y = (__bfloat162float(px[i]) - mu) * r * __bfloat162float(w[i]) + (b ? __bfloat162float(b[i]) : 0.f);
    out[row * C + i] = __float2bfloat16(y);
  }
}
// dx = rstd * (g - mean(g) - xhat * mean(g * xhat)) with g = dy * w, xhat = (x - mean) * rstd; dw += sum dy * xhat, db += sum dy.
// One warp per row; a block folds its rows' dw / db contributions in shared memory (C floats each) before the fp32 atomics.
__global__ void __launch_bounds__(256) layernorm_bwd_k(bf16* __restrict__ dx, float* __restrict__ dw, float* __restrict__ db,
                                                       const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                       const float* __restrict__ mean, const float* __restrict__ rstd, long rows, int C) {
  extern __shared__ float sh[];     // dw partial [C], db partial [C]
  float* sdw = sh;
  float* sdb = sh + C;
  for (int i = threadIdx.x; i < 2 * C; i += blockDim.x) sh[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row < rows) {
    const float mu = mean[row], r = rstd[row];
    const bf16* px = x + row * C;
    const bf16* pd = dy + row * C;
    float sg = 0.f, sgx = 0.f;
    for (int i = lane; i < C; i += 32) {
      const float g = __bfloat162float(pd[i]) * __bfloat162float(w[i]), xh = (__bfloat162float(px[i]) - mu) * r;
      sg += g; sgx += g * xh;
    }
    sg = warp_sum(sg) / (float)C;
    sgx = warp_sum(sgx) / (float)C;
    for (int i = lane; i < C; i += 32) {
      const float d = __bfloat162float(pd[i]), xh = (__bfloat162float(px[i]) - mu) * r;
      dx[row * C + i] = __float2bfloat16(r * (d * __bfloat162float(w[i]) - sg - xh * sgx));
      atomicAdd(&sdw[i], d * xh);
      if (db) atomicAdd(&sdb[i], d);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    atomicAdd(&dw[i], sdw[i]);
    if (db) atomicAdd(&db[i], sdb[i]);
  }
}

// ------------------------------------------------------------------ RMSNorm backward, ONE launch, deterministic
// dx = add + rstd*w*dy - x*rstd^3/C * sum_c(dy*w*x);   dw[c] += sum_rows dy*x*rstd.
// Each block walks a strided set of rows (warp per row) keeping per-column dw partial sums in registers/shared
// memory, writes its partial row to `partial[block][C]`; the partial rows are then folded into dw in a fixed order
// by whichever blocks finish last (see the end of the kernel).  Scratch: `partial` = (gridDim.x + RMS_GROUPS) * C
// floats, `ticket` = 1 + RMS_GROUPS ints that are 0 on entry and left 0 on exit.
constexpr int RMS_GROUPS = 16;
// Up to 32 blocks (256 rows) there is one group, and its last block adds the partial rows up with all of its threads.
// VPL = C / 256 (vectors of 8 per lane) up to 3; PART: one vector per lane of rows narrower than 256 (C % 8 == 0); 0 = generic C (scalar path).
template <int VPL, bool PART = false>
__global__ void __launch_bounds__(256, 2) rmsnorm_bwd_k(bf16* __restrict__ dx, float* __restrict__ dw, const bf16* __restrict__ dy,
                                                     const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                     const float* __restrict__ rstd, const bf16* __restrict__ add, long rows,
                                                     int C, float* __restrict__ partial, int* __restrict__ ticket) {
  mlb_pdl_sync();
  extern __shared__ float sh[];  // C floats: block-level dw partial
  __shared__ int is_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  for (int i = threadIdx.x; i < C; i += blockDim.x) sh[i] = 0.f;
  __syncthreads();
  const float invC = 1.f / (float)C;
  if (VPL > 0) {
    constexpr int NV = VPL > 0 ? VPL : 1;
    constexpr bool CACHE_W = NV <= 2;  // the weight vector stays in registers (two resident blocks per SM leave 128 per thread)
    constexpr int NW = CACHE_W ? NV : 1;
    float acc[NV][8];
    float ww[NW][8] = {};
    const bool mine = !PART || lane * 8 < C;      // this lane has columns
#pragma unroll
    for (int v = 0; v < NV; v++) {
      if (CACHE_W && mine) load8(w + (v * 32 + lane) * 8, ww[v]);
#pragma unroll
      for (int j = 0; j < 8; j++) acc[v][j] = 0.f;
    }
    for (long row = (long)blockIdx.x * nwarp + warp; row < rows; row += (long)gridDim.x * nwarp) {
      const float r = rstd[row];
      // The row's x, dy and residual-stream gradient stay in registers PACKED (four registers per eight values) between
      // the two passes, and every load of the row is issued before the row's reduction: `add` does not depend on it, and
      // fetching it only afterwards cost a second DRAM round trip per row.
      uint4 xr[NV], dr[NV], ar[NV];
      float dot = 0.f;
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const long off = row * C + (v * 32 + lane) * 8;
        const int cw = CACHE_W ? v : 0;
        xr[v] = mine ? *reinterpret_cast<const uint4*>(x + off) : make_uint4(0, 0, 0, 0);
        dr[v] = mine ? *reinterpret_cast<const uint4*>(dy + off) : make_uint4(0, 0, 0, 0);
        ar[v] = add && mine ? *reinterpret_cast<const uint4*>(add + off) : make_uint4(0, 0, 0, 0);
        if (!CACHE_W) load8(w + (v * 32 + lane) * 8, ww[0]);
        float xf[8], df[8];
        unpack8(xr[v], xf);
        unpack8(dr[v], df);
#pragma unroll
        for (int j = 0; j < 8; j++) dot += df[j] * ww[cw][j] * xf[j];
      }
      dot = warp_sum(dot);
      const float k = r * r * r * invC * dot;
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const long off = row * C + (v * 32 + lane) * 8;
        const int cw = CACHE_W ? v : 0;
        if (!CACHE_W) load8(w + (v * 32 + lane) * 8, ww[0]);
        float xf[8], df[8], o[8];
        unpack8(xr[v], xf);
        unpack8(dr[v], df);
        unpack8(ar[v], o);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          o[j] += df[j] * ww[cw][j] * r - xf[j] * k;
          acc[v][j] += df[j] * xf[j] * r;
        }
        if (mine) store8(dx + off, o);
      }
    }
    // fold the 8 warps' register partials in warp order (deterministic)
    for (int wv = 0; wv < nwarp; wv++) {
      if (warp == wv && mine) {
#pragma unroll
        for (int v = 0; v < NV; v++)
#pragma unroll
          for (int j = 0; j < 8; j++) sh[(v * 32 + lane) * 8 + j] += acc[v][j];
      }
      __syncthreads();
    }
  } else {
    for (long row = (long)blockIdx.x * nwarp + warp; row < rows; row += (long)gridDim.x * nwarp) {
      const float r = rstd[row];
      float dot = 0.f;
      for (int i = lane; i < C; i += 32)
        dot += __bfloat162float(dy[row * C + i]) * __bfloat162float(w[i]) * __bfloat162float(x[row * C + i]);
      dot = warp_sum(dot);
      const float k = r * r * r * invC * dot;
      for (int i = lane; i < C; i += 32) {
        float d = __bfloat162float(dy[row * C + i]), xx = __bfloat162float(x[row * C + i]);
        float o = d * __bfloat162float(w[i]) * r - xx * k;
        if (add) o += __bfloat162float(add[row * C + i]);
        dx[row * C + i] = __float2bfloat16(o);
        atomicAdd(&sh[i], d * xx * r);  // shared-memory atomics; this path is for odd C only
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < C; i += blockDim.x) partial[(long)blockIdx.x * C + i] = sh[i];
  // Two-level fold, deterministic and parallel: blocks form RMS_GROUPS groups by index; the block that arrives last in
  // its group sums the group's partial rows in index order into gpartial[group]; the block that completes the last
  // group sums the group rows in order into dw.  Who does the summing depends on timing, the summation order does not.
  const int nb = (int)gridDim.x;
  const int gsz = nb <= 32 ? nb : (nb + RMS_GROUPS - 1) / RMS_GROUPS;
  const int grp = blockIdx.x / gsz;
  const int g_lo = grp * gsz, g_hi = min(nb, g_lo + gsz);
  const int ngroups = (nb + gsz - 1) / gsz;
  float* gpartial = partial + (long)nb * C;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = (atomicAdd(&ticket[1 + grp], 1) == (g_hi - g_lo) - 1);
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  if (PART && nb <= 32) {
    // slice q of the threads takes rows q, q + slices, ...; the slices are added in order (C < 256: at least four of them, at most 1024 floats)
    const int vecs = C >> 2, slices = (int)blockDim.x / vecs, q = threadIdx.x / vecs, c = threadIdx.x % vecs * 4;
    if (q < slices) {
      float a[4] = {};
#pragma unroll 8
      for (int b = q; b < nb; b += slices) {
        const float4 p = __ldcg(reinterpret_cast<const float4*>(&partial[(long)b * C + c]));
        a[0] += p.x; a[1] += p.y; a[2] += p.z; a[3] += p.w;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) sh[q * C + c + j] = a[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < C; i += blockDim.x) {
      float t = 0.f;
      for (int g = 0; g < slices; g++) t += sh[g * C + i];
      dw[i] += t;
    }
    if (threadIdx.x == 0) ticket[1] = 0;
    return;
  }
  const bool vec4 = ((C & 3) == 0) && ((reinterpret_cast<uintptr_t>(dw) & 15) == 0) && ((reinterpret_cast<uintptr_t>(partial) & 15) == 0);
  for (int c = threadIdx.x * 4; c < C; c += blockDim.x * 4) {
    if (vec4) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int b = g_lo; b < g_hi; b++) {
        const float4 p = __ldcg(reinterpret_cast<const float4*>(&partial[(long)b * C + c]));
        a.x += p.x; a.y += p.y; a.z += p.z; a.w += p.w;
      }
      *reinterpret_cast<float4*>(&gpartial[(long)grp * C + c]) = a;
    } else {
      for (int cc = c; cc < min(C, c + 4); cc++) {
        float a = 0.f;
        for (int b = g_lo; b < g_hi; b++) a += __ldcg(&partial[(long)b * C + cc]);
        gpartial[(long)grp * C + cc] = a;
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    ticket[1 + grp] = 0;
    is_last = (atomicAdd(&ticket[0], 1) == ngroups - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  for (int c = threadIdx.x * 4; c < C; c += blockDim.x * 4) {
    if (vec4) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int g2 = 0; g2 < ngroups; g2++) {
        const float4 p = __ldcg(reinterpret_cast<const float4*>(&gpartial[(long)g2 * C + c]));
        a.x += p.x; a.y += p.y; a.z += p.z; a.w += p.w;
      }
      float4 d = *reinterpret_cast<float4*>(&dw[c]);
      d.x += a.x; d.y += a.y; d.z += a.z; d.w += a.w;
      *reinterpret_cast<float4*>(&dw[c]) = d;
    } else {
      for (int cc = c; cc < min(C, c + 4); cc++) {
        float a = 0.f;
        for (int g2 = 0; g2 < ngroups; g2++) a += __ldcg(&gpartial[(long)g2 * C + cc]);
        dw[cc] += a;
      }
    }
  }
  if (threadIdx.x == 0) ticket[0] = 0;
}

// ------------------------------------------------------------------ column sums in two launches, deterministic
// 16 bytes global -> shared without a register; `bytes` 0: zeros, nothing is read.  The copying thread itself reads them back after its wait.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes = 16) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// Ring of the norm backward kernels: two stages of 256 threads x `vecs` 16-byte vectors, a thread's own
static constexpr int norm_ring_bytes(int vecs) { return 2 * 256 * 16 * vecs; }

// Norm backward over whole rows per thread group: C / 8 threads share a row, each owning 8 columns for all of the group's rows, so the
// column sums (dw, and db of LayerNorm) stay in 8 (16) registers and need no folding over a warp's rows.  Three rows at a time:
// their 6-9 16-byte loads are in flight together and their dots cost one barrier.  One warp per row (rmsnorm_bwd_k)
// needs C / 4 accumulators per lane, which at C = 2048 spill: 72 us for 16384 rows against 44 here and 4 for the fold.
// Partial sums: partial[block][C (RMS) | 2 C (LN: dw, db)], added up by fold_cols_k.
// Shapes: C % 256 == 0 and C <= 2048 (whole warps, at most 256 threads a row).
constexpr int NB_ROWS = 3;
template <bool LN>
__global__ void __launch_bounds__(256, 2) norm_bwd_rows_k(bf16* __restrict__ dx, const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                                          const bf16* __restrict__ w, const float* __restrict__ mean,
                                                          const float* __restrict__ rstd, const bf16* __restrict__ add, long rows, int C,
                                                          float* __restrict__ partial) {
  mlb_pdl_sync();
  __shared__ float red[2][NB_ROWS][2][8];
  __shared__ float fold[2048];
  const int gt = C >> 3, G = blockDim.x / gt, grp = threadIdx.x / gt, t = threadIdx.x % gt;      // group = the threads of one row
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, w0 = grp * (gt >> 5), nw = gt >> 5;
  float aw[8], ab[8];
  const uint4 wr = *reinterpret_cast<const uint4*>(w + t * 8);
#pragma unroll
  for (int j = 0; j < 8; j++) aw[j] = ab[j] = 0.f;
  const float invC = 1.f / (float)C;
  int buf = 0;
  // The next rows come into the thread's own places in shared memory (in registers they spill) while these are reduced and stored: with
  // loads only at the top of a round the memory idles meanwhile.  16384 x 2048, 201 MB: 58.8 -> 43.9 us, 3152 x 768 LayerNorm 8.3 -> 7.6, without the fold
  extern __shared__ uint4 norm_ring[];
  uint4* ring = norm_ring + threadIdx.x;
  constexpr int NT = LN ? 2 : 3;      // tensors
  const long step = (long)gridDim.x * G * NB_ROWS, base0 = ((long)blockIdx.x * G + grp) * NB_ROWS;
  float mn[NB_ROWS], rn[NB_ROWS];
  auto fetch = [&](long base, int st) {
    if (base < rows) {
#pragma unroll
      for (int k = 0; k < NB_ROWS; k++) {
        const bool live = base + k < rows;
        const size_t off = (size_t)(live ? base + k : base) * C + t * 8;
        uint4* to = ring + (st * NB_ROWS + k) * NT * 256;
        cp_async16(to, x + off);
        cp_async16(to + 256, dy + off, live ? 16 : 0);      // a row past the end adds nothing
        if (!LN && add) cp_async16(to + 512, add + off);
        rn[k] = rstd[live ? base + k : base];
        if (LN) mn[k] = mean[live ? base + k : base];
      }
    }
    cp_async_commit();
  };
  fetch(base0, 0);
  for (long base = base0; base < rows; base += step, buf ^= 1) {
    uint4 xr[NB_ROWS], dr[NB_ROWS];
    float mu[NB_ROWS], rs[NB_ROWS];
#pragma unroll
    for (int k = 0; k < NB_ROWS; k++) {
      rs[k] = rn[k];
      if (LN) mu[k] = mn[k];
    }
    fetch(base + step, buf ^ 1);
    cp_async_wait<1>();
#pragma unroll
    for (int k = 0; k < NB_ROWS; k++) {
      const uint4* from = ring + (buf * NB_ROWS + k) * NT * 256;
      xr[k] = from[0];
      dr[k] = from[256];
    }
#pragma unroll
    for (int k = 0; k < NB_ROWS; k++) {
      float xf[8], df[8], ww[8], s = 0.f, sx = 0.f;
      unpack8(wr, ww);
      unpack8(xr[k], xf);
      unpack8(dr[k], df);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float g = df[j] * ww[j];
        if (LN) { s += g; sx += g * ((xf[j] - mu[k]) * rs[k]); }
        else sx += g * xf[j];
      }
      sx = warp_sum(sx);
      if (LN) s = warp_sum(s);
      if (lane == 0) {
        red[buf][k][0][warp] = sx;
        if (LN) red[buf][k][1][warp] = s;
      }
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(gt) : "memory");      // (two buffers: one barrier per round is enough)
#pragma unroll
    for (int k = 0; k < NB_ROWS; k++) {
      if (base + k >= rows) break;
      float s = 0.f, sx = 0.f;
      for (int i = 0; i < nw; i++) {
        sx += red[buf][k][0][w0 + i];
        if (LN) s += red[buf][k][1][w0 + i];
      }
      float xf[8], df[8], ww[8], o[8];
      unpack8(wr, ww);
      unpack8(xr[k], xf);
      unpack8(dr[k], df);
      const float r = rs[k];
      if (LN) {
        s *= invC;
        sx *= invC;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float xh = (xf[j] - mu[k]) * r;
          o[j] = r * (df[j] * ww[j] - s - xh * sx);
          aw[j] += df[j] * xh;
          ab[j] += df[j];
        }
      } else {
        const float kk = r * r * r * invC * sx;
        unpack8(add ? ring[((buf * NB_ROWS + k) * NT + 2) * 256] : make_uint4(0, 0, 0, 0), o);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          o[j] += df[j] * ww[j] * r - xf[j] * kk;
          aw[j] += df[j] * xf[j] * r;
        }
      }
      store8(dx + (size_t)(base + k) * C + t * 8, o);
    }
  }
  // the block's groups in order
  float* out = partial + (size_t)blockIdx.x * (LN ? 2 * C : C);
#pragma unroll
  for (int half = 0; half < (LN ? 2 : 1); half++) {
    const float* acc = half ? ab : aw;
    for (int g = 0; g < G; g++) {
      if (grp == g) {
#pragma unroll
        for (int j = 0; j < 8; j++) fold[t * 8 + j] = acc[j] + (g ? fold[t * 8 + j] : 0.f);
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < C; i += blockDim.x) out[half * C + i] = fold[i];
    __syncthreads();
  }
}
// partial[split][N]: column sums of x[M, N] over the split's rows; a warp takes 256 columns of every 8th row
__global__ void __launch_bounds__(256) colsum_k(float* __restrict__ partial, const bf16* __restrict__ x, long M, int N) {
  mlb_pdl_sync();
  __shared__ float red[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = (blockIdx.x * 32 + lane) * 8;
  const long per = (M + gridDim.y - 1) / gridDim.y, r0 = per * blockIdx.y, r1 = min(M, r0 + per);
  float a[8] = {};
  if (c < N) {
#pragma unroll 4
    for (long r = r0 + warp; r < r1; r += 8) {
      float f[8];
      load8(x + (size_t)r * N + c, f);
#pragma unroll
      for (int j = 0; j < 8; j++) a[j] += f[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) red[warp][lane * 8 + j] = a[j];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col >= N) return;
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) s += red[i][threadIdx.x];
  partial[(size_t)blockIdx.y * N + col] = s;
}
// The partial rows added up in a fixed order: columns [0, C) to dw, [C, W) to db (either may be null).  bf16: rounded and stored;
// fp32: added to what is there.  A block takes 32 columns; slice q of eight adds rows q, q + 8, ... and the slices are added in order.
// Bound by latency, so the rows come in one trip of FOLD_ROWS loads a thread: up to 80 rows to eight warps, each of which adds what it loads
// (with 32: column sums of 1003 x 4096 4.5 -> 4.9 us); more rows, 296 at most here, to 32 warps, from which they wait in shared memory for the
// eight that add them (with 8, four trips; norm backward and fold of 3152 x 768 9.3 -> 8.5 us, LayerNorm 10.4 -> 9.3, 16384 x 768 20.2 -> 19.0).
// TREE: for RMSNorm's fp32 dw, where no order is promised: as many slices as warps, a trip's loads and the slices added as trees
// (16384 x 768 normal numbers: off by 1.7e-5 rms, 2.2e-5 in the order above).
constexpr int FOLD_ROWS = 10;
template <bool BF, bool TREE, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) fold_cols_k(void* __restrict__ dw, void* __restrict__ db, const float* __restrict__ partial, int nrows, int C, int W) {
  mlb_pdl_sync();
  constexpr int TRIP = WARPS * FOLD_ROWS, SL = TREE ? WARPS : 8;
  __shared__ float rowbuf[SL == WARPS ? 1 : TRIP][32], red[SL][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (!TREE && SL == WARPS) {      // (the columns asked about once and not in each load: 40 registers, 32 in the other form; column sums of 3152 x 2304 4.60 -> 4.39 us)
    if (c < W) {
      for (int r = warp; r < nrows; r += TRIP) {
        float v[FOLD_ROWS];
#pragma unroll
        for (int k = 0; k < FOLD_ROWS; k++) v[k] = r + WARPS * k < nrows ? partial[(size_t)(r + WARPS * k) * W + c] : 0.f;
#pragma unroll
        for (int k = 0; k < FOLD_ROWS; k++) s += v[k];
      }
    }
  } else {
    for (int r0 = 0; r0 < nrows; r0 += TRIP) {
      float v[FOLD_ROWS];
#pragma unroll
      for (int k = 0; k < FOLD_ROWS; k++) {
        const int r = r0 + warp + WARPS * k;
        v[k] = r < nrows && c < W ? partial[(size_t)r * W + c] : 0.f;
      }
      if (TREE) {
#pragma unroll
        for (int w = 1; w < FOLD_ROWS; w *= 2)
#pragma unroll
          for (int k = 0; k + w < FOLD_ROWS; k += 2 * w) v[k] += v[k + w];
        s += v[0];
      } else {
        if (r0 > 0) __syncthreads();
#pragma unroll
        for (int k = 0; k < FOLD_ROWS; k++) rowbuf[warp + WARPS * k][lane] = v[k];
        __syncthreads();
        if (warp < SL) {
          const int n = min(TRIP, nrows - r0);
#pragma unroll 8
          for (int r = warp; r < n; r += SL) s += rowbuf[r][lane];
        }
      }
    }
  }
  if (warp < SL) red[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || c >= W) return;
  if (TREE) {
    float v[SL];
#pragma unroll
    for (int k = 0; k < SL; k++) v[k] = red[k][lane];
#pragma unroll
    for (int w = 1; w < SL; w *= 2)
#pragma unroll
      for (int k = 0; k + w < SL; k += 2 * w) v[k] += v[k + w];
    s = v[0];
  } else {
#pragma unroll
    for (int i = 1; i < SL; i++) s += red[i][lane];
  }
  void* dst = c < C ? dw : db;
  if (dst == nullptr) return;
  const int i = c < C ? c : c - C;
  if (BF) ((bf16*)dst)[i] = __float2bfloat16(s);
  else ((float*)dst)[i] += s;
}
template <bool BF, bool TREE = false>
static void fold_launch(void* dw, void* db, const float* partial, int nrows, int C, int W, cudaStream_t st) {
  if (nrows > 8 * FOLD_ROWS) mlb_launch(fold_cols_k<BF, TREE, 32>, dim3((W + 31) / 32), dim3(1024), 0, st, dw, db, partial, nrows, C, W);
  else mlb_launch(fold_cols_k<BF, TREE, 8>, dim3((W + 31) / 32), dim3(256), 0, st, dw, db, partial, nrows, C, W);
}

// ------------------------------------------------------------------ RoPE (in place on the Q and K slices of qkv[B*T, 3C])
// pairs (i, i + hd/2); fwd: x0' = x0 c - x1 s, x1' = x1 c + x0 s; bwd uses -s.
__global__ void rope_k(bf16* __restrict__ qkv, const float* __restrict__ cosT, const float* __restrict__ sinT, long rows, int T,
                       int H, int hd, float sign) {
  mlb_pdl_sync();
  const int h2 = hd >> 1;
  const int per_row = 2 * H * (h2 >> 3);  // vectors of 8 pairs per row (q and k)
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * per_row) return;
  const long row = idx / per_row;
  int r = idx % per_row;
  const int which = r / (H * (h2 >> 3));
  r %= H * (h2 >> 3);
  const int h = r / (h2 >> 3), v = r % (h2 >> 3);
  const int t = row % T;
  bf16* p0 = qkv + row * (3L * H * hd) + (long)which * H * hd + h * hd + v * 8;
  bf16* p1 = p0 + h2;
  float a[8], b[8];
  load8(p0, a);
  load8(p1, b);
  const float4* c4 = reinterpret_cast<const float4*>(cosT + (long)t * h2 + v * 8);
  const float4* s4 = reinterpret_cast<const float4*>(sinT + (long)t * h2 + v * 8);
  float c[8], s[8];
  *reinterpret_cast<float4*>(c) = c4[0]; *reinterpret_cast<float4*>(c + 4) = c4[1];
  *reinterpret_cast<float4*>(s) = s4[0]; *reinterpret_cast<float4*>(s + 4) = s4[1];
  float o0[8], o1[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float sj = s[j] * sign;
    o0[j] = a[j] * c[j] - b[j] * sj;
    o1[j] = b[j] * c[j] + a[j] * sj;
  }
  store8(p0, o0);
  store8(p1, o1);
}
// Out of place, and from grouped heads: src rows are [H query | Hkv key | Hkv value] heads, dst rows [H | H | H] with Q and K rotated
// and every key / value head repeated for its H / Hkv query heads (Hkv = H: a plain copy of V).  One read and one write of the
// tensors, which is what bounds it (qkv[16384, 6144]: 402 MB); copying first and rotating in place moves 670 MB, expanding the heads
// with copies more.  32-bit index arithmetic (the host checks the range); a thread takes 8 rotation pairs of one
// dst head, or the same two 16-byte units of V.
__global__ void __launch_bounds__(256) rope_copy_k(bf16* __restrict__ dst, const bf16* __restrict__ src, const float* __restrict__ cosT,
                                                   const float* __restrict__ sinT, unsigned total, int T, int H, int Hkv, int hd) {
  mlb_pdl_sync();
  const unsigned idx = blockIdx.x * 256u + threadIdx.x;
  if (idx >= total) return;
  const unsigned h2 = (unsigned)hd >> 1, vph = h2 >> 3, per_row = 3u * H * vph, rep = (unsigned)(H / Hkv);
  const unsigned row = idx / per_row, r = idx % per_row, head = r / vph, v = r % vph;      // head of [Q | K | V]
  const unsigned sh = head < (unsigned)H ? head : head < 2u * H ? H + (head - H) / rep : H + Hkv + (head - 2u * H) / rep;
  const bf16* s0 = src + (size_t)row * ((unsigned)(H + 2 * Hkv) * hd) + sh * hd + v * 8;
  bf16* d0 = dst + (size_t)row * (3u * H * hd) + head * hd + v * 8;
  const uint4 ra = __ldg(reinterpret_cast<const uint4*>(s0)), rb = __ldg(reinterpret_cast<const uint4*>(s0 + h2));
  if (head >= 2u * H) {
    *reinterpret_cast<uint4*>(d0) = ra;
    *reinterpret_cast<uint4*>(d0 + h2) = rb;
    return;
  }
  float a[8], b[8], c[8], s[8], o0[8], o1[8];
  unpack8(ra, a);
  unpack8(rb, b);
  const size_t te = (size_t)(row % (unsigned)T) * h2 + v * 8;
  *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(cosT + te); *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(cosT + te + 4);
  *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(sinT + te); *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(sinT + te + 4);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    o0[j] = a[j] * c[j] - b[j] * s[j];
    o1[j] = b[j] * c[j] + a[j] * s[j];
  }
  store8(d0, o0);
  store8(d0 + h2, o1);
}
// Its backward for grouped heads (behind the attention backward, which has undone the rotation): Q copied, the gradients of the
// H / Hkv copies of a key / value head added in fp32 and rounded once.
__global__ void __launch_bounds__(256) kv_group_sum_k(bf16* __restrict__ dst, const bf16* __restrict__ src, unsigned total, int H, int Hkv, int hd) {
  mlb_pdl_sync();
  const unsigned idx = blockIdx.x * 256u + threadIdx.x;
  if (idx >= total) return;
  const unsigned vph = (unsigned)hd >> 3, heads = (unsigned)(H + 2 * Hkv), rep = (unsigned)(H / Hkv);
  const unsigned row = idx / (heads * vph), r = idx % (heads * vph), head = r / vph, v = r % vph;
  const bf16* s0 = src + (size_t)row * (3u * H * hd) + v * 8;
  bf16* d0 = dst + (size_t)row * (heads * hd) + head * hd + v * 8;
  if (head < (unsigned)H) {
    *reinterpret_cast<uint4*>(d0) = *reinterpret_cast<const uint4*>(s0 + head * hd);
    return;
  }
  const unsigned first = head < (unsigned)(H + Hkv) ? H + (head - H) * rep : 2u * H + (head - H - Hkv) * rep;
  float acc[8] = {};
  for (unsigned i = 0; i < rep; i++) {
    float x[8];
    load8(s0 + (size_t)(first + i) * hd, x);
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] += x[j];
  }
  store8(d0, acc);
}
__global__ void rope_scalar_k(bf16* __restrict__ qkv, const float* __restrict__ cosT, const float* __restrict__ sinT, long rows,
                              int T, int H, int hd, float sign) {
  const int h2 = hd >> 1;
  const int per_row = 2 * H * h2;
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * per_row) return;
  const long row = idx / per_row;
  int r = idx % per_row;
  const int which = r / (H * h2);
  r %= H * h2;
  const int h = r / h2, i = r % h2;
  const int t = row % T;
  bf16* p0 = qkv + row * (3L * H * hd) + (long)which * H * hd + h * hd + i;
  float a = __bfloat162float(p0[0]), b = __bfloat162float(p0[h2]);
  float c = cosT[(long)t * h2 + i], s = sinT[(long)t * h2 + i] * sign;
  p0[0] = __float2bfloat16(a * c - b * s);
  p0[h2] = __float2bfloat16(b * c + a * s);
}

// ------------------------------------------------------------------ SwiGLU on gu[rows, 2I] = [gate | up]
__global__ void swiglu_fwd_k(bf16* __restrict__ out, const bf16* __restrict__ gu, long rows, int I) {
  mlb_pdl_sync();
  const int vpr = I >> 3;
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * vpr) return;
  const long row = idx / vpr;
  const int v = idx % vpr;
  float g[8], u[8], o[8];
  load8(gu + row * 2L * I + v * 8, g);
  load8(gu + row * 2L * I + I + v * 8, u);
#pragma unroll
  for (int j = 0; j < 8; j++) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
  store8(out + row * (long)I + v * 8, o);
}
// The same with an E4M3 copy of the fp32 result (x scale) for the 8-bit down projection (train/gpt_kernels.cuh:605-613).
__global__ void swiglu_fwd_fp8_k(bf16* __restrict__ out, uint8_t* __restrict__ out8, const bf16* __restrict__ gu, long rows, int I, float s8) {
  mlb_pdl_sync();
  const int vpr = I >> 3;
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * vpr) return;
  const long row = idx / vpr;
  const int v = idx % vpr;
  float g[8], u[8], o[8];
  load8(gu + row * 2L * I + v * 8, g);
  load8(gu + row * 2L * I + I + v * 8, u);
#pragma unroll
  for (int j = 0; j < 8; j++) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
  store8(out + row * (long)I + v * 8, o);
  store8_e4m3(out8 + row * (long)I + v * 8, o, s8);
}
__global__ void swiglu_bwd_k(bf16* __restrict__ dgu, const bf16* __restrict__ dout, const bf16* __restrict__ gu, long rows, int I) {
  mlb_pdl_sync();
  const int vpr = I >> 3;
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * vpr) return;
  const long row = idx / vpr;
  const int v = idx % vpr;
  float g[8], u[8], d[8], dg[8], du[8];
  load8(gu + row * 2L * I + v * 8, g);
  load8(gu + row * 2L * I + I + v * 8, u);
  load8(dout + row * (long)I + v * 8, d);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float s = 1.f / (1.f + __expf(-g[j]));
    dg[j] = d[j] * u[j] * s * (1.f + g[j] * (1.f - s));
    du[j] = d[j] * g[j] * s;
  }
  store8(dgu + row * 2L * I + v * 8, dg);
  store8(dgu + row * 2L * I + I + v * 8, du);
}
__global__ void swiglu_fwd_scalar_k(bf16* out, const bf16* gu, long rows, int I) {
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * I) return;
  long row = idx / I;
  int i = idx % I;
  float g = __bfloat162float(gu[row * 2L * I + i]), u = __bfloat162float(gu[row * 2L * I + I + i]);
  out[idx] = __float2bfloat16(g / (1.f + __expf(-g)) * u);
}
__global__ void swiglu_bwd_scalar_k(bf16* dgu, const bf16* dout, const bf16* gu, long rows, int I) {
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * I) return;
  long row = idx / I;
  int i = idx % I;
  float g = __bfloat162float(gu[row * 2L * I + i]), u = __bfloat162float(gu[row * 2L * I + I + i]);
  float d = __bfloat162float(dout[idx]);
  float s = 1.f / (1.f + __expf(-g));
  dgu[row * 2L * I + i] = __float2bfloat16(d * u * s * (1.f + g * (1.f - s)));
  dgu[row * 2L * I + I + i] = __float2bfloat16(d * g * s);
}

// ------------------------------------------------------------------ fused cross-entropy (one block per row, in place)
// pass 1: online max / sum-exp over the row; pass 2 (row is L2-resident): logits <- (softmax - onehot) * dscale.
// Rows with tgt < 0: loss 0, gradient row zeroed.
__device__ __forceinline__ float exp2f_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__global__ void __launch_bounds__(512, 4) ce_fwd_bwd_k(float* __restrict__ losses, bf16* dlogits, const bf16* logits,
                                                    const int* __restrict__ tgt, int V, long ld, float dscale,
                                                    const float* __restrict__ dscale_dev) {
  mlb_pdl_sync();
  __shared__ float red[32];
  const long row = blockIdx.x;
  const bf16* z = logits + row * ld;
  bf16* dz = dlogits + row * ld;
  const bool grad = dlogits != nullptr;
  const int t = tgt[row];
  const bool vec = ((V & 7) == 0) && ((ld & 7) == 0);
  if (t >= V && threadIdx.x == 0) mlb_set_error(MLB_ERR_BOUNDS, 0xCE);      // treated like an ignored row
  if (t < 0 || t >= V) {
    if (threadIdx.x == 0) losses[row] = 0.f;
    if (grad && vec) {
      for (int i = threadIdx.x * 8; i < V; i += blockDim.x * 8) *reinterpret_cast<uint4*>(dz + i) = make_uint4(0, 0, 0, 0);
    } else if (grad) {
      for (int i = threadIdx.x; i < V; i += blockDim.x) dz[i] = __float2bfloat16(0.f);
    }
    return;
  }
  float m = -INFINITY, s = 0.f;
  constexpr float L2E = 1.4426950408889634f;
  if (vec) {
    // two 16-byte loads in flight per thread and step (one row per block: the bytes in flight are what keeps HBM busy);
    // exponentials as exp2 of one fused multiply-add
    const int step = blockDim.x * 8;
    for (int i = threadIdx.x * 8; i < V; i += 2 * step) {
      const bool two = i + step < V;
      const uint4 ra = *reinterpret_cast<const uint4*>(z + i);
      const uint4 rb = two ? *reinterpret_cast<const uint4*>(z + i + step) : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -inf
      float xa[8], xb[8];
      unpack8(ra, xa);
      unpack8(rb, xb);
      float mx = fmaxf(xa[0], xb[0]);
#pragma unroll
      for (int j = 1; j < 8; j++) mx = fmaxf(mx, fmaxf(xa[j], xb[j]));
      if (mx > m) { s *= exp2f_fast((m - mx) * L2E); m = mx; }
      const float nm = -m * L2E;
#pragma unroll
      for (int j = 0; j < 8; j++) s += exp2f_fast(fmaf(xa[j], L2E, nm)) + exp2f_fast(fmaf(xb[j], L2E, nm));
    }
  } else {
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      float x = __bfloat162float(z[i]);
      if (x > m) { s *= __expf(m - x); m = x; }
      s += __expf(x - m);
    }
  }
  const float M = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - M);
  const float S = block_sum(s, red);
  const float zt = __bfloat162float(z[t]);
  __syncthreads();  // everyone has read z[t] before anyone overwrites it
  if (threadIdx.x == 0) losses[row] = __logf(S) + M - zt;
  if (!grad) return;
  if (dscale_dev) dscale = *dscale_dev;
  const float inv = dscale / S;
  if (vec) {
    const int step = blockDim.x * 8;
    const float nM = -M * L2E;
    for (int i = threadIdx.x * 8; i < V; i += 2 * step) {
      const bool two = i + step < V;
      const uint4 ra = *reinterpret_cast<const uint4*>(z + i);
      uint4 rb = make_uint4(0, 0, 0, 0);
      if (two) rb = *reinterpret_cast<const uint4*>(z + i + step);
      float xa[8], xb[8];
      unpack8(ra, xa);
      unpack8(rb, xb);
#pragma unroll
      for (int j = 0; j < 8; j++) xa[j] = exp2f_fast(fmaf(xa[j], L2E, nM)) * inv - ((i + j == t) ? dscale : 0.f);
      store8(dz + i, xa);
      if (two) {
#pragma unroll
        for (int j = 0; j < 8; j++) xb[j] = exp2f_fast(fmaf(xb[j], L2E, nM)) * inv - ((i + step + j == t) ? dscale : 0.f);
        store8(dz + i + step, xb);
      }
    }
  } else {
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      float x = __bfloat162float(z[i]);
      dz[i] = __float2bfloat16(__expf(x - M) * inv - ((i == t) ? dscale : 0.f));
    }
  }
}

// ------------------------------------------------------------------ cross-entropy over vocabulary chunks
// The LM head's logits exist only one [rows, n] chunk at a time (columns off .. off+n of the vocabulary).
// ce_chunk_stats_k folds a chunk into the running per-row maximum m, sum s = sum exp(z - m) and target logit zt
// (train/gpt_kernels.cuh:1244-1277); after the last chunk the row's loss is log(s) + m - zt.
// ce_chunk_grad_k turns a recomputed chunk into dlogits = (exp(z - m) / s - onehot) * dscale in place and writes the
// loss (train/gpt_kernels.cuh:1279-1299).  Rows with tgt < 0: loss 0, zero gradient.  One block per row.
__global__ void __launch_bounds__(256) ce_chunk_stats_k(float* __restrict__ rowmax, float* __restrict__ rowsum,
                                                        float* __restrict__ tgt_logit, const bf16* __restrict__ chunk,
                                                        const int* __restrict__ tgt, int n, long ld, int off) {
  __shared__ float red[32];
  const long row = blockIdx.x;
  const int t = tgt[row];
  if (t < 0) return;                    // (uniform over the block)
  const bf16* z = chunk + row * ld;
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float x = __bfloat162float(z[i]);
    if (x > m) { s *= __expf(m - x); m = x; }
    s += __expf(x - m);
  }
  const float M = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - M);
  const float S = block_sum(s, red);
  if (threadIdx.x == 0) {
    const float m0 = rowmax[row], s0 = rowsum[row];
    const float mn = fmaxf(m0, M);
    rowsum[row] = ((m0 == -INFINITY) ? 0.f : s0 * __expf(m0 - mn)) + S * __expf(M - mn);
    rowmax[row] = mn;
    if (t >= off && t < off + n) tgt_logit[row] = __bfloat162float(z[t - off]);
  }
}
__global__ void __launch_bounds__(256) ce_chunk_grad_k(float* __restrict__ losses, bf16* __restrict__ chunk,
                                                       const int* __restrict__ tgt, const float* __restrict__ rowmax,
                                                       const float* __restrict__ rowsum, const float* __restrict__ tgt_logit,
                                                       int n, long ld, int off, float dscale) {
  const long row = blockIdx.x;
  const int t = tgt[row];
  bf16* z = chunk + row * ld;
  if (t < 0) {
    if (threadIdx.x == 0) losses[row] = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) z[i] = __float2bfloat16(0.f);
    return;
  }
  const float M = rowmax[row], S = rowsum[row];
  if (threadIdx.x == 0) losses[row] = __logf(S) + M - tgt_logit[row];
  const float inv = dscale / S;
  const int tl = t - off;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float x = __bfloat162float(z[i]);
    z[i] = __float2bfloat16(__expf(x - M) * inv - ((i == tl) ? dscale : 0.f));
  }
}

// Same result with ONE exponential per logit (the two-pass kernel above spends 2 x rows x V of them and is limited by
// the special-function unit, not by memory): the row is parked in shared memory.
//   pass 1  global -> shared (raw bf16) + row maximum            (no exponential)
//   pass 2  shared: e = exp(x - max) in fp32 -> row sum; e parked as fp16 (11-bit mantissa; the output is bf16)
//   pass 3  shared -> global: e / sum * dscale - onehot
// Needs V % 8 == 0, ld % 8 == 0 and V * 2 bytes of dynamic shared memory (two blocks per SM up to V ~ 56 k).
__global__ void __launch_bounds__(512) ce_fwd_bwd_smem_k(float* __restrict__ losses, bf16* __restrict__ logits,
                                                         const int* __restrict__ tgt, int V, long ld, float dscale) {
  mlb_pdl_sync();
  extern __shared__ uint4 ce_row[];      // V / 8 vectors of 8 x 16 bit
  __shared__ float red[32];
  const long row = blockIdx.x;
  bf16* z = logits + row * ld;
  const int t = tgt[row];
  const int nv = V >> 3;
  if (t >= V && threadIdx.x == 0) mlb_set_error(MLB_ERR_BOUNDS, 0xCE);
  if (t < 0 || t >= V) {
    if (threadIdx.x == 0) losses[row] = 0.f;
    for (int i = threadIdx.x; i < nv; i += blockDim.x) reinterpret_cast<uint4*>(z)[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  float m = -INFINITY;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(z) + i);
    ce_row[i] = v;
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; j++) m = fmaxf(m, fmaxf(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u)));
  }
  const float M = block_max(m, red);       // contains a __syncthreads: the whole row is in shared memory after it
  float s = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const uint4 v = ce_row[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float e0 = __expf(__uint_as_float(w[j] << 16) - M), e1 = __expf(__uint_as_float(w[j] & 0xffff0000u) - M);
      s += e0 + e1;
      const __half2 h = __floats2half2_rn(e0, e1);
      o[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    ce_row[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  const float S = block_sum(s, red);
  const float zt = __bfloat162float(z[t]);   // global memory still holds the logits
  if (threadIdx.x == 0) losses[row] = __logf(S) + M - zt;
  __syncthreads();                            // z[t] has been read by everyone before it is overwritten
  const float inv = dscale / S;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const uint4 v = ce_row[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float x[8];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
      x[2 * j] = f.x * inv;
      x[2 * j + 1] = f.y * inv;
    }
    const int d = t - i * 8;
    if (d >= 0 && d < 8) {
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j == d) x[j] -= dscale;
    }
    store8(z + i * 8, x);
  }
}

// ------------------------------------------------------------------ special-function-unit micro-benchmark
// Every thread runs `iters` rounds of eight independent exponentials: fp32 `ex2.approx.ftz.f32` (mode 0) or packed
// `ex2.approx.ftz.bf16x2` (mode 1, two results per instruction).  cycles[block] = SM cycles of the block.
__global__ void __launch_bounds__(512) mufu_probe_k(long long* cycles, float* sink, int mode, int iters) {
  float acc = 0.f;
  float x[8];
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = -0.001f * (float)(threadIdx.x + j);
  __syncthreads();
  const long long t0 = clock64();
  if (mode == 0) {
    for (int i = 0; i < iters; i++) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float y;
        asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x[j]));
        x[j] = y - 1.0f;
      }
    }
  } else {
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; j++) h[j] = pack_bf16(x[j], x[j] * 0.5f);
    for (int i = 0; i < iters; i++) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        uint32_t y;
        asm volatile("ex2.approx.ftz.bf16x2 %0, %1;" : "=r"(y) : "r"(h[j]));
        h[j] = y ^ 0x80008000u;   // negate both halves: keeps the argument in (-1, 0]
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] = __uint_as_float(h[j] << 16);
  }
  const long long t1 = clock64();
#pragma unroll
  for (int j = 0; j < 8; j++) acc += x[j];
  if (threadIdx.x == 0) cycles[blockIdx.x] = t1 - t0;
  if (acc == 12345.678f) sink[0] = acc;
}
MLB_API int mlb_mufu_probe(long long* cycles, float* sink, int mode, int iters, int blocks, cudaStream_t st) {
  mufu_probe_k<<<blocks, 512, 0, st>>>(cycles, sink, mode, iters);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------ AdamW (fp32 master/m/v, bf16 copy written in the same pass)
__global__ void adamw_k(float* __restrict__ master, bf16* __restrict__ params, const float* __restrict__ grads,
                        float* __restrict__ m, float* __restrict__ v, long n, float lr, float b1, float b2, float eps, float wd,
                        float inv_bc1, float inv_bc2, float grad_scale, const float* __restrict__ dev_hyper,
                        uint8_t* __restrict__ params8 = nullptr, float s8 = 1.f) {
  mlb_pdl_sync();
  // params8 (optional): E4M3 copy of the updated fp32 weights x s8 for the 8-bit forward (train/gpt_kernels.cuh:1402-1416)
  // dev_hyper (optional, device memory): {lr, 1/bc1, 1/bc2, grad_scale} override the launch arguments, so a captured
  // CUDA graph can be replayed with the step-dependent bias corrections of the current step.
  if (dev_hyper) { lr = dev_hyper[0]; inv_bc1 = dev_hyper[1]; inv_bc2 = dev_hyper[2]; grad_scale = dev_hyper[3]; }
  long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 3 < n) {
    float4 g = *reinterpret_cast<const float4*>(grads + i);
    float4 mm = *reinterpret_cast<const float4*>(m + i);
    float4 vv = *reinterpret_cast<const float4*>(v + i);
    float4 p = *reinterpret_cast<const float4*>(master + i);
    float* gp = &g.x; float* mp = &mm.x; float* vp = &vv.x; float* pp = &p.x;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float gj = gp[j] * grad_scale;
      mp[j] = b1 * mp[j] + (1.f - b1) * gj;
      vp[j] = b2 * vp[j] + (1.f - b2) * gj * gj;
      pp[j] -= lr * (mp[j] * inv_bc1 / (sqrtf(vp[j] * inv_bc2) + eps) + wd * pp[j]);
    }
    *reinterpret_cast<float4*>(m + i) = mm;
    *reinterpret_cast<float4*>(v + i) = vv;
    *reinterpret_cast<float4*>(master + i) = p;
    if (params) {
      uint2 o;
      o.x = pack_bf16(p.x, p.y);
      o.y = pack_bf16(p.z, p.w);
      *reinterpret_cast<uint2*>(params + i) = o;
    }
    if (params8) {
      const uint32_t q = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(p.x * s8, p.y * s8), __NV_SATFINITE, __NV_E4M3) |
                         ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(p.z * s8, p.w * s8), __NV_SATFINITE, __NV_E4M3) << 16);
      *reinterpret_cast<uint32_t*>(params8 + i) = q;
    }
  } else {
    for (; i < n; i++) {
      const float gj = grads[i] * grad_scale;
      float mj = b1 * m[i] + (1.f - b1) * gj, vj = b2 * v[i] + (1.f - b2) * gj * gj, pj = master[i];
      pj -= lr * (mj * inv_bc1 / (sqrtf(vj * inv_bc2) + eps) + wd * pj);
      m[i] = mj; v[i] = vj; master[i] = pj;
      if (params) params[i] = __float2bfloat16(pj);
      if (params8) params8[i] = (uint8_t)__nv_cvt_float_to_fp8(pj * s8, __NV_SATFINITE, __NV_E4M3);
    }
  }
}

// ------------------------------------------------------------------ casts / utilities
// bf16 -> E4M3 storage (x scale), 8 elements per thread (train/gpt_kernels.cuh:211-214)
__global__ void cast_b2e4m3_k(uint8_t* __restrict__ out, const bf16* __restrict__ in, long n, float scale) {
  long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i + 7 < n) {
    float x[8];
    load8(in + i, x);
    store8_e4m3(out + i, x, scale);
  } else {
    for (; i < n; i++) out[i] = (uint8_t)__nv_cvt_float_to_fp8(__bfloat162float(in[i]) * scale, __NV_SATFINITE, __NV_E4M3);
  }
}
__global__ void cast_f2b_k(bf16* __restrict__ out, const float* __restrict__ in, long n, float scale) {
  mlb_pdl_sync();
  long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 3 < n) {
    float4 f = *reinterpret_cast<const float4*>(in + i);
    uint2 o;
    o.x = pack_bf16(f.x * scale, f.y * scale);
    o.y = pack_bf16(f.z * scale, f.w * scale);
    *reinterpret_cast<uint2*>(out + i) = o;
  } else {
    for (; i < n; i++) out[i] = __float2bfloat16(in[i] * scale);
  }
}
// E4M3 rounding of a bf16 tensor, kept in bf16: out = e4m3_saturate(x * scale) / scale (round to nearest even, +-448
// saturation; train/gpt_kernels.cuh:203-218 is the reference's cast to FP8 storage).  With a power-of-two scale the
// result is exact in bf16 (3 mantissa bits), so a bf16 GEMM on such operands has the numerics of an E4M3 x E4M3 GEMM
// with fp32 accumulation.
__global__ void fp8_qdq_k(bf16* __restrict__ out, const bf16* __restrict__ in, long n, float scale, float inv_scale) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const __nv_fp8_e4m3 q(__bfloat162float(in[i]) * scale);
  out[i] = __float2bfloat16(float(q) * inv_scale);
}
// out[0] = scale * sum(x[0..n)): one block, fixed summation order (deterministic); the per-row losses of a step.
__global__ void __launch_bounds__(1024) sum_scale_k(float* __restrict__ out, const float* __restrict__ x, long n, float scale) {
  __shared__ float red[32];
  float s = 0.f;
  for (long i = threadIdx.x; i < n; i += blockDim.x) s += x[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[0] = s * scale;
}
// stats[0] = 1 / max(n, 1) with n = targets >= 0, stats[1] = max(n, 1) (as an integer): one block, the targets are a few 10 KB
__global__ void __launch_bounds__(1024) ce_count_k(float* __restrict__ stats, const int* __restrict__ tgt, long rows) {
  __shared__ int red[32];
  int c = 0;
  for (long i = threadIdx.x; i < rows; i += 1024) c += tgt[i] >= 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    c = max(__reduce_add_sync(0xffffffffu, red[threadIdx.x]), 1);
    if (threadIdx.x == 0) { stats[0] = (float)(1.0 / (double)c); stats[1] = __int_as_float(c); }
  }
}
// out[0] = sum(x) / n, summed in double in a fixed order
__global__ void __launch_bounds__(1024) sum_mean_k(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ stats, long rows) {
  __shared__ double red[32];
  double s = 0.0;
  for (long i = threadIdx.x; i < rows; i += 1024) s += (double)x[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out[0] = (float)(s / (double)__float_as_int(stats[1]));
  }
}
// out = x * s[0] in bf16 (fp32 product, one rounding), s in device memory: the gradient of the logits times the gradient of the
// loss.  Two 16-byte loads in flight per thread; bound by the read and the write (1.65 GB each way at 16384 x 50304).
__global__ void __launch_bounds__(256) scale_dev_k(bf16* __restrict__ out, const bf16* __restrict__ x, const float* __restrict__ s, long n) {
  mlb_pdl_sync();
  const float f = *s;
  const long i = ((long)blockIdx.x * 512 + threadIdx.x) * 8, i2 = i + 256 * 8;
  if (i2 + 7 < n) {
    const uint4 ra = __ldcs(reinterpret_cast<const uint4*>(x + i)), rb = __ldcs(reinterpret_cast<const uint4*>(x + i2));
    float a[8], b[8];
    unpack8(ra, a);
    unpack8(rb, b);
#pragma unroll
    for (int j = 0; j < 8; j++) { a[j] *= f; b[j] *= f; }
    store8(out + i, a);
    store8(out + i2, b);
    return;
  }
  for (int h = 0; h < 2; h++)
    for (long e = h ? i2 : i, end = e + 8; e < end && e < n; e++) out[e] = __float2bfloat16(__bfloat162float(x[e]) * f);
}
// x *= s[0], in place, rounded as above.  A factor of one (the usual gradient of a mean loss) leaves every value as it is, so the blocks
// read the scalar and return: at 16384 x 50304 that saves the 3.3 GB pass (head and loss, forward and backward: 4213 -> 3791 us).  A grid of resident blocks
// that walk the tensor, because the 200 K blocks of the kernel above take as long to come and go as a quarter of that.
__global__ void __launch_bounds__(256) scale_dev_inplace_k(bf16* x, const float* __restrict__ s, long n) {
  mlb_pdl_sync();
  const float f = *s;
  if (f == 1.f) return;
  const long step = (long)gridDim.x * 4096;
  for (long i = ((long)blockIdx.x * 512 + threadIdx.x) * 8; i < n; i += step) {
    const long i2 = i + 256 * 8;
    if (i2 + 7 < n) {
      const uint4 ra = __ldcs(reinterpret_cast<const uint4*>(x + i)), rb = __ldcs(reinterpret_cast<const uint4*>(x + i2));
      float a[8], b[8];
      unpack8(ra, a);
      unpack8(rb, b);
#pragma unroll
      for (int j = 0; j < 8; j++) { a[j] *= f; b[j] *= f; }
      store8(x + i, a);
      store8(x + i2, b);
      continue;
    }
    for (int h = 0; h < 2; h++)
      for (long e = h ? i2 : i, end = e + 8; e < end && e < n; e++) x[e] = __float2bfloat16(__bfloat162float(x[e]) * f);
  }
}
__global__ void cast_b2f_k(float* __restrict__ out, const bf16* __restrict__ in, long n, float scale) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __bfloat162float(in[i]) * scale;
}
__global__ void scale_f32_k(float* __restrict__ x, long n, float scale) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] *= scale;
}
__global__ void residual_add_k(bf16* __restrict__ out, const bf16* __restrict__ a, const bf16* __restrict__ b, long n) {
  mlb_pdl_sync();
  long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i + 7 < n) {
    float x[8], y[8];
    load8(a + i, x);
    load8(b + i, y);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += y[j];
    store8(out + i, x);
  } else {
    for (; i < n; i++) out[i] = __float2bfloat16(__bfloat162float(a[i]) + __bfloat162float(b[i]));
  }
}

// ------------------------------------------------------------------ vision helpers
// pixels fp32 [B, Cin, Himg, Wimg] -> patches bf16 [B*gh*gw, Cin*P*P] with element order (c, py, px).
__global__ void patchify_k(bf16* __restrict__ out, const float* __restrict__ px, int B, int Cin, int Himg, int Wimg, int P) {
  const int gh = Himg / P, gw = Wimg / P, pd = Cin * P * P;
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long n = (long)B * gh * gw * pd;
  if (idx >= n) return;
  int e = idx % pd;
  long pr = idx / pd;
  int pxl = e % P, pyl = (e / P) % P, c = e / (P * P);
  int pw = pr % gw, ph = (pr / gw) % gh, b = pr / (gw * gh);
  out[idx] = __float2bfloat16(px[(((long)b * Cin + c) * Himg + ph * P + pyl) * Wimg + pw * P + pxl]);
}
// The same, eight pixels of one patch row per thread (P a multiple of 8, 16-byte aligned rows): two 16-byte loads, one
// 16-byte store, index arithmetic once per eight values.
__global__ void patchify8_k(bf16* __restrict__ out, const float* __restrict__ px, int B, int Cin, int Himg, int Wimg, int P) {
  mlb_pdl_sync();
  const int gh = Himg / P, gw = Wimg / P, pd8 = Cin * P * P / 8, p8 = P / 8;
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)B * gh * gw * pd8) return;
  const int e = (int)(idx % pd8);
  const long pr = idx / pd8;
  const int x8 = e % p8, pyl = (e / p8) % P, c = e / (p8 * P);
  const int pw = (int)(pr % gw), ph = (int)((pr / gw) % gh), b = (int)(pr / ((long)gw * gh));
  const float4* src = reinterpret_cast<const float4*>(px + (((long)b * Cin + c) * Himg + ph * P + pyl) * Wimg + pw * P + x8 * 8);
  const float4 a = __ldcs(src), d = __ldcs(src + 1);
  uint4 o;
  o.x = pack_bf16(a.x, a.y); o.y = pack_bf16(a.z, a.w); o.z = pack_bf16(d.x, d.y); o.w = pack_bf16(d.z, d.w);
  *reinterpret_cast<uint4*>(out + idx * 8) = o;
}
__global__ void add_posembed_k(bf16* __restrict__ x, const bf16* __restrict__ pos, long NP, int n_patch, int vC) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NP * vC) return;
  long r = i / vC;
  int c = i % vC;
  x[i] = __float2bfloat16(__bfloat162float(x[i]) + __bfloat162float(pos[(r % n_patch) * vC + c]));
}
// dpos[p, c] += sum_b dx[b*n_patch + p, c]  (one thread per (p,c): deterministic, no atomics)
__global__ void posembed_grad_k(float* __restrict__ dpos, const bf16* __restrict__ dx, long NP, int n_patch, int vC) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n_patch * vC) return;
  int nb = NP / n_patch;
  float s = 0.f;
  for (int b = 0; b < nb; b++) s += __bfloat162float(dx[(long)b * n_patch * vC + i]);
  dpos[i] += s;
}

inline int gs(long n, int per_block) { return (int)((n + per_block - 1) / per_block); }

}  // namespace

#define LAUNCH_RET return (int)cudaGetLastError()
static int g_ce_smem = 0;     // tuning hook: 0 = always the two-pass cross-entropy kernel
MLB_API void mlb_ce_mode(int smem_row) { g_ce_smem = smem_row; }

// Does a row get a block?  Where its items (vectors, or elements where it has none) are more than the 128 that a warp has in flight, and up to as many
// rows as leave the start of blocks to spare.  With a block and with a warp, us: forward 1184 x 1024 1.57 and 1.93, 1536 x 1024 1.87 and 2.07, 2048 x 1024
// 2.40 and 1.81; long rows are bound by memory sooner (768 x 4096 2.4 ... 3.1 and 2.7).  Backward 768 x 1024 1.93 and 2.01, 1184 x 1024 2.39 and 2.13;
// single additions, 2048 x 1001 3.6 and 4.7, 4096 x 1001 5.7 and 5.8, 16384 x 513 17.7 and 10.8.
static bool embed_fwd_wide(long rows, int C) { return (C % 8 == 0 ? C / 8 : C) >= 128 && rows <= 1184 && rows * C <= 1L << 21; }
static bool embed_bwd_wide(long rows, int C, bool vec) { return vec ? C >= 512 && rows <= 1024 : C >= 128 && rows <= (C >= 512 ? 2048 : 1024); }
MLB_API int mlb_embed_fwd(void* out, const void* wte, const int* ids, long BT, int C, int V, cudaStream_t st) {
  if (embed_fwd_wide(BT, C))
    mlb_launch(embed_fwd_k<128>, dim3((unsigned)BT), dim3(128), 0, st, (bf16*)out, (const bf16*)wte, ids, (long)BT, C, V);
  else
    mlb_launch(embed_fwd_k<32>, dim3((unsigned)((BT + 3) / 4)), dim3(128), 0, st, (bf16*)out, (const bf16*)wte, ids, (long)BT, C, V);
  LAUNCH_RET;
}
MLB_API int mlb_embed_bwd(float* dwte, const void* dout, const int* ids, long BT, int C, int V, int T, int n_pre, cudaStream_t st) {
  const bool vec = C % 4 == 0 && (((uintptr_t)dwte & 15) | ((uintptr_t)dout & 7)) == 0;
  if (embed_bwd_wide(BT, C, vec))
    mlb_launch(embed_bwd_k<128>, dim3((unsigned)BT), dim3(128), 0, st, dwte, (const bf16*)dout, ids, (long)BT, C, V, T, n_pre, vec);
  else
    mlb_launch(embed_bwd_k<32>, dim3((unsigned)((BT + 3) / 4)), dim3(128), 0, st, dwte, (const bf16*)dout, ids, (long)BT, C, V, T, n_pre, vec);
  LAUNCH_RET;
}
MLB_API int mlb_set_prefix(void* x, const void* prefix, int B, int T, int n_pre, int C, cudaStream_t st) {
  long n = (long)B * n_pre * C;
  if (n == 0) return 0;
  mlb_launch(set_prefix_k, dim3(gs(n, 256)), dim3(256), 0, st, (bf16*)x, (const bf16*)prefix, B, T, n_pre, C);
  LAUNCH_RET;
}
MLB_API int mlb_gather_prefix_grad(void* dprefix, const void* dresid, int B, int T, int n_pre, int C, cudaStream_t st) {
  long n = (long)B * n_pre * C;
  if (n == 0) return 0;
  mlb_launch(gather_prefix_k, dim3(gs(n, 256)), dim3(256), 0, st, (bf16*)dprefix, (const bf16*)dresid, B, T, n_pre, C);
  LAUNCH_RET;
}
// Rows of 256, 512, 768 or 1024 aligned columns take the register-resident form of the kernel.
template <bool ADD, bool F8>
static void rmsnorm_fwd_launch(void* out, void* out8, float* rstd, void* resid, const void* a, const void* b, const void* w, long rows, int C,
                               float eps, float scale, cudaStream_t st) {
  const bool al = (C % 256 == 0) && C <= 1024 && ((uintptr_t)a % 16 == 0) && (!ADD || ((uintptr_t)b % 16 == 0 && (uintptr_t)resid % 16 == 0)) &&
                  ((uintptr_t)w % 16 == 0) && ((uintptr_t)out % 16 == 0) && (!F8 || (uintptr_t)out8 % 8 == 0);
#define RF(NV)                                                                                                                   \
  mlb_launch(rmsnorm_fwd_k<ADD, F8, NV>, dim3(gs(rows, 8)), dim3(256), 0, st, (bf16*)out, rstd, (bf16*)resid, (const bf16*)a, (const bf16*)b, \
             (const bf16*)w, rows, C, eps, (uint8_t*)out8, scale)
  switch (al ? C / 256 : 0) {
    case 1: RF(1); break;
    case 2: RF(2); break;
    case 3: RF(3); break;
    case 4: RF(4); break;
    default: RF(0); break;
  }
#undef RF
}
MLB_API int mlb_rmsnorm_fwd(void* out, float* rstd, const void* x, const void* w, long rows, int C, float eps, cudaStream_t st) {
  rmsnorm_fwd_launch<false, false>(out, nullptr, rstd, nullptr, x, nullptr, w, rows, C, eps, 1.f, st);
  LAUNCH_RET;
}
MLB_API int mlb_add_rmsnorm_fwd(void* resid, void* out, float* rstd, const void* a, const void* b, const void* w, long rows, int C,
                                float eps, cudaStream_t st) {
  rmsnorm_fwd_launch<true, false>(out, nullptr, rstd, resid, a, b, w, rows, C, eps, 1.f, st);
  LAUNCH_RET;
}

// The two forward norms with an additional E4M3 copy of the output (x scale) for the 8-bit forward GEMMs
// (train/gpt_kernels.cuh:291-312, :474-493).  C must be a multiple of 8 for the vector path; other widths take the
// scalar path of the same kernel.
MLB_API int mlb_rmsnorm_fwd_fp8(void* out, void* out8, float* rstd, const void* x, const void* w, long rows, int C, float eps, float scale,
                                cudaStream_t st) {
  rmsnorm_fwd_launch<false, true>(out, out8, rstd, nullptr, x, nullptr, w, rows, C, eps, scale, st);
  LAUNCH_RET;
}
MLB_API int mlb_add_rmsnorm_fwd_fp8(void* resid, void* out, void* out8, float* rstd, const void* a, const void* b, const void* w, long rows,
                                    int C, float eps, float scale, cudaStream_t st) {
  rmsnorm_fwd_launch<true, true>(out, out8, rstd, resid, a, b, w, rows, C, eps, scale, st);
  LAUNCH_RET;
}
MLB_API int mlb_swiglu_fwd_fp8(void* out, void* out8, const void* gu, long rows, int I, float scale, cudaStream_t st) {
  if (I % 8 != 0) return -1;
  mlb_launch(swiglu_fwd_fp8_k, dim3(gs(rows * (I / 8), 256)), dim3(256), 0, st, (bf16*)out, (uint8_t*)out8, (const bf16*)gu, rows, I, scale);
  LAUNCH_RET;
}
MLB_API int mlb_cast_bf16_fp8(void* out8, const void* in, long n, float scale, cudaStream_t st) {
  if (n <= 0) return 0;
  cast_b2e4m3_k<<<gs((n + 7) / 8, 256), 256, 0, st>>>((uint8_t*)out8, (const bf16*)in, n, scale);
  LAUNCH_RET;
}
MLB_API int mlb_adamw_fp8(float* master, void* params, void* params8, const float* grads, float* m, float* v, long n, float lr, float b1,
                          float b2, float eps, float wd, float bc1, float bc2, float grad_scale, float w_scale, const float* dev_hyper,
                          cudaStream_t st) {
  if (n == 0) return 0;
  mlb_launch(adamw_k, dim3(gs((n + 3) / 4, 256)), dim3(256), 0, st, master, (bf16*)params, grads, m, v, n, lr, b1, b2, eps, wd, 1.f / bc1, 1.f / bc2,
             grad_scale, dev_hyper, (uint8_t*)params8, w_scale);
  LAUNCH_RET;
}

MLB_API int mlb_layernorm_fwd(void* out, float* mean, float* rstd, const void* x, const void* w, const void* b, long rows, int C, float eps,
                              cudaStream_t st) {
  const bool vec = C % 256 == 0 && C <= 2048 && (((uintptr_t)out | (uintptr_t)x | (uintptr_t)w | (uintptr_t)b) & 15) == 0;
#define LN(NV) \
  mlb_launch(layernorm_fwd_k<NV>, dim3(gs(rows, 8)), dim3(256), 0, st, (bf16*)out, mean, rstd, (const bf16*)x, (const bf16*)w, (const bf16*)b, rows, C, eps)
  switch (vec ? C / 256 : 0) {
    case 1: LN(1); break;
    case 2: LN(2); break;
    case 3: LN(3); break;
    case 4: LN(4); break;
    case 5: LN(5); break;
    case 6: LN(6); break;
    case 7: LN(7); break;
    case 8: LN(8); break;
    default: LN(0); break;
  }
#undef LN
  LAUNCH_RET;
}
// dw / db (fp32, db may be NULL) are accumulated into; C * 8 bytes of shared memory must fit the default 48 KB.
MLB_API int mlb_layernorm_bwd(void* dx, float* dw, float* db, const void* dy, const void* x, const void* w, const float* mean,
                              const float* rstd, long rows, int C, cudaStream_t st) {
  if ((size_t)C * 8 > 48 * 1024) return -1;
  layernorm_bwd_k<<<gs(rows, 8), 256, (size_t)C * 8, st>>>((bf16*)dx, dw, db, (const bf16*)dy, (const bf16*)x, (const bf16*)w, mean, rstd, rows, C);
  LAUNCH_RET;
}

// Number of blocks rmsnorm_bwd uses for `rows`; the caller provides scratch of (blocks + 16) * C floats and
// 17 zeroed ints.
// Number of the graph capture `st` takes part in, 0 if none
MLB_API unsigned long long mlb_capture_id(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(st, &cs, &id) != cudaSuccess) { cudaGetLastError(); return 0; }
  return cs == cudaStreamCaptureStatusActive ? id : 0;
}
MLB_API int mlb_rmsnorm_bwd_blocks(long rows) {
  long b = (rows + 7) / 8;
  return (int)(b < 296 ? b : 296);
}
// Norm backward with the column sums in `partial` (mlb_rmsnorm_bwd_blocks(rows) rows of C floats, 2 C for LayerNorm, contents do not
// matter) and then dw (and db): bf16 and overwritten, or fp32 and added to.  -7: not a shape of these kernels.
static bool norm_rows_ok(const void* dx, const void* dy, const void* x, const void* w, const void* add, long rows, int C) {
  return rows > 0 && C % 256 == 0 && C <= 2048 &&
         (((uintptr_t)dx | (uintptr_t)dy | (uintptr_t)x | (uintptr_t)w | (uintptr_t)add) & 15) == 0;
}
template <bool LN>
static void norm_rows_launch(void* dx, void* dw, void* db, bool bf, const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                             const void* add, long rows, int C, float* partial, cudaStream_t st) {
  const int blocks = mlb_rmsnorm_bwd_blocks(rows), gt = C / 8, W = LN ? 2 * C : C;
  constexpr int ring = norm_ring_bytes(NB_ROWS * (LN ? 2 : 3));
  static std::atomic<unsigned long long> allowed{0};
  if (mlb_allow_smem(norm_bwd_rows_k<LN>, ring, allowed) != cudaSuccess) return;      // (the caller asks for the error)
  mlb_launch(norm_bwd_rows_k<LN>, dim3(blocks), dim3(256 / gt * gt), ring, st, (bf16*)dx, (const bf16*)dy, (const bf16*)x, (const bf16*)w, mean, rstd,
             (const bf16*)add, rows, C, partial);
  if (bf) fold_launch<true>(dw, db, partial, blocks, C, W, st);
  else fold_launch<false, !LN>(dw, db, partial, blocks, C, W, st);
}
MLB_API int mlb_rmsnorm_bwd_cast(void* dx, void* dw, const void* dy, const void* x, const void* w, const float* rstd, const void* add, long rows, int C,
                                 float* partial, cudaStream_t st) {
  if (!norm_rows_ok(dx, dy, x, w, add, rows, C)) return -7;
  norm_rows_launch<false>(dx, dw, nullptr, true, dy, x, w, nullptr, rstd, add, rows, C, partial, st);
  LAUNCH_RET;
}
MLB_API int mlb_layernorm_bwd2(void* dx, void* dw, void* db, int bf, const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                               long rows, int C, float* partial, cudaStream_t st) {
  if (!norm_rows_ok(dx, dy, x, w, nullptr, rows, C)) return -7;
  norm_rows_launch<true>(dx, dw, db, bf != 0, dy, x, w, mean, rstd, nullptr, rows, C, partial, st);
  LAUNCH_RET;
}
// Splits of the rows colsum_k works with: enough blocks to fill the machine twice, at least 32 rows each
MLB_API int mlb_colsum_splits(long M, int N) {
  const long cols = (N + 255) / 256, want = (296 + cols - 1) / cols, most = (M + 31) / 32;
  return (int)(want < most ? want : (most < 1 ? 1 : most));
}
// out[N] (bf16) = column sums of x[M, N], fp32 inside; partial: mlb_colsum_splits(M, N) * N floats
MLB_API int mlb_colsum(void* out, const void* x, long M, int N, float* partial, cudaStream_t st) {
  if (M <= 0 || N <= 0 || N % 8 != 0 || ((uintptr_t)x & 15)) return -7;
  const int S = mlb_colsum_splits(M, N);
  mlb_launch(colsum_k, dim3((N + 255) / 256, S), dim3(256), 0, st, partial, (const bf16*)x, M, N);
  fold_launch<true>(out, nullptr, partial, S, N, N, st);
  LAUNCH_RET;
}
// (ticket null: the first 32 words of `partial` are the tickets)
MLB_API int mlb_rmsnorm_bwd(void* dx, float* dw, const void* dy, const void* x, const void* w, const float* rstd, const void* add,
                            long rows, int C, float* partial, int* ticket, cudaStream_t st) {
  if (ticket == nullptr) {
    ticket = (int*)partial;
    partial += 32;
  }
  const int blocks = mlb_rmsnorm_bwd_blocks(rows);
  const size_t sh = (size_t)std::max(C, 1024) * sizeof(float);
#define RB(...)                                                                                                         \
  mlb_launch(rmsnorm_bwd_k<__VA_ARGS__>, dim3(blocks), dim3(256), sh, st, (bf16*)dx, dw, (const bf16*)dy, (const bf16*)x, (const bf16*)w, rstd,   \
                                            (const bf16*)add, rows, C, partial, ticket)
  if (sh > 48 * 1024) return -3;
  // Whole multiples of 256 columns: a block's threads share a row instead of a warp having one, and the partial rows are folded by a
  // kernel of their own, which overlaps this one's end.  One warp a row, with the fold by the blocks that finish last, against this, inputs
  // not in L2: 16384 x 768 31.7 -> 27.6 us, 4096 x 768 21 -> 15.4, 65536 x 256 46 -> 33.8, 4096 x 512 17.4 -> 15.4, 16384 x 512 25.6 -> 23.6
  // (in L2 14.1 = 14.1; without a residual gradient 18.0 -> 14.7 and 22.3 -> 19.4 at 16384 x 512 and 768, but in L2 13.1 -> 13.6 and 17.2 -> 18.0).
  // In a small model's step, though, the host's launches are the bound and one less is worth more than the 2 us by which
  // this is shorter there too; the step's products grow as rows C^2, and so does the line.  Steps of two layers, us, one launch and two: 256 wide,
  // 512 rows 358 and 368, 4096 rows 363 and 374, 8192 rows 444 and 443; 512 wide, 1024 rows 361 and 370, 2048 rows 411 and 399; 768 wide,
  // 128 rows 392 and 401, 512 rows 459 and 443.  (All of that uncaptured: a captured step, which has no launches to save, pays the 2 us a norm below the line.)
  const bool rows_ok = norm_rows_ok(dx, dy, x, w, add, rows, C);
  if (rows_ok && (C >= 1024 || rows * C * C > 1L << 28)) {
    norm_rows_launch<false>(dx, dw, nullptr, false, dy, x, w, nullptr, rstd, add, rows, C, partial, st);
    LAUNCH_RET;
  }
  const bool narrow = C < 256 && C % 8 == 0 && (((uintptr_t)dx | (uintptr_t)dy | (uintptr_t)x | (uintptr_t)w | (uintptr_t)add | (uintptr_t)partial) & 15) == 0;
  if (narrow) { RB(1, true); LAUNCH_RET; }
  switch (rows_ok ? C / 256 : 0) {
    case 1: RB(1); break;
    case 2: RB(2); break;
    case 3: RB(3); break;
    default: RB(0); break;
  }
#undef RB
  LAUNCH_RET;
}
MLB_API int mlb_rope(void* qkv, const float* cosT, const float* sinT, long rows, int T, int H, int hd, float sign, cudaStream_t st) {
  const int h2 = hd / 2;
  if (h2 % 8 == 0 && (H * hd) % 8 == 0) {
    long n = rows * 2L * H * (h2 / 8);
    mlb_launch(rope_k, dim3(gs(n, 256)), dim3(256), 0, st, (bf16*)qkv, cosT, sinT, rows, T, H, hd, sign);
  } else {
    long n = rows * 2L * H * h2;
    rope_scalar_k<<<gs(n, 256), 256, 0, st>>>((bf16*)qkv, cosT, sinT, rows, T, H, hd, sign);
  }
  LAUNCH_RET;
}
// -7: the shape or alignment does not take these kernels (nothing was launched); -1: the key / value heads do not divide the query heads
MLB_API int mlb_rope_copy(void* dst, const void* src, const float* cosT, const float* sinT, long rows, int T, int H, int Hkv, int hd,
                          cudaStream_t st) {
  if (H <= 0 || Hkv <= 0 || H % Hkv != 0 || T <= 0) return -1;
  const long n = rows * 3L * H * (hd / 16);
  if (hd % 16 != 0 || n <= 0 || n >= (1L << 31) || (((uintptr_t)dst | (uintptr_t)src | (uintptr_t)cosT | (uintptr_t)sinT) & 15)) return -7;
  mlb_launch(rope_copy_k, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, (bf16*)dst, (const bf16*)src, cosT, sinT, (unsigned)n, T, H, Hkv, hd);
  LAUNCH_RET;
}
MLB_API int mlb_kv_group_sum(void* dst, const void* src, long rows, int H, int Hkv, int hd, cudaStream_t st) {
  if (H <= 0 || Hkv <= 0 || H % Hkv != 0) return -1;
  const long n = rows * (H + 2L * Hkv) * (hd / 8);
  if (hd % 8 != 0 || n <= 0 || n >= (1L << 31) || (((uintptr_t)dst | (uintptr_t)src) & 15)) return -7;
  mlb_launch(kv_group_sum_k, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, (bf16*)dst, (const bf16*)src, (unsigned)n, H, Hkv, hd);
  LAUNCH_RET;
}
MLB_API int mlb_swiglu_fwd(void* out, const void* gu, long rows, int I, cudaStream_t st) {
  if (I % 8 == 0) mlb_launch(swiglu_fwd_k, dim3(gs(rows * (I / 8), 256)), dim3(256), 0, st, (bf16*)out, (const bf16*)gu, rows, I);
  else swiglu_fwd_scalar_k<<<gs(rows * I, 256), 256, 0, st>>>((bf16*)out, (const bf16*)gu, rows, I);
  LAUNCH_RET;
}
MLB_API int mlb_swiglu_bwd(void* dgu, const void* dout, const void* gu, long rows, int I, cudaStream_t st) {
  if (I % 8 == 0) mlb_launch(swiglu_bwd_k, dim3(gs(rows * (I / 8), 256)), dim3(256), 0, st, (bf16*)dgu, (const bf16*)dout, (const bf16*)gu, rows, I);
  else swiglu_bwd_scalar_k<<<gs(rows * I, 256), 256, 0, st>>>((bf16*)dgu, (const bf16*)dout, (const bf16*)gu, rows, I);
  LAUNCH_RET;
}
// Threads of a block, `most` at most: a row of up to 1024 logits gives work to 128, and a block of 512 is then bound by its barriers and its start
// (the same sums: 16384 x 512 57.4 -> 20.6 us, 8192 x 1024 32.9 -> 16.4).  Longer rows keep what they had: from 32768 on fewer threads are slower (fewer
// rows at a time stay in the L2 for their second reading: 16384 x 50304 592 us, 724 with 256), between them more logits a thread err a little more.
static int ce_threads(int V, int most) { return V <= 1024 && most > 128 ? 128 : most; }
MLB_API int mlb_ce_fwd_bwd(float* losses, void* logits, const int* tgt, long rows, int V, long ld, float dscale, int threads,
                           cudaStream_t st) {
  if (threads != 128 && threads != 256 && threads != 512) threads = 512;
  const size_t sh = (size_t)V * 2;
  if (g_ce_smem && (V % 8 == 0) && (ld % 8 == 0) && ((uintptr_t)logits % 16 == 0) && sh <= 112 * 1024) {
    static bool attr_done = false;
    if (!attr_done) {
      if (cudaFuncSetAttribute(ce_fwd_bwd_smem_k, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess) return -5;
      attr_done = true;
    }
    mlb_launch(ce_fwd_bwd_smem_k, dim3((unsigned)rows), dim3(512), sh, st, losses, (bf16*)logits, tgt, V, ld, dscale);
    LAUNCH_RET;
  }
  if (V % 8 == 0 && ld % 8 == 0) threads = ce_threads(V, threads);
  mlb_launch(ce_fwd_bwd_k, dim3((unsigned)rows), dim3(threads), 0, st, losses, (bf16*)logits, (const bf16*)logits, tgt, V, ld, dscale, (const float*)nullptr);
  LAUNCH_RET;
}
// Mean cross-entropy over the rows with a target, out of place and without a word of it on the host: stats[0] = 1 / rows with a
// target (at least 1), losses per row, dlogits (may be null: losses only) = d loss / d logits, loss[0] = the mean.
MLB_API int mlb_ce_mean(float* loss, float* losses, float* stats, void* dlogits, const void* logits, const int* tgt, long rows, int V, cudaStream_t st) {
  // (without this check a vector access could be misaligned: the in-place entry's callers own their buffers, this one's may pass views)
  if ((((uintptr_t)dlogits | (uintptr_t)logits) & 15) && V % 8 == 0) return -7;
  if (rows > 0) {
    ce_count_k<<<1, 1024, 0, st>>>(stats, tgt, rows);
    mlb_launch(ce_fwd_bwd_k, dim3((unsigned)rows), dim3(V % 8 == 0 ? ce_threads(V, 512) : 512), 0, st, losses, (bf16*)dlogits, (const bf16*)logits, tgt, V, (long)V, 0.f, (const float*)stats);
    sum_mean_k<<<1, 1024, 0, st>>>(loss, losses, stats, rows);
  }
  LAUNCH_RET;
}
// out == x: in place, and no pass at all when the factor turns out to be one
MLB_API int mlb_scale_dev(void* out, const void* x, const float* s, long n, cudaStream_t st) {
  if (((uintptr_t)out | (uintptr_t)x) & 15) return -7;
  if (n > 0 && out == x) {
    mlb_launch(scale_dev_inplace_k, dim3((unsigned)std::min((n + 4095) / 4096, 8L * mlb_sm_count())), dim3(256), 0, st, (bf16*)out, s, n);
    LAUNCH_RET;
  }
  if (n > 0) mlb_launch(scale_dev_k, dim3((unsigned)((n + 4095) / 4096)), dim3(256), 0, st, (bf16*)out, (const bf16*)x, s, n);
  LAUNCH_RET;
}
MLB_API int mlb_ce_chunk_stats(float* rowmax, float* rowsum, float* tgt_logit, const void* chunk, const int* tgt, long rows, int n,
                               long ld, int off, cudaStream_t st) {
  if (rows <= 0 || n <= 0) return 0;
  ce_chunk_stats_k<<<(unsigned)rows, 256, 0, st>>>(rowmax, rowsum, tgt_logit, (const bf16*)chunk, tgt, n, ld, off);
  LAUNCH_RET;
}
MLB_API int mlb_ce_chunk_grad(float* losses, void* chunk, const int* tgt, const float* rowmax, const float* rowsum,
                              const float* tgt_logit, long rows, int n, long ld, int off, float dscale, cudaStream_t st) {
  if (rows <= 0 || n <= 0) return 0;
  ce_chunk_grad_k<<<(unsigned)rows, 256, 0, st>>>(losses, (bf16*)chunk, tgt, rowmax, rowsum, tgt_logit, n, ld, off, dscale);
  LAUNCH_RET;
}
MLB_API int mlb_adamw(float* master, void* params, const float* grads, float* m, float* v, long n, float lr, float b1, float b2,
                      float eps, float wd, float bc1, float bc2, float grad_scale, const float* dev_hyper, cudaStream_t st) {
  if (n == 0) return 0;
  mlb_launch(adamw_k, dim3(gs((n + 3) / 4, 256)), dim3(256), 0, st, master, (bf16*)params, grads, m, v, n, lr, b1, b2, eps, wd, 1.f / bc1, 1.f / bc2,
                                                grad_scale, dev_hyper, (uint8_t*)nullptr, 1.f);
  LAUNCH_RET;
}
// out[0] = scale * sum of n floats (the mean loss of a step, left on the device for one 4-byte read-back)
MLB_API int mlb_sum_scale(float* out, const float* x, long n, float scale, cudaStream_t st) {
  sum_scale_k<<<1, 1024, 0, st>>>(out, x, n, scale);
  LAUNCH_RET;
}
// Zero-fill of a buffer (the gradient buffer at the start of backward: cudaMemsetAsync as in train/gpt.cu:600)
MLB_API int mlb_zero(void* p, long nbytes, cudaStream_t st) { return (int)cudaMemsetAsync(p, 0, (size_t)nbytes, st); }
MLB_API int mlb_cast_f2b(void* out, const float* in, long n, float scale, cudaStream_t st) {
  mlb_launch(cast_f2b_k, dim3(gs((n + 3) / 4, 256)), dim3(256), 0, st, (bf16*)out, in, n, scale);
  LAUNCH_RET;
}
MLB_API int mlb_fp8_qdq(void* out, const void* in, long n, float scale, cudaStream_t st) {
  if (n <= 0) return 0;
  if (!(scale > 0.f)) return -3;
  fp8_qdq_k<<<gs(n, 256), 256, 0, st>>>((bf16*)out, (const bf16*)in, n, scale, 1.0f / scale);
  LAUNCH_RET;
}
MLB_API int mlb_cast_b2f(float* out, const void* in, long n, float scale, cudaStream_t st) {
  cast_b2f_k<<<gs(n, 256), 256, 0, st>>>(out, (const bf16*)in, n, scale);
  LAUNCH_RET;
}
MLB_API int mlb_scale_f32(float* x, long n, float scale, cudaStream_t st) {
  scale_f32_k<<<gs(n, 256), 256, 0, st>>>(x, n, scale);
  LAUNCH_RET;
}
MLB_API int mlb_residual_add(void* out, const void* a, const void* b, long n, cudaStream_t st) {
  mlb_launch(residual_add_k, dim3(gs((n + 7) / 8, 256)), dim3(256), 0, st, (bf16*)out, (const bf16*)a, (const bf16*)b, n);
  LAUNCH_RET;
}
MLB_API int mlb_patchify(void* out, const float* px, int B, int Cin, int Himg, int Wimg, int P, cudaStream_t st) {
  long n = (long)B * (Himg / P) * (Wimg / P) * Cin * P * P;
  if (P % 8 == 0 && Wimg % 4 == 0 && ((uintptr_t)px % 16 == 0) && ((uintptr_t)out % 16 == 0)) {
    mlb_launch(patchify8_k, dim3(gs(n / 8, 256)), dim3(256), 0, st, (bf16*)out, px, B, Cin, Himg, Wimg, P);
    LAUNCH_RET;
  }
  patchify_k<<<gs(n, 256), 256, 0, st>>>((bf16*)out, px, B, Cin, Himg, Wimg, P);
  LAUNCH_RET;
}
MLB_API int mlb_add_posembed(void* x, const void* pos, long NP, int n_patch, int vC, cudaStream_t st) {
  add_posembed_k<<<gs(NP * vC, 256), 256, 0, st>>>((bf16*)x, (const bf16*)pos, NP, n_patch, vC);
  LAUNCH_RET;
}
MLB_API int mlb_posembed_grad(float* dpos, const void* dx, long NP, int n_patch, int vC, cudaStream_t st) {
  posembed_grad_k<<<gs((long)n_patch * vC, 256), 256, 0, st>>>(dpos, (const bf16*)dx, NP, n_patch, vC);
  LAUNCH_RET;
}

// ------------------------------------------------------------------ allocation-free RMSNorm backward
// See csrc/no_alloc.h.  Scratch layout inside the fixed array: (296 + RMS_GROUPS) partial rows of MLB_NOALLOC_RMS_MAX_C
// floats, then 32 counters.  In host code the array's name only stands for the symbol; its device address is fetched
// once per device with cudaGetSymbolAddress and that pointer is what the kernel receives.
namespace {
constexpr long NOALLOC_ROWS = 296 + RMS_GROUPS;
constexpr long NOALLOC_FLOATS = NOALLOC_ROWS * MLB_NOALLOC_RMS_MAX_C;
constexpr int NOALLOC_TICKETS = 32;
constexpr int NOALLOC_MAX_DEVICES = 64;
}  // namespace
static __device__ __align__(256) float g_rms_noalloc_scratch[NOALLOC_FLOATS + NOALLOC_TICKETS];

namespace {
float* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};
thread_local char g_noalloc_msg[256] = "";
}  // namespace

MLB_API const char* mlb_rmsnorm_bwd_noalloc_error(void) { return g_noalloc_msg; }

MLB_API int mlb_rmsnorm_bwd_noalloc(void* dx, float* dw, const void* dy, const void* x, const void* w, const float* rstd,
                                    const void* add, long rows, int C, cudaStream_t st) {
  g_noalloc_msg[0] = 0;
  if (C < 1 || rows < 1) {
    snprintf(g_noalloc_msg, sizeof g_noalloc_msg, "rmsnorm_bwd_noalloc: rows=%ld C=%d must be positive", rows, C);
    return MLB_NOALLOC_ERR_TOO_LARGE;
  }
  if (C > MLB_NOALLOC_RMS_MAX_C || (size_t)C * sizeof(float) > 48 * 1024) {
    snprintf(g_noalloc_msg, sizeof g_noalloc_msg,
             "rmsnorm_bwd_noalloc: C=%d exceeds the built-in scratch (max C = %d); use mlb_rmsnorm_bwd with caller scratch", C,
             MLB_NOALLOC_RMS_MAX_C);
    return MLB_NOALLOC_ERR_TOO_LARGE;
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
    snprintf(g_noalloc_msg, sizeof g_noalloc_msg, "rmsnorm_bwd_noalloc: cannot identify the current device (%d, cuda error %d)", dev, (int)e);
    return MLB_NOALLOC_ERR_SETUP;
  }
  if (g_noalloc_ptr[dev] == nullptr) {   // first call on this device: resolve the symbol while that device is current
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_rms_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      snprintf(g_noalloc_msg, sizeof g_noalloc_msg, "rmsnorm_bwd_noalloc: cudaGetSymbolAddress failed on device %d (cuda error %d)", dev, (int)e);
      return MLB_NOALLOC_ERR_SETUP;
    }
    g_noalloc_ptr[dev] = p;
  }
  float* partial = g_noalloc_ptr[dev];
  int* ticket = reinterpret_cast<int*>(partial + NOALLOC_FLOATS);
  // the counters must be zero on entry; the rest of the scratch is fully rewritten before it is read
  e = cudaMemsetAsync(ticket, 0, NOALLOC_TICKETS * sizeof(int), st);
  if (e != cudaSuccess) return (int)e;
  return mlb_rmsnorm_bwd(dx, dw, dy, x, w, rstd, add, rows, C, partial, ticket, st);
}
