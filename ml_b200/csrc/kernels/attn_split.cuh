// Attention with full-precision probabilities on the tensor cores: bidirectional attention (the image encoder's) and causal
// attention at the head sizes the kernels of attn.cu are not built for (any multiple of 16 up to 128 but 64 and 128).
// Included by attn.cu (shares its error word and helpers).
//
// The scalar kernels these replace keep P and dS in fp32, so a bf16 operand alone would lose precision.  Each value goes
// to the tensor core as two bf16 terms, x = hi + lo with hi = bf16(x), lo = bf16(x - hi): 16 significant bits, and Q, K, V, dO are
// bf16 to begin with, so a product costs one more MMA pass and its error (2^-17) disappears under the bf16 rounding of the result.
//
// One CTA of 128 threads (thread = one row of the 128-row tile) per tile, (head, sample); the other operand streams in
// 64-row blocks, double buffered by TMA.  The hi / lo terms are written over the TMEM columns of the scores they came from
// (32 fp32 scores -> 16 columns hi + 16 columns lo) and feed the next product as its A operand from there, so no shared
// memory is spent on them and two (backward) to four (forward) CTAs share an SM: their MMAs, exponentials and loads
// overlap across CTAs, which is why a CTA by itself is a plain sequence.  What bounds it is that sequence's latency, not a
// unit.  64-row blocks because the encoder's sequences are short (197 tokens = 3.1 blocks of 64, 1.5 of 128).
// The next block's scores overwrite those columns.  MMAs are promised to run in the order of their issue only where accumulator and
// shape are the same, so the products that read the columns are waited for first.
// Sequences are the third dimension of the tensor maps: rows past a sample's end arrive as zeros, never as the next
// sample's values (0 * inf would be NaN).  Within a sample the products do multiply a masked key's zero with its V (or Q, K, dO), and the
// two terms of an infinite product may cancel.  With finite values neither matters, and otherwise the row is NaN: such rows are done
// again, at the end, by the scalar kernels' row functions, which skip masked keys.
struct SplitArgs {
  int B, T, H, hd, causal;
  float scale;
  bf16* out;            // forward: out[B*T, C]; backward: dqkv[B*T, 3C]
  float* lse;           // [B,H,T]
  const float* delta;   // [B,H,T]
  const bf16* qkv;
  const bf16* dout;
};

constexpr int SPLIT_THREADS = 128;
constexpr int BOX_BYTES = 64 * 64 * 2;      // one TMA box: 64 rows x 64 columns, 128-byte swizzled rows

// Offsets to a tile's first descriptor, in its address units of 16 bytes, all known at compile time: an issuing thread adds a constant.
// k-step ks of 16 elements of a K-major tile whose 64-column chunks are `chunk` bytes apart; of 16 rows of an MN-major tile.
__host__ __device__ constexpr uint64_t off_k(int ks, int chunk) { return (uint64_t)((ks >> 2) * (chunk >> 4) + (ks & 3) * 2); }
__host__ __device__ constexpr uint64_t off_mn(int ks) { return (uint64_t)(ks * 128); }
__device__ __forceinline__ uint64_t desc64_base_mn(uint32_t base) { return tc::smem_desc_sw128(base, BOX_BYTES, 1024); }
// TMEM column of the hi term of k-step ks (16 rows of the 64-row block); the lo term is 16 columns further
__device__ __forceinline__ uint32_t split_col(int ks) { return (uint32_t)((ks >> 1) * 32 + (ks & 1) * 8); }

__device__ __forceinline__ void split2(uint64_t ab, uint32_t& hi, uint32_t& lo) {      // (two values an instruction, here and in the kernels)
  float a, b;
  upk2(ab, a, b);
  hi = pack_bf16(a, b);
  upk2(add2(ab, pk2(-__uint_as_float(hi << 16), -__uint_as_float(hi & 0xffff0000u))), a, b);
  lo = pack_bf16(a, b);
}

// rows [r0, r0 + 64 * boxes) of `CH` 64-column chunks starting at column x0 of sample z
template <int CH>
__device__ __forceinline__ void split_load(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int x0, int r0, int z, int boxes) {
  for (int c = 0; c < CH; c++)
    for (int i = 0; i < boxes; i++) tc::tma_load_3d(dst + (c * boxes + i) * BOX_BYTES, tm, bar, x0 + c * 64, r0 + i * 64, z);
}

// Rows r0 + bit of the CTA's NaN rows (one word per warp), one after the other by the whole CTA; the tiles' shared memory is free.
// Out of line: its registers must not be the kernels'.
template <int FORM>      // 0 forward, 1 dK and dV, 2 dQ
__device__ __noinline__ void split_redo(uint4 nan_rows, SplitArgs a, int r0, int h, int b, float* sc) {
  for (int i = 0; i < 128; i++) {
    const unsigned word = i < 32 ? nan_rows.x : i < 64 ? nan_rows.y : i < 96 ? nan_rows.z : nan_rows.w;
    if (!(word >> (i & 31) & 1)) continue;
    if (FORM == 1) {      // NaN all over, rightly: nothing to do again
      bool seen = false;
      for (int q = (a.causal ? r0 + i : 0) + threadIdx.x; q < a.T; q += SPLIT_THREADS) {
        const float L = a.lse[((size_t)b * a.H + h) * a.T + q];
        seen |= L != L;
      }
      if (__syncthreads_or(seen)) continue;
    }
    if (FORM == 0) attn_fwd_simt_row(a.out, a.lse, a.qkv, r0 + i, h, b, a.T, a.H, a.hd, a.scale, a.causal, sc);
    else if (FORM == 1) attn_bwd_kv_simt_row(a.out, a.dout, a.qkv, a.lse, a.delta, r0 + i, h, b, a.T, a.H, a.hd, a.scale, a.causal, sc);
    else attn_bwd_q_simt_row(a.out, a.dout, a.qkv, a.lse, a.delta, r0 + i, h, b, a.T, a.H, a.hd, a.scale, a.causal, sc);
    __syncthreads();
  }
}
// acc is NaN from the first value on that is NaN or infinite (times zero), two values an instruction: comparing each one is a chain of
// predicates, 4 us of the dK / dV kernel's 43 (32 x 197 tokens, 12 heads of 64)
__device__ __forceinline__ uint64_t note_nan(uint64_t acc, float x, float y) { return fma2(pk2(x, y), pk2(0.f, 0.f), acc); }
__device__ __forceinline__ bool noted_nan(uint64_t a, uint64_t b) {
  float x, y;
  upk2(add2(a, b), x, y);
  x += y;
  return x != x;
}

// hd columns of the warp's 32 TMEM rows, times f, as bf16 to memory (16-byte aligned, hd a multiple of 16): dst = the lane's row,
// rows `pitch` apart, nlive of them exist.  Whole warp.  Is the lane's row (it may not exist) NaN or infinite somewhere?
template <int HDT>
__device__ __forceinline__ bool split_store_rows(bf16* dst, long pitch, uint32_t taddr, int hd, float f, int lane, int nlive) {
  uint64_t n0 = pk2(0.f, 0.f), n1 = n0;
#pragma unroll
  for (int c = 0; c < HDT; c += 32) {
    uint32_t r[32];
    tc::tmem_ld32_wait(taddr + c, r);
#pragma unroll
    for (int g = 0; g < 32; g += 16) {
      if (c + g >= hd) break;
#pragma unroll
      for (int i = g; i < g + 16; i += 4) {
        n0 = note_nan(n0, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
        n1 = note_nan(n1, __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
      }
    }
    uint4 u[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const float* x = reinterpret_cast<const float*>(r) + v * 8;
      u[v] = make_uint4(pack_bf16(x[0] * f, x[1] * f), pack_bf16(x[2] * f, x[3] * f), pack_bf16(x[4] * f, x[5] * f), pack_bf16(x[6] * f, x[7] * f));
    }
    quad_transpose(u, lane);
    const int q = lane & 3;
    bf16* base = dst - q * pitch + c + q * 8;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if ((lane & ~3) + k < nlive && c + q * 8 < hd) *reinterpret_cast<uint4*>(base + k * pitch) = u[k];
  }
  return noted_nan(n0, n1);
}

template <int HDT>
struct SplitFwdSmem {
  static constexpr int CH = HDT == 128 ? 2 : 1;
  static constexpr int Q = 0;
  static constexpr int K = Q + 2 * CH * BOX_BYTES;      // 2 buffers
  static constexpr int V = K + 2 * CH * BOX_BYTES;      // 2 buffers
  static constexpr int BAR = V + 2 * CH * BOX_BYTES;
  static constexpr int TOTAL = BAR + 128 + 1024;
};

template <int HDT>
__global__ void __launch_bounds__(SPLIT_THREADS) attn_split_fwd_k(const __grid_constant__ CUtensorMap tm, const SplitArgs a) {
  __shared__ __align__(16) unsigned s_nan[4];      // rows to do again
  using S = SplitFwdSmem<HDT>;
  constexpr int CH = S::CH;
  constexpr uint32_t TMEM_COLS = HDT == 128 ? 256 : 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_q = bars, *bar_k = bars + 1 /*[2]*/, *bar_v = bars + 3 /*[2]*/, *bar_s = bars + 5, *bar_o = bars + 6, *bar_end = bars + 7;
  uint32_t* tmem_slot = (uint32_t*)(bars + 8);
  volatile int* s_abort = (volatile int*)(bars + 9);
  if (attn_given_up()) { mlb_pdl_sync(); return; }      // (nobody behind this kernel starts before the one in front of it has ended)

  const int ntile = (a.T + 127) / 128;
  const int qt = ntile - 1 - (int)blockIdx.x, h = blockIdx.y, b = blockIdx.z;     // (causal: longest rows first)
  const int q0 = qt * 128, C = a.H * a.hd;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int i = 0; i < 8; i++) tc::mbar_init(&bars[i], 1);
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
  }
  // The threads that multiply and that load (whole warps ask): of two warps, each has its own rows to work on besides
  auto leader = [&]() -> bool { return warp == 0 && tc::elect_one(); };
  auto loader = [&]() -> bool { return warp == 3 && tc::elect_one(); };
  if (warp == 0) tc::tmem_alloc(tmem_slot, TMEM_COLS);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  mlb_pdl_sync();
  const uint32_t t_s = *tmem_slot, t_o = t_s + 64, lane_addr = (uint32_t)(warp * 32) << 16;
  // Bounded, sticky: after one expiry every later wait of the CTA returns at once and all threads keep the same sequence of barriers
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) { return tc::mbar_wait_sticky(bar, phase, where, s_abort); };
  const int nblk = (a.T + 63) / 64;
  const int nkb = a.causal ? min(nblk, q0 / 64 + 2) : nblk;
  const uint32_t idesc_s = tc::idesc_bf16(128, 64, 0, 0), idesc_o = tc::idesc_bf16(128, a.hd, 0, 1);
  const int nks = a.hd >> 4;
  const uint64_t dQ = desc_base_k(tc::smem_u32(smem + S::Q)), dK0 = desc_base_k(tc::smem_u32(smem + S::K)),
                 dV0 = desc64_base_mn(tc::smem_u32(smem + S::V));
  int loads = 0;      // blocks of K and V asked for (loader)
  auto load_kv = [&](int j) {
    const int sl = j & 1;
    loads = j + 1;
    tc::mbar_expect_tx(&bar_k[sl], CH * BOX_BYTES);
    split_load<CH>(smem + S::K + sl * CH * BOX_BYTES, &tm, &bar_k[sl], C + h * a.hd, j * 64, b, 1);
    tc::mbar_expect_tx(&bar_v[sl], CH * BOX_BYTES);
    split_load<CH>(smem + S::V + sl * CH * BOX_BYTES, &tm, &bar_v[sl], 2 * C + h * a.hd, j * 64, b, 1);
  };
  auto issue_s = [&](int j) {
    wait(&bar_k[j & 1], (j >> 1) & 1, 41);
    tc::tc_fence_after();
    const uint64_t dK = dK0 + (uint64_t)((j & 1) * (CH * BOX_BYTES >> 4));
    if (!*s_abort) {
#pragma unroll
      for (int ks = 0; ks < HDT / 16; ks++)
        if (ks < nks) tc::mma_bf16_ss(t_s, dQ + off_k(ks, TILE_BYTES), dK + off_k(ks, BOX_BYTES), idesc_s, ks > 0);
    }
    tc::mma_commit(bar_s);
  };
  if (loader()) {
    tc::mbar_expect_tx(bar_q, 2 * CH * BOX_BYTES);
    split_load<CH>(smem + S::Q, &tm, bar_q, h * a.hd, q0, b, 2);
    load_kv(0);
  }
  if (leader()) {
    wait(bar_q, 0, 40);
    issue_s(0);
  }
  const float sl2 = a.scale * LOG2E;
  const int qrow = q0 + tid;
  float m = -INFINITY, l = 0.f;
  float o[HDT];
#pragma unroll
  for (int i = 0; i < HDT; i++) o[i] = 0.f;
  for (int j = 0; j < nkb; j++) {
    if (loader() && j + 1 < nkb && !*s_abort) load_kv(j + 1);     // (block j - 1, the buffers' last reader, is complete: bar_o of it was waited for)
    wait(bar_s, j & 1, 42);
    __syncwarp();
    tc::tc_fence_after();
    const int k0 = j * 64;
    const int last = a.causal ? min(qrow, a.T - 1) : a.T - 1;      // last key this row sees
    // The scores are read twice, 32 at a time (once for the maximum): a row's 64 in registers on top of its HDT output columns
    // would cost a resident CTA.  At 128 output columns it is more than that: the 255 registers it takes, and the build (nvcc 12.9) then
    // forms the operand addresses of this loop's score products wrongly from the second k-step on (the first is right, the rest come
    // from elsewhere; the descriptors' values in the source are right, and the prologue's product is).
    auto load_scores = [&](int half, uint32_t (&r)[32]) {
      tc::tmem_ld32_wait(t_s + half * 32 + lane_addr, r);
      if (k0 + half * 32 + 31 > last) {
#pragma unroll
        for (int i = 0; i < 32; i++)
          if (k0 + half * 32 + i > last) r[i] = 0xff800000u;
      }
    };
    // (an encoder's sequence is a square and the class token: its last block has few keys, and the second half of it none)
    const bool both = k0 + 32 < a.T;
    float top = -INFINITY;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      if (half && !both) break;
      uint32_t r[32];
      load_scores(half, r);
#pragma unroll
      for (int i = 0; i < 32; i += 2) top = max3(top, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
    }
    const float mx = fmaxf(m, top * sl2);      // (the largest product is that of the largest score)
    const float mu = mx == -INFINITY ? 0.f : mx;      // nothing finite seen yet: exp2(-inf - 0) = 0
    const float alpha = ex2_approx(m - mu);
    const uint64_t sl2x2 = pk2(sl2, sl2), nmu2 = pk2(-mu, -mu), alpha2 = pk2(alpha, alpha);
    m = mx;
    float rs = 0.f;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      if (half && !both) break;
      uint32_t r[32], hi[16], lo[16];
      load_scores(half, r);
#pragma unroll
      for (int i = 0; i < 16; i++) {
        float p0, p1;
        upk2(fma2(pk2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), sl2x2, nmu2), p0, p1);
        p0 = ex2_approx(p0);
        p1 = ex2_approx(p1);
        rs += p0 + p1;
        split2(pk2(p0, p1), hi[i], lo[i]);
      }
      tc::tmem_st16(t_s + half * 32 + lane_addr, hi);
      tc::tmem_st16(t_s + half * 32 + 16 + lane_addr, lo);
    }
    l = l * alpha + rs;
    tc::tmem_st_wait();
    tc::tc_fence_before();
    __syncthreads();
    if (leader()) {
      wait(&bar_v[j & 1], (j >> 1) & 1, 43);
      tc::tc_fence_after();
      const uint64_t dV = dV0 + (uint64_t)((j & 1) * (CH * BOX_BYTES >> 4));
      if (!*s_abort) {
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
          if (ks >= 2 && !both) break;
          tc::mma_bf16_ts(t_o, t_s + split_col(ks), dV + off_mn(ks), idesc_o, ks > 0);
          tc::mma_bf16_ts(t_o, t_s + split_col(ks) + 16, dV + off_mn(ks), idesc_o, 1);
        }
      }
      tc::mma_commit(bar_o);
      if (j + 1 < nkb) {      // these scores replace P, which the product above reads
        wait(bar_o, j & 1, 44);
        issue_s(j + 1);
      }
    }
    wait(bar_o, j & 1, 44);
    __syncwarp();
    tc::tc_fence_after();
#pragma unroll
    for (int c = 0; c < HDT; c += 32) {
      uint32_t ro[32];
      tc::tmem_ld32_wait(t_o + c + lane_addr, ro);
#pragma unroll
      for (int i = 0; i < 32; i += 2)
        upk2(fma2(pk2(o[c + i], o[c + i + 1]), alpha2, pk2(__uint_as_float(ro[i]), __uint_as_float(ro[i + 1]))), o[c + i], o[c + i + 1]);
    }
    tc::tc_fence_before();
  }
  const float inv = 1.f / l;
  uint64_t n0 = pk2(0.f, 0.f), n1 = n0;
  const int lane = tid & 31, nlive = *s_abort ? 0 : a.T - (qrow - lane);
  bf16* dst = a.out + ((size_t)b * a.T + qrow) * C + h * a.hd;
  __syncwarp();
#pragma unroll
  for (int c = 0; c < HDT; c += 32) {
    uint4 u[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const float* x = o + c + v * 8;
      if (c + v * 8 < a.hd) {
        n0 = note_nan(note_nan(n0, x[0], x[1]), x[2], x[3]);
        n1 = note_nan(note_nan(n1, x[4], x[5]), x[6], x[7]);
      }
      u[v] = make_uint4(pack_bf16(x[0] * inv, x[1] * inv), pack_bf16(x[2] * inv, x[3] * inv), pack_bf16(x[4] * inv, x[5] * inv),
                        pack_bf16(x[6] * inv, x[7] * inv));
    }
    quad_transpose(u, lane);
    const int q = lane & 3;
    bf16* base = dst - q * (long)C + c + q * 8;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if ((lane & ~3) + k < nlive && c + q * 8 < a.hd) *reinterpret_cast<uint4*>(base + k * (long)C) = u[k];
  }
  if (lane < nlive) a.lse[((size_t)b * a.H + h) * a.T + qrow] = (m + log2f(l)) * LN2;
  const bool nan = noted_nan(n0, n1) && l == l;      // (a NaN among the scores is in all of the row, rightly)
  const unsigned rows = __ballot_sync(0xffffffffu, nan && lane < nlive);
  if (lane == 0) s_nan[warp] = rows;
  tc::tc_fence_before();
  __syncthreads();
  if (*s_abort) {
    if (leader()) {
      tc::report_given_up(s_abort);
      tc::mma_commit(bar_end);
      attn_settle(bar_end, 1);
    }
    if (loader()) {
      attn_settle(bar_q, 1);
      for (int sl = 0; sl < 2; sl++) {
        attn_settle(&bar_k[sl], (loads + 1 - sl) / 2);
        attn_settle(&bar_v[sl], (loads + 1 - sl) / 2);
      }
    }
    __syncthreads();
  }
  if (warp == 0) tc::tmem_dealloc(t_s, TMEM_COLS);
  const uint4 again = *reinterpret_cast<const uint4*>(s_nan);
  if (again.x | again.y | again.z | again.w) split_redo<0>(again, a, q0, h, b, (float*)smem);
}

// Backward, KV = true: dK and dV of a 128-key tile, streaming Q / dO;  KV = false: dQ of a 128-query tile, streaming K / V.
// X, Y are the resident tiles (K, V or Q, dO), x, y the streamed ones (Q, dO or K, V); per block
//   s = X x^T,  d = Y y^T  (scores, and the gradient of the probabilities; transposed in the KV form)
//   p = exp2(s c - lse),  g = p (d - delta);    KV: dV += p dO, dK += g Q      else: dQ += g K
template <int HDT, bool KV>
struct SplitBwdSmem {
  static constexpr int CH = HDT == 128 ? 2 : 1;
  static constexpr int RX = 0;
  static constexpr int RY = RX + 2 * CH * BOX_BYTES;
  static constexpr int SX = RY + 2 * CH * BOX_BYTES;      // 2 buffers
  static constexpr int SY = SX + 2 * CH * BOX_BYTES;      // 2 buffers
  static constexpr int STAT = SY + 2 * CH * BOX_BYTES;    // 2 buffers x (lse [64], delta [64])
  static constexpr int BAR = STAT + 1024;
  static constexpr int TOTAL = BAR + 128 + 1024;
};

template <int HDT, bool KV>
__global__ void __launch_bounds__(SPLIT_THREADS) attn_split_bwd_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do,
                                                                  const SplitArgs a) {
  __shared__ __align__(16) unsigned s_nan[4];      // rows to do again
  using S = SplitBwdSmem<HDT, KV>;
  constexpr int CH = S::CH;
  constexpr uint32_t TMEM_COLS = (KV && HDT == 128) ? 512 : 256;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_r = bars, *bar_x = bars + 1 /*[2]*/, *bar_s = bars + 3, *bar_g = bars + 4, *bar_end = bars + 5;
  uint32_t* tmem_slot = (uint32_t*)(bars + 6);
  volatile int* s_abort = (volatile int*)(bars + 7);
  float* stat = (float*)(smem + S::STAT);
  if (attn_given_up()) { mlb_pdl_sync(); return; }      // (nobody behind this kernel starts before the one in front of it has ended)

  const int tid = threadIdx.x, warp = tid >> 5;
  const int ntile = (a.T + 127) / 128;
  const int tile = KV ? (int)blockIdx.x : ntile - 1 - (int)blockIdx.x, h = blockIdx.y, b = blockIdx.z;   // (causal: longest first)
  const int r0 = tile * 128, C = a.H * a.hd, xh = h * a.hd;
  if (tid == 0) {
    for (int i = 0; i < 6; i++) tc::mbar_init(&bars[i], 1);
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
    tc::tma_prefetch_desc(&tm_do);
  }
  // The threads that multiply and that load (whole warps ask): of two warps, each has its own rows to work on besides
  auto leader = [&]() -> bool { return warp == 0 && tc::elect_one(); };
  auto loader = [&]() -> bool { return warp == 3 && tc::elect_one(); };
  if (warp == 0) tc::tmem_alloc(tmem_slot, TMEM_COLS);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  mlb_pdl_sync();
  const uint32_t t_s = *tmem_slot, t_d = t_s + 64, t_a0 = t_s + 128, t_a1 = t_a0 + HDT;      // a0: dV or dQ, a1: dK
  const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) { return tc::mbar_wait_sticky(bar, phase, where, s_abort); };
  const int nblk = (a.T + 63) / 64;
  const int i0 = (KV && a.causal) ? r0 / 64 : 0;
  const int n = (!KV && a.causal) ? min(nblk, r0 / 64 + 2) : nblk - i0;
  const uint32_t idesc_s = tc::idesc_bf16(128, 64, 0, 0), idesc_g = tc::idesc_bf16(128, a.hd, 0, 1);
  const int nks = a.hd >> 4;
  const size_t si = ((size_t)b * a.H + h) * a.T;
  const uint64_t drx = desc_base_k(tc::smem_u32(smem + S::RX)), dry = desc_base_k(tc::smem_u32(smem + S::RY));
  const uint64_t dsx = desc_base_k(tc::smem_u32(smem + S::SX)), dsy = desc_base_k(tc::smem_u32(smem + S::SY));      // as B of the scores
  const uint64_t gsx = desc64_base_mn(tc::smem_u32(smem + S::SX)), gsy = desc64_base_mn(tc::smem_u32(smem + S::SY));   // as B of the gradients
  int loads = 0;      // streamed blocks asked for (loader)
  auto load_x = [&](int it) {
    const int sl = it & 1, y = (i0 + it) * 64;
    loads = it + 1;
    tc::mbar_expect_tx(&bar_x[sl], 2 * CH * BOX_BYTES);
    split_load<CH>(smem + S::SX + sl * CH * BOX_BYTES, &tm, &bar_x[sl], KV ? xh : C + xh, y, b, 1);
    split_load<CH>(smem + S::SY + sl * CH * BOX_BYTES, KV ? &tm_do : &tm, &bar_x[sl], KV ? xh : 2 * C + xh, y, b, 1);
  };
  auto issue_scores = [&](int it) {
    const int sl = it & 1;
    wait(&bar_x[sl], (it >> 1) & 1, 46);
    tc::tc_fence_after();
    const uint64_t slot = (uint64_t)(sl * (CH * BOX_BYTES >> 4)), sx = dsx + slot, sy = dsy + slot;
    if (!*s_abort) {
#pragma unroll
      for (int ks = 0; ks < HDT / 16; ks++)
        if (ks < nks) tc::mma_bf16_ss(t_s, drx + off_k(ks, TILE_BYTES), sx + off_k(ks, BOX_BYTES), idesc_s, ks > 0);
#pragma unroll
      for (int ks = 0; ks < HDT / 16; ks++)
        if (ks < nks) tc::mma_bf16_ss(t_d, dry + off_k(ks, TILE_BYTES), sy + off_k(ks, BOX_BYTES), idesc_s, ks > 0);
    }
  };
  // statistics of the 64 streamed queries (KV form), -lse log2 e and -delta; a query past the end has lse = +inf: p = 0
  auto load_stat = [&](int it) {
    const int q = (i0 + it) * 64 + (tid & 63);
    float* st = stat + (it & 1) * 128;
    if (tid < 64) st[tid] = q < a.T ? -a.lse[si + q] * LOG2E : -INFINITY;
    else st[tid] = q < a.T ? -a.delta[si + q] : 0.f;
  };
  if (loader()) {
    tc::mbar_expect_tx(bar_r, 4 * CH * BOX_BYTES);
    split_load<CH>(smem + S::RX, &tm, bar_r, KV ? C + xh : xh, r0, b, 2);
    split_load<CH>(smem + S::RY, KV ? &tm : &tm_do, bar_r, KV ? 2 * C + xh : xh, r0, b, 2);
    load_x(0);
  }
  if (leader()) {
    wait(bar_r, 0, 45);
    issue_scores(0);
    tc::mma_commit(bar_s);
  }
  const float sl2 = a.scale * LOG2E;
  const int row = r0 + tid;
  const uint64_t sl2x2 = pk2(sl2, sl2);
  float nlse_r = -INFINITY, ndelta_r = 0.f;      // dQ form: this thread's query, -lse log2 e and -delta
  if (KV) {
    load_stat(0);
  } else if (row < a.T) {
    nlse_r = -a.lse[si + row] * LOG2E;
    ndelta_r = -a.delta[si + row];
  }
  __syncthreads();
  for (int it = 0; it < n; it++) {
    wait(bar_s, it & 1, 47);
    __syncwarp();
    tc::tc_fence_after();
    if (loader() && it + 1 < n && !*s_abort) load_x(it + 1);      // every MMA issued so far is complete: the other buffer is free
    const int c0 = (i0 + it) * 64;
    const float* st = stat + (it & 1) * 128;
    const bool both = c0 + 32 < a.T;      // (as in forward)
    const bool cut = KV ? a.causal && c0 < r0 + 128 : (a.causal && c0 + 63 > r0) || c0 + 64 > a.T;      // is any of the tile's pairs masked?
#pragma unroll
    for (int half = 0; half < 2; half++) {
      if (half && !both) break;
      uint32_t rs[32], rd[32];
      tc::tmem_ld32x2_wait(t_s + half * 32 + lane_addr, rs, t_d + half * 32 + lane_addr, rd);
      float p[32];
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 nl = KV ? *reinterpret_cast<const float4*>(st + half * 32 + e) : make_float4(nlse_r, nlse_r, nlse_r, nlse_r);
        float z[4];
        upk2(fma2(pk2(__uint_as_float(rs[e]), __uint_as_float(rs[e + 1])), sl2x2, pk2(nl.x, nl.y)), z[0], z[1]);
        upk2(fma2(pk2(__uint_as_float(rs[e + 2]), __uint_as_float(rs[e + 3])), sl2x2, pk2(nl.z, nl.w)), z[2], z[3]);
#pragma unroll
        for (int x = 0; x < 4; x++) p[e + x] = ex2_approx(z[x]);
      }
      if (cut) {      // causal: the key may not lie behind the query; dQ form: keys past the end are not there (KV form: lse = +inf)
#pragma unroll
        for (int e = 0; e < 32; e++) {
          const int col = c0 + half * 32 + e;
          if (KV ? col < row : ((a.causal && col > row) || col >= a.T)) p[e] = 0.f;
        }
      }
      uint32_t hi[16], lo[16], gh[16], gl[16];
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 nd = KV ? *reinterpret_cast<const float4*>(st + 64 + half * 32 + e) : make_float4(ndelta_r, ndelta_r, ndelta_r, ndelta_r);
        const uint64_t p01 = pk2(p[e], p[e + 1]), p23 = pk2(p[e + 2], p[e + 3]);
        if (KV) {
          split2(p01, hi[e / 2], lo[e / 2]);
          split2(p23, hi[e / 2 + 1], lo[e / 2 + 1]);
        }
        split2(mul2(p01, add2(pk2(__uint_as_float(rd[e]), __uint_as_float(rd[e + 1])), pk2(nd.x, nd.y))), gh[e / 2], gl[e / 2]);
        split2(mul2(p23, add2(pk2(__uint_as_float(rd[e + 2]), __uint_as_float(rd[e + 3])), pk2(nd.z, nd.w))), gh[e / 2 + 1], gl[e / 2 + 1]);
      }
      if (KV) {
        tc::tmem_st16(t_s + half * 32 + lane_addr, hi);
        tc::tmem_st16(t_s + half * 32 + 16 + lane_addr, lo);
      }
      tc::tmem_st16(t_d + half * 32 + lane_addr, gh);
      tc::tmem_st16(t_d + half * 32 + 16 + lane_addr, gl);
    }
    tc::tmem_st_wait();
    if (KV && it + 1 < n) load_stat(it + 1);
    tc::tc_fence_before();
    __syncthreads();
    if (leader()) {
      tc::tc_fence_after();
      const uint64_t slot = (uint64_t)((it & 1) * (CH * BOX_BYTES >> 4)), sx = gsx + slot, sy = gsy + slot;
      if (!*s_abort) {
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
          if (ks >= 2 && !both) break;
          if (KV) {
            tc::mma_bf16_ts(t_a0, t_s + split_col(ks), sy + off_mn(ks), idesc_g, (it > 0 || ks > 0));
            tc::mma_bf16_ts(t_a0, t_s + split_col(ks) + 16, sy + off_mn(ks), idesc_g, 1);
          }
          tc::mma_bf16_ts(KV ? t_a1 : t_a0, t_d + split_col(ks), sx + off_mn(ks), idesc_g, (it > 0 || ks > 0));
          tc::mma_bf16_ts(KV ? t_a1 : t_a0, t_d + split_col(ks) + 16, sx + off_mn(ks), idesc_g, 1);
        }
      }
      if (it + 1 < n) {      // these scores replace p and g, which the products above read
        tc::mma_commit(bar_g);
        wait(bar_g, it & 1, 49);
        issue_scores(it + 1);
      }
      tc::mma_commit(bar_s);
    }
  }
  wait(bar_s, n & 1, 48);
  __syncwarp();
  tc::tc_fence_after();
  const int lane = tid & 31, nlive = *s_abort ? 0 : a.T - (row - lane);
  bf16* dst = a.out + ((size_t)b * a.T + row) * 3 * C + xh;
  __syncwarp();
  // (a query whose lse or delta is NaN makes all of its dQ NaN, rightly, and a NaN lse all of the dK and dV that see it)
  bool nan = split_store_rows<HDT>(KV ? dst + C : dst, 3L * C, (KV ? t_a1 : t_a0) + lane_addr, a.hd, a.scale, lane, nlive);
  if (KV) nan |= split_store_rows<HDT>(dst + 2 * C, 3L * C, t_a0 + lane_addr, a.hd, 1.f, lane, nlive);
  if (!KV) nan = nan && nlse_r == nlse_r && ndelta_r == ndelta_r;
  const unsigned rows = __ballot_sync(0xffffffffu, nan && lane < nlive);
  if (lane == 0) s_nan[warp] = rows;
  tc::tc_fence_before();
  __syncthreads();
  if (*s_abort) {
    if (leader()) {
      tc::report_given_up(s_abort);
      tc::mma_commit(bar_end);
      attn_settle(bar_end, 1);
    }
    if (loader()) {
      attn_settle(bar_r, 1);
      for (int sl = 0; sl < 2; sl++) attn_settle(&bar_x[sl], (loads + 1 - sl) / 2);
    }
    __syncthreads();
  }
  if (warp == 0) tc::tmem_dealloc(t_s, TMEM_COLS);
  const uint4 again = *reinterpret_cast<const uint4*>(s_nan);
  if (again.x | again.y | again.z | again.w) split_redo<KV ? 1 : 2>(again, a, r0, h, b, (float*)smem);
}

// Do the kernels start under the one before them?  Four CTAs of the forward fit an SM at head sizes up to 64, two of the backward (at 128: two and
// one), so the limit is two to eight waves.  It is where the gain has become small, not where something gets slower: forward + backward without a
// mask, 197 tokens, 12 heads of 64, us apart and early (kernels a tenth slower than these): 0.6 CTAs per SM 43.1 and 38.3, 2.6 73.6 and 64.5, 5.2 114.6 and 107.7, 7.8 162.8 and
// 156.7, 10 212.9 and 207.7, 21 383.9 and 377.7.  Slower where the backward's CTAs are just short of one wave, which the early ones
// take up unevenly (1.9: 51.2 and 53.0; 577 tokens, 1.6: 96.7 and 107.0).
static bool split_early(const SplitArgs& a) { return (long)((a.T + 127) / 128) * a.H * a.B <= 8L * mlb_sm_count(); }
template <int HDT>
static int split_fwd_launch(const CUtensorMap* tm, const SplitArgs& a, cudaStream_t st) {
  static int once = (int)cudaFuncSetAttribute(attn_split_fwd_k<HDT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitFwdSmem<HDT>::TOTAL);
  if (once) return once;
  mlb_launch_tmem(split_early(a), attn_split_fwd_k<HDT>, dim3((a.T + 127) / 128, a.H, a.B), dim3(SPLIT_THREADS), SplitFwdSmem<HDT>::TOTAL, st, *tm, a);
  return (int)cudaGetLastError();
}
template <int HDT>
static int split_bwd_launch(const CUtensorMap* tm, const CUtensorMap* td, const SplitArgs& a, cudaStream_t st) {
  static int once = (int)cudaFuncSetAttribute(attn_split_bwd_k<HDT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitBwdSmem<HDT, true>::TOTAL) |
                    (int)cudaFuncSetAttribute(attn_split_bwd_k<HDT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitBwdSmem<HDT, false>::TOTAL);
  if (once) return once;
  const dim3 grid((a.T + 127) / 128, a.H, a.B);
  mlb_launch_tmem(split_early(a), attn_split_bwd_k<HDT, true>, grid, dim3(SPLIT_THREADS), SplitBwdSmem<HDT, true>::TOTAL, st, *tm, *td, a);
  mlb_launch_tmem(split_early(a), attn_split_bwd_k<HDT, false>, grid, dim3(SPLIT_THREADS), SplitBwdSmem<HDT, false>::TOTAL, st, *tm, *td, a);
  return (int)cudaGetLastError();
}

// The shapes the kernels above take: head sizes that are multiples of the MMA's k-step, 16-byte aligned rows and heads.
// T up to what the scalar kernels' score row in shared memory allows, so that a call is taken or refused as there.
static bool split_ok(const void* qkv, const void* a, const void* b, int T, int hd, size_t floats_per_key) {
  return !g_attn_force_simt && hd % 16 == 0 && hd >= 16 && hd <= 128 && (((uintptr_t)qkv | (uintptr_t)a | (uintptr_t)b) & 15) == 0 &&
         (floats_per_key * T + 32) * sizeof(float) <= 48 * 1024;
}
static int split_fwd(void* out, float* lse, const void* qkv, int B, int T, int H, int hd, int causal, cudaStream_t st) {
  const CUtensorMap* tm = mlb_tmap_seq3d_cached(qkv, B, T, 3L * H * hd);
  if (!tm) return -2;
  SplitArgs a{B, T, H, hd, causal, 1.0f / sqrtf((float)hd), (bf16*)out, lse, nullptr, (const bf16*)qkv, nullptr};
  return hd <= 32 ? split_fwd_launch<32>(tm, a, st) : hd <= 64 ? split_fwd_launch<64>(tm, a, st) : split_fwd_launch<128>(tm, a, st);
}
// `delta` = rowsum(dO * O) is already there
static int split_bwd(void* dqkv, const void* dout, const void* qkv, const float* lse, const float* delta, int B, int T, int H, int hd, int causal,
                     cudaStream_t st) {
  const CUtensorMap* tm = mlb_tmap_seq3d_cached(qkv, B, T, 3L * H * hd);
  const CUtensorMap* td = mlb_tmap_seq3d_cached(dout, B, T, (long)H * hd);
  if (!tm || !td) return -2;
  SplitArgs a{B, T, H, hd, causal, 1.0f / sqrtf((float)hd), (bf16*)dqkv, const_cast<float*>(lse), delta, (const bf16*)qkv, (const bf16*)dout};
  return hd <= 32 ? split_bwd_launch<32>(tm, td, a, st) : hd <= 64 ? split_bwd_launch<64>(tm, td, a, st) : split_bwd_launch<128>(tm, td, a, st);
}
