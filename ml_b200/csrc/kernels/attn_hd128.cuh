// Causal attention at head size 128, forward and backward.  Included by attn.cu behind attn_split.cuh (shares their helpers).
//
// At this head size the four products of a forward step over 256 queries x 128 keys take the tensor core as long as their
// exponentials take the special-function units (2048 cycles each), and in backward the products lead (2048 / 1536 cycles against
// 1024), so the kernels are built around never letting one wait for the other; tensor memory is the constraint (a 128 x 128
// fp32 tile is 128 of its 512 columns).  P and dS are written as bf16 pairs over the score columns they came from and are read
// from there as the A operand of the next product: no shared memory, and no columns of their own.  MMAs issued by one
// thread run in order, so a product that overwrites such columns is simply issued behind the one that reads them.
// All three kernels are persistent, one CTA per SM over a balanced table of items (attn_schedule); every wait is bounded and
// sticky (after one expiry the CTA's later waits return at once and its roles still walk the same sequence of barriers).
// Loads go through per-sequence tensor maps: rows past a sample's end are zeros.
constexpr int H128 = 128;
constexpr int T128_BYTES = 2 * TILE_BYTES;      // one [128 x 128] bf16 tile: two 64-column chunks
constexpr uint64_t T128_UNITS = T128_BYTES >> 4;   // the same in descriptor address units

struct Fwd128Smem {
  static constexpr int Q = 0;                              // one tile per query tile of the pair
  static constexpr int K = Q + 2 * T128_BYTES;             // 2 slots
  static constexpr int V = K + 2 * T128_BYTES;             // 2 slots
  static constexpr int OST = V + 2 * T128_BYTES;           // O staging: 8 warps x [32 rows x 128 B], swizzled
  static constexpr int BAR = OST + 8 * 4096;
  static constexpr int SCHED = BAR + 256;                  // this CTA's first 64 items
  static constexpr int TOTAL = SCHED + 256 + 1024;
};
constexpr int FWD128_THREADS = 11 * 32;      // 4 + 4 softmax warps (tile 0 / 1), MMA warp of tile 0, loader, MMA warp of tile 1

// This CTA's li-th work item, or -1
struct ItemList {
  const int* row;
  const int* head;      // shared-memory copy of the first 64 entries
  int first, stride, total;
  __device__ __forceinline__ int at(int li) const {
    if (row) return li < 64 ? head[li] : __ldg(row + li);
    const int x = first + li * stride;
    return x < total ? x : -1;
  }
};

// Forward over pairs of query tiles (256 queries) of one (sample, head).  TMEM: S0 S1 O0 O1.  Per tile and key block
//   S = Q K^T -> one thread per row: m, p = exp2(s c - m) -> P over S -> O += P V -> next S
// is a chain; the two tiles run it out of phase, one on the tensor core while the other takes exponentials.  P V starts
// when the first half of P is there.  m is the maximum of an earlier block as long as no row of the warp has grown past it
// by more than 2^8; only then O (in place) and l are rescaled.
__global__ void __launch_bounds__(FWD128_THREADS, 1) attn_fwd128_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_out,
                                                                   const AttnArgs a) {
  mlb_pdl_sync();
  using S = Fwd128Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_q = bars, *bar_qf = bars + 2, *bar_k = bars + 4, *bar_kf = bars + 6, *bar_v = bars + 8, *bar_vf = bars + 10, *bar_s = bars + 12,
           *bar_pa = bars + 14, *bar_pb = bars + 16, *bar_o = bars + 18;      // [2] each: per tile (q, s, p, o) or slot (k, v)
  uint32_t* tmem_slot = (uint32_t*)(bars + 20);
  volatile int* s_abort = (volatile int*)(bars + 21);
  if (attn_given_up()) return;
  const int nq = (a.T + 127) / 128, npair = (nq + 1) / 2, BH = a.B * a.H, C = a.H * H128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* srow = a.sched ? a.sched + (size_t)blockIdx.x * a.sched_stride : nullptr;
  int* s_sched = (int*)(smem + S::SCHED);
  if (srow && tid < 64) s_sched[tid] = tid < a.sched_stride ? __ldg(srow + tid) : -1;
  const ItemList items{srow, s_sched, (int)blockIdx.x, (int)gridDim.x, npair * BH};
  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      tc::mbar_init(&bar_q[i], 1); tc::mbar_init(&bar_qf[i], 1); tc::mbar_init(&bar_k[i], 1); tc::mbar_init(&bar_kf[i], 2);
      tc::mbar_init(&bar_v[i], 1); tc::mbar_init(&bar_vf[i], 2); tc::mbar_init(&bar_s[i], 1); tc::mbar_init(&bar_pa[i], 4);
      tc::mbar_init(&bar_pb[i], 4); tc::mbar_init(&bar_o[i], 1);
    }
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
    tc::tma_prefetch_desc(&tm_out);
  }
  if (warp == 8) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) {
    if (tc::mbar_try(bar, phase) || *s_abort) return;
    if (!tc::mbar_wait(bar, phase, where)) *s_abort = 1;
  };
  // item w = pair (heaviest first) of (sample, head); tile t of it has n(t) key blocks (none when the pair has no second tile)
  struct Item { int pair, b, h, nkb; };
  auto item_of = [&](int w) {
    const int bh = w % BH, pair = npair - 1 - w / BH;
    return Item{pair, bh / a.H, bh % a.H, min(2 * pair + 2, nq)};
  };
  auto blocks_of = [&](const Item& it, int t) { return 2 * it.pair + t < nq ? 2 * it.pair + t + 1 : 0; };

  if (warp == 9) {
    if (lane == 0) {
      int g = 0, cq[2] = {0, 0};
      for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
        const Item it = item_of(w);
        auto load_q = [&](int t) {
          if (blocks_of(it, t) == 0) return;
          if (cq[t] > 0) wait(&bar_qf[t], (cq[t] - 1) & 1, 50);
          cq[t]++;
          tc::mbar_expect_tx(&bar_q[t], T128_BYTES);
          split_load<2>(smem + S::Q + t * T128_BYTES, &tm, &bar_q[t], it.h * H128, (2 * it.pair + t) * 128, it.b, 2);
        };
        for (int j = 0; j < it.nkb; j++, g++) {
          const int sl = g & 1, ph = ((g >> 1) + 1) & 1;
          if (g >= 2) wait(&bar_kf[sl], ph, 51);
          tc::mbar_expect_tx(&bar_k[sl], T128_BYTES);
          split_load<2>(smem + S::K + sl * T128_BYTES, &tm, &bar_k[sl], C + it.h * H128, j * 128, it.b, 2);
          if (j == 0) { load_q(0); load_q(1); }
          if (g >= 2) wait(&bar_vf[sl], ph, 52);
          tc::mbar_expect_tx(&bar_v[sl], T128_BYTES);
          split_load<2>(smem + S::V + sl * T128_BYTES, &tm, &bar_v[sl], 2 * C + it.h * H128, j * 128, it.b, 2);
        }
      }
    }
  } else if (warp == 8 || warp == 10) {
    if (lane == 0) {
      const int t = warp == 8 ? 0 : 1;
      constexpr uint32_t idesc_s = tc::idesc_bf16(128, 128, 0, 0), idesc_o = tc::idesc_bf16(128, H128, 0, 1);
      const uint32_t t_s = tmem + t * 128, t_o = tmem + 256 + t * 128;
      const uint64_t dQ = desc_base_k(tc::smem_u32(smem + S::Q + t * T128_BYTES)), dK0 = desc_base_k(tc::smem_u32(smem + S::K)),
                     dV0 = desc_base_mn(tc::smem_u32(smem + S::V));
      int g = 0, gt = 0, cq = 0;
      for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
        const Item it = item_of(w);
        const int n = blocks_of(it, t);
        auto scores = [&](int j) {
          const int sl = (g + j) & 1;
          wait(&bar_k[sl], ((g + j) >> 1) & 1, 53);
          tc::tc_fence_after();
          const uint64_t dK = dK0 + sl * T128_UNITS;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_s, dQ + off_k(ks, TILE_BYTES), dK + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(&bar_s[t]);
          tc::mma_commit(&bar_kf[sl]);
          if (j == n - 1) tc::mma_commit(&bar_qf[t]);
        };
        if (n > 0) {
          wait(&bar_q[t], cq & 1, 54);
          cq++;
          scores(0);
        }
        for (int j = 0; j < n; j++, gt++) {
          const int sl = (g + j) & 1;
          const uint64_t dV = dV0 + sl * T128_UNITS;
          wait(&bar_v[sl], ((g + j) >> 1) & 1, 55);
          wait(&bar_pa[t], gt & 1, 56);
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 4; ks++) tc::mma_bf16_ts(t_o, t_s + ks * 8, dV + off_mn(ks), idesc_o, (j > 0 || ks > 0));
          wait(&bar_pb[t], gt & 1, 57);
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 4; ks < 8; ks++) tc::mma_bf16_ts(t_o, t_s + ks * 8, dV + off_mn(ks), idesc_o, 1);
          tc::mma_commit(&bar_o[t]);
          tc::mma_commit(&bar_vf[sl]);
          if (j + 1 < n) scores(j + 1);      // behind P V, which reads P out of these columns
        }
        for (int j = n; j < it.nkb; j++) {      // blocks only the other tile sees: released once they have landed
          const int sl = (g + j) & 1, ph = ((g + j) >> 1) & 1;
          wait(&bar_k[sl], ph, 53);
          tc::mbar_arrive(&bar_kf[sl]);
          wait(&bar_v[sl], ph, 55);
          tc::mbar_arrive(&bar_vf[sl]);
        }
        g += it.nkb;
      }
    }
  } else {
    const int t = warp >> 2, lg = warp & 3, row = lg * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
    const uint32_t t_s = tmem + t * 128 + lane_addr, t_o = tmem + 256 + t * 128 + lane_addr;
    const float sl2 = a.scale * LOG2E;
    const uint64_t sl2x2 = pk2(sl2, sl2);
    uint8_t* stage = smem + S::OST + warp * 4096;
    int gt = 0;
    for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
      const Item it = item_of(w);
      const int n = blocks_of(it, t);
      if (n == 0) continue;
      const int qt = 2 * it.pair + t, qrow = qt * 128 + row;
      float m = 0.f, l = 0.f;
      for (int j = 0; j < n; j++, gt++) {
        wait(&bar_s[t], gt & 1, 58);
        __syncwarp();
        tc::tc_fence_after();
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; c++) tc::tmem_ld32(t_s + c * 32, r[c]);
        tc::tmem_ld_wait();
        if (j == n - 1) {      // the diagonal block
#pragma unroll
          for (int i = 0; i < 128; i++)
            if (i > row) r[i >> 5][i & 31] = 0xff800000u;
        }
        float mx = -INFINITY;
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
          for (int i = 0; i < 32; i += 2) mx = max3(mx, __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
        const float z = mx * sl2;
        if (j == 0) {
          m = z == -INFINITY ? 0.f : z;
        } else if (__any_sync(0xffffffffu, z > m + 8.f)) {
          const float mn = fmaxf(m, z), alpha = ex2_approx(m - mn);
          m = mn;
          l *= alpha;
          wait(&bar_o[t], (gt - 1) & 1, 59);
          __syncwarp();
          tc::tc_fence_after();
#pragma unroll
          for (int c = 0; c < 8; c++) {
            uint32_t o[16];
            tc::tmem_ld16(t_o + c * 16, o);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tc::tmem_st16(t_o + c * 16, o);
          }
          tc::tmem_st_wait();
        }
        const uint64_t nm2 = pk2(-m, -m);
        uint64_t rs2 = pk2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 4; c++) {
          uint32_t pw[16];
#pragma unroll
          for (int i = 0; i < 16; i++) {
            float z0, z1;
            upk2(fma2(pk2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), sl2x2, nm2), z0, z1);
            const float p0 = ex2_approx(z0), p1 = ex2_approx(z1);
            rs2 = add2(rs2, pk2(p0, p1));
            pw[i] = pack_bf16(p0, p1);
          }
          tc::tmem_st16(t_s + c * 16, pw);
          if (c == 1 || c == 3) {
            tc::tmem_st_wait();
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(c == 1 ? &bar_pa[t] : &bar_pb[t]);
          }
        }
        float lo, hi;
        upk2(rs2, lo, hi);
        l += lo + hi;
      }
      // ---- epilogue: O / l as bf16
      wait(&bar_o[t], (gt - 1) & 1, 60);
      __syncwarp();
      tc::tc_fence_after();
      const float inv = 1.f / l;
      const bool live = qrow < a.T && !*s_abort;
      bf16* dst = a.out + ((size_t)(it.b * a.T + (live ? qrow : 0))) * C + it.h * H128;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        if (a.out_tma) {
          if (lane == 0) tc::tma_wait_group_read<0>();      // the previous store has read the staging tile
          __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t o[32];
          tc::tmem_ld32(t_o + half * 64 + c * 32, o);
          tc::tmem_ld_wait();
#pragma unroll
          for (int v = 0; v < 4; v++) {
            uint4 x;
            x.x = pack_bf16(__uint_as_float(o[v * 8]) * inv, __uint_as_float(o[v * 8 + 1]) * inv);
            x.y = pack_bf16(__uint_as_float(o[v * 8 + 2]) * inv, __uint_as_float(o[v * 8 + 3]) * inv);
            x.z = pack_bf16(__uint_as_float(o[v * 8 + 4]) * inv, __uint_as_float(o[v * 8 + 5]) * inv);
            x.w = pack_bf16(__uint_as_float(o[v * 8 + 6]) * inv, __uint_as_float(o[v * 8 + 7]) * inv);
            if (a.out_tma) *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + v) ^ (lane & 7)) << 4)) = x;
            else if (live) *reinterpret_cast<uint4*>(dst + half * 64 + c * 32 + v * 8) = x;
          }
        }
        if (a.out_tma) {
          tc::fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (!*s_abort) tc::tma_store_2d(&tm_out, stage, it.h * H128 + half * 64, it.b * a.T + qt * 128 + lg * 32);
            tc::tma_commit_group();
          }
        }
      }
      tc::tc_fence_before();
      if (live) a.lse[((size_t)it.b * a.H + it.h) * a.T + qrow] = (m + log2f(l)) * LN2;
    }
    if (a.out_tma && lane == 0) tc::tma_wait_group<0>();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) tc::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------ backward
// dK / dV of a 128-key tile, streaming query blocks.  TMEM: S^T, dP^T, dV, dK.  The tensor core's sequence is
//   dV(i)  S^T(i+1)  dK(i)  dP^T(i+1)  dV(i+1) ...
// so the exponentials of block i+1 run under dK(i) and dP^T(i+1), and dS(i+1) under dV(i+1) and S^T(i+2).  256 element-wise threads: a
// thread has one key and 64 of the block's 128 queries; its P^T / dS^T go over its own score columns.
struct BwdKV128Smem {
  static constexpr int K = 0;
  static constexpr int V = K + T128_BYTES;
  static constexpr int Q = V + T128_BYTES;               // 2 slots
  static constexpr int DO = Q + 2 * T128_BYTES;          // 2 slots
  static constexpr int STAT = DO + 2 * T128_BYTES;       // 8 warps x 2 buffers x (lse * log2 e [64], delta [64])
  static constexpr int BAR = STAT + 8 * 1024;
  static constexpr int SCHED = BAR + 256;
  static constexpr int TOTAL = SCHED + 256 + 1024;
};
// dQ of a 128-query tile, streaming key blocks.  TMEM: S in two buffers, dP, dQ; dS goes over the S it came from:
//   dP(j+1)  dQ(j)  S(j+2)  dP(j+2) ...
// keeps scores one block ahead, so the element-wise threads never wait for them.
struct BwdQ128Smem {
  static constexpr int Q = 0;
  static constexpr int DO = Q + T128_BYTES;
  static constexpr int K = DO + T128_BYTES;              // 3 slots (S runs ahead of dQ, which reads K last)
  static constexpr int V = K + 3 * T128_BYTES;           // 2 slots
  static constexpr int BAR = V + 2 * T128_BYTES;
  static constexpr int SCHED = BAR + 256;
  static constexpr int TOTAL = SCHED + 256 + 1024;
};
constexpr int BWD128_THREADS = 10 * 32;      // 8 element-wise warps (lane group w & 3, column half w >> 2), MMA warp, loader
// A-operand columns of k-step ks of a bf16 tile whose two 64-column halves sit over their own fp32 columns
__device__ __forceinline__ uint32_t half_col(int ks) { return (uint32_t)((ks >> 2) * 64 + (ks & 3) * 8); }

__global__ void __launch_bounds__(BWD128_THREADS, 1) attn_bwd_kv128_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do,
                                                                      const AttnArgs a) {
  mlb_pdl_sync();
  using S = BwdKV128Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_kv = bars, *bar_kvf = bars + 1, *bar_q = bars + 2 /*[2]*/, *bar_qf = bars + 4 /*[2]*/, *bar_do = bars + 6 /*[2]*/, *bar_dof = bars + 8 /*[2]*/,
           *bar_s = bars + 10, *bar_dp = bars + 11, *bar_p = bars + 12, *bar_ds = bars + 13, *bar_done = bars + 14;
  uint32_t* tmem_slot = (uint32_t*)(bars + 15);
  volatile int* s_abort = (volatile int*)(bars + 16);
  if (attn_given_up()) return;
  const int nq = (a.T + 127) / 128, BH = a.B * a.H, C = a.H * H128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* srow = a.sched ? a.sched + (size_t)blockIdx.x * a.sched_stride : nullptr;
  int* s_sched = (int*)(smem + S::SCHED);
  if (srow && tid < 64) s_sched[tid] = tid < a.sched_stride ? __ldg(srow + tid) : -1;
  const ItemList items{srow, s_sched, (int)blockIdx.x, (int)gridDim.x, nq * BH};
  if (tid == 0) {
    for (int i = 0; i < 15; i++) tc::mbar_init(&bars[i], (i == 12 || i == 13) ? 8 : 1);
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
    tc::tma_prefetch_desc(&tm_do);
  }
  if (warp == 8) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t t_s = tmem, t_dp = tmem + 128, t_dv = tmem + 256, t_dk = tmem + 384;
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) {
    if (tc::mbar_try(bar, phase) || *s_abort) return;
    if (!tc::mbar_wait(bar, phase, where)) *s_abort = 1;
  };
  // item w = key tile (heaviest, the first, first) of (sample, head)
  if (warp == 9) {
    if (lane == 0) {
      int g = 0;
      for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
        const int kt = w / BH, bh = w % BH, b = bh / a.H, xh = (bh % a.H) * H128;
        if (li > 0) wait(bar_kvf, (li - 1) & 1, 61);
        tc::mbar_expect_tx(bar_kv, 2 * T128_BYTES);
        split_load<2>(smem + S::K, &tm, bar_kv, C + xh, kt * 128, b, 2);
        split_load<2>(smem + S::V, &tm, bar_kv, 2 * C + xh, kt * 128, b, 2);
        for (int i = kt; i < nq; i++, g++) {
          const int sl = g & 1, ph = ((g >> 1) + 1) & 1;
          if (g >= 2) wait(&bar_qf[sl], ph, 62);
          tc::mbar_expect_tx(&bar_q[sl], T128_BYTES);
          split_load<2>(smem + S::Q + sl * T128_BYTES, &tm, &bar_q[sl], xh, i * 128, b, 2);
          if (g >= 2) wait(&bar_dof[sl], ph, 63);
          tc::mbar_expect_tx(&bar_do[sl], T128_BYTES);
          split_load<2>(smem + S::DO + sl * T128_BYTES, &tm_do, &bar_do[sl], xh, i * 128, b, 2);
        }
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = tc::idesc_bf16(128, 128, 0, 0), idesc_g = tc::idesc_bf16(128, H128, 0, 1);
      const uint64_t dK = desc_base_k(tc::smem_u32(smem + S::K)), dV = desc_base_k(tc::smem_u32(smem + S::V));
      const uint64_t dQ0 = desc_base_k(tc::smem_u32(smem + S::Q)), dO0 = desc_base_k(tc::smem_u32(smem + S::DO));      // as B of the scores
      const uint64_t gQ0 = desc_base_mn(tc::smem_u32(smem + S::Q)), gO0 = desc_base_mn(tc::smem_u32(smem + S::DO));    // as B of the gradients
      int g = 0;
      for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
        const int n = nq - w / BH;
        auto scores = [&](int gb) {
          wait(&bar_q[gb & 1], (gb >> 1) & 1, 64);
          tc::tc_fence_after();
          const uint64_t dQ = dQ0 + (gb & 1) * T128_UNITS;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_s, dK + off_k(ks, TILE_BYTES), dQ + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(bar_s);
        };
        auto dprobs = [&](int gb, bool last) {
          wait(&bar_do[gb & 1], (gb >> 1) & 1, 65);
          tc::tc_fence_after();
          const uint64_t dO = dO0 + (gb & 1) * T128_UNITS;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_dp, dV + off_k(ks, TILE_BYTES), dO + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(bar_dp);
          if (last) tc::mma_commit(bar_kvf);
        };
        wait(bar_kv, li & 1, 66);
        scores(g);
        dprobs(g, n == 1);
        for (int i = 0; i < n; i++, g++) {
          const int sl = g & 1;
          const uint64_t gQ = gQ0 + sl * T128_UNITS, gO = gO0 + sl * T128_UNITS;
          wait(bar_p, g & 1, 67);      // (of an item's first block: also the accumulators of the previous item have been read out)
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ts(t_dv, t_s + half_col(ks), gO + off_mn(ks), idesc_g, (i > 0 || ks > 0));
          tc::mma_commit(&bar_dof[sl]);
          if (i + 1 < n) scores(g + 1);
          wait(bar_ds, g & 1, 68);
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ts(t_dk, t_dp + half_col(ks), gQ + off_mn(ks), idesc_g, (i > 0 || ks > 0));
          tc::mma_commit(&bar_qf[sl]);
          if (i + 1 < n) dprobs(g + 1, i + 2 == n);
          else tc::mma_commit(bar_done);
        }
      }
    }
  } else {
    const int lg = warp & 3, hf = warp >> 2, row = lg * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
    const uint32_t ts = t_s + hf * 64 + lane_addr, tdp = t_dp + hf * 64 + lane_addr;
    const float sl2 = a.scale * LOG2E;
    float* stat = (float*)(smem + S::STAT + warp * 1024);
    int g = 0;
    for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
      const int kt = w / BH, bh = w % BH, b = bh / a.H, h = bh % a.H;
      const size_t si = ((size_t)b * a.H + h) * a.T;
      const int krow = kt * 128 + row;
      // statistics of the warp's 64 queries; a query past the end has lse = +inf: p = 0
      float sv[4];
      auto fetch = [&](int i) {
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const int q = i * 128 + hf * 64 + x * 32 + lane;
          sv[x] = q < a.T ? a.lse[si + q] * LOG2E : INFINITY;
          sv[2 + x] = q < a.T ? a.delta[si + q] : 0.f;
        }
      };
      auto publish = [&](int gb) {
#pragma unroll
        for (int x = 0; x < 4; x++) stat[(gb & 1) * 128 + x * 32 + lane] = sv[x];
        __syncwarp();
      };
      fetch(kt);
      publish(g);
      for (int i = kt; i < nq; i++, g++) {
        const float* st = stat + (g & 1) * 128;
        if (i + 1 < nq) fetch(i + 1);
        wait(bar_s, g & 1, 69);
        __syncwarp();
        tc::tc_fence_after();
        float p[64];
        {
          uint32_t r[2][32];
          tc::tmem_ld32(ts, r[0]);
          tc::tmem_ld32(ts + 32, r[1]);
          tc::tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 64; e += 4) {
            const float4 L = *reinterpret_cast<const float4*>(st + e);
            p[e] = ex2_approx(fmaf(__uint_as_float(r[e >> 5][e & 31]), sl2, -L.x));
            p[e + 1] = ex2_approx(fmaf(__uint_as_float(r[e >> 5][(e & 31) + 1]), sl2, -L.y));
            p[e + 2] = ex2_approx(fmaf(__uint_as_float(r[e >> 5][(e & 31) + 2]), sl2, -L.z));
            p[e + 3] = ex2_approx(fmaf(__uint_as_float(r[e >> 5][(e & 31) + 3]), sl2, -L.w));
          }
        }
        if (i == kt) {      // the diagonal block: query before key
#pragma unroll
          for (int e = 0; e < 64; e++)
            if (hf * 64 + e < row) p[e] = 0.f;
        }
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t pw[16];
#pragma unroll
          for (int x = 0; x < 16; x++) pw[x] = pack_bf16(p[c * 32 + 2 * x], p[c * 32 + 2 * x + 1]);
          tc::tmem_st16(ts + c * 16, pw);
        }
        tc::tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_p);
        wait(bar_dp, g & 1, 70);
        __syncwarp();
        tc::tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t d[32], dw[16];
          tc::tmem_ld32(tdp + c * 32, d);
          tc::tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            const int e = c * 32 + x;
            const float4 D = *reinterpret_cast<const float4*>(st + 64 + e);
            dw[x / 2] = pack_bf16(p[e] * (__uint_as_float(d[x]) - D.x), p[e + 1] * (__uint_as_float(d[x + 1]) - D.y));
            dw[x / 2 + 1] = pack_bf16(p[e + 2] * (__uint_as_float(d[x + 2]) - D.z), p[e + 3] * (__uint_as_float(d[x + 3]) - D.w));
          }
          tc::tmem_st16(tdp + c * 16, dw);
        }
        tc::tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_ds);
        if (i + 1 < nq) publish(g + 1);
      }
      // ---- epilogue: warps 0-3 store dK (softmax scale and RoPE's backward rotation applied), warps 4-7 dV
      wait(bar_done, li & 1, 71);
      __syncwarp();
      tc::tc_fence_after();
      const bool live = krow < a.T && !*s_abort;
      bf16* dst = a.out + ((size_t)(b * a.T + (live ? krow : 0))) * 3 * C + (hf == 0 ? C : 2 * C) + h * H128;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32)
        store_pairs_rope<H128>(dst, (hf == 0 ? t_dk : t_dv) + lane_addr, c0, live, hf == 0 ? a.cosT : nullptr, hf == 0 ? a.sinT : nullptr, krow,
                               hf == 0 ? a.scale : 1.f);
      tc::tc_fence_before();
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) tc::tmem_dealloc(tmem, 512);
}

__global__ void __launch_bounds__(BWD128_THREADS, 1) attn_bwd_q128_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do,
                                                                     const AttnArgs a) {
  mlb_pdl_sync();
  using S = BwdQ128Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_x = bars, *bar_xf = bars + 1, *bar_k = bars + 2 /*[3]*/, *bar_kf = bars + 5 /*[3]*/, *bar_v = bars + 8 /*[2]*/, *bar_vf = bars + 10 /*[2]*/,
           *bar_s = bars + 12 /*[2]*/, *bar_dp = bars + 14, *bar_done = bars + 15, *bar_ds = bars + 16;
  uint32_t* tmem_slot = (uint32_t*)(bars + 17);
  volatile int* s_abort = (volatile int*)(bars + 18);
  if (attn_given_up()) return;
  const int nq = (a.T + 127) / 128, BH = a.B * a.H, C = a.H * H128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* srow = a.sched ? a.sched + (size_t)blockIdx.x * a.sched_stride : nullptr;
  int* s_sched = (int*)(smem + S::SCHED);
  if (srow && tid < 64) s_sched[tid] = tid < a.sched_stride ? __ldg(srow + tid) : -1;
  const ItemList items{srow, s_sched, (int)blockIdx.x, (int)gridDim.x, nq * BH};
  if (tid == 0) {
    for (int i = 0; i < 17; i++) tc::mbar_init(&bars[i], i == 16 ? 8 : 1);
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
    tc::tma_prefetch_desc(&tm_do);
  }
  if (warp == 8) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t t_dp = tmem + 256, t_dq = tmem + 384;      // S buffers at +0 and +128
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) {
    if (tc::mbar_try(bar, phase) || *s_abort) return;
    if (!tc::mbar_wait(bar, phase, where)) *s_abort = 1;
  };
  // item w = query tile (heaviest, the last, first) of (sample, head), with qt + 1 key blocks
  if (warp == 9) {
    if (lane == 0) {
      int g = 0;
      for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
        const int qt = nq - 1 - w / BH, bh = w % BH, b = bh / a.H, xh = (bh % a.H) * H128;
        if (li > 0) wait(bar_xf, (li - 1) & 1, 72);
        tc::mbar_expect_tx(bar_x, 2 * T128_BYTES);
        split_load<2>(smem + S::Q, &tm, bar_x, xh, qt * 128, b, 2);
        split_load<2>(smem + S::DO, &tm_do, bar_x, xh, qt * 128, b, 2);
        for (int j = 0; j <= qt; j++, g++) {
          const int ks = g % 3, vs = g & 1;
          if (g >= 3) wait(&bar_kf[ks], (g / 3 + 1) & 1, 73);
          tc::mbar_expect_tx(&bar_k[ks], T128_BYTES);
          split_load<2>(smem + S::K + ks * T128_BYTES, &tm, &bar_k[ks], C + xh, j * 128, b, 2);
          if (g >= 2) wait(&bar_vf[vs], ((g >> 1) + 1) & 1, 74);
          tc::mbar_expect_tx(&bar_v[vs], T128_BYTES);
          split_load<2>(smem + S::V + vs * T128_BYTES, &tm, &bar_v[vs], 2 * C + xh, j * 128, b, 2);
        }
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = tc::idesc_bf16(128, 128, 0, 0), idesc_g = tc::idesc_bf16(128, H128, 0, 1);
      const uint64_t dQ = desc_base_k(tc::smem_u32(smem + S::Q)), dO = desc_base_k(tc::smem_u32(smem + S::DO));
      const uint64_t dK0 = desc_base_k(tc::smem_u32(smem + S::K)), dV0 = desc_base_k(tc::smem_u32(smem + S::V));
      const uint64_t gK0 = desc_base_mn(tc::smem_u32(smem + S::K));      // as B of dQ
      int g = 0, kr = 0;      // kr = g % 3
      for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
        const int n = nq - w / BH;
        auto scores = [&](int gb) {
          const int sl = gb % 3;
          wait(&bar_k[sl], (gb / 3) & 1, 75);
          tc::tc_fence_after();
          const uint64_t dK = dK0 + sl * T128_UNITS;
          const uint32_t t_s = tmem + (gb & 1) * 128;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_s, dQ + off_k(ks, TILE_BYTES), dK + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(&bar_s[gb & 1]);
        };
        auto dprobs = [&](int gb, bool last) {
          wait(&bar_v[gb & 1], (gb >> 1) & 1, 76);
          tc::tc_fence_after();
          const uint64_t dV = dV0 + (gb & 1) * T128_UNITS;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_dp, dO + off_k(ks, TILE_BYTES), dV + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(bar_dp);
          tc::mma_commit(&bar_vf[gb & 1]);
          if (last) tc::mma_commit(bar_xf);      // (the last scores were issued before)
        };
        wait(bar_x, li & 1, 77);
        scores(g);
        if (n > 1) scores(g + 1);
        dprobs(g, n == 1);
        for (int j = 0; j < n; j++, g++) {
          wait(bar_ds, g & 1, 78);      // dP(j) read, dS(j) stored (of an item's first block: the previous dQ read out)
          tc::tc_fence_after();
          if (j + 1 < n) dprobs(g + 1, j + 2 == n);
          const uint64_t gK = gK0 + kr * T128_UNITS;
          const uint32_t t_ds = tmem + (g & 1) * 128;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ts(t_dq, t_ds + half_col(ks), gK + off_mn(ks), idesc_g, (j > 0 || ks > 0));
          tc::mma_commit(&bar_kf[kr]);
          kr = kr == 2 ? 0 : kr + 1;
          if (j + 2 < n) scores(g + 2);      // over dS(j), behind dQ(j)
          if (j + 1 == n) tc::mma_commit(bar_done);
        }
      }
    }
  } else {
    const int lg = warp & 3, hf = warp >> 2, row = lg * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
    const float sl2 = a.scale * LOG2E;
    int g = 0;
    for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
      const int qt = nq - 1 - w / BH, bh = w % BH, b = bh / a.H, h = bh % a.H;
      const int qrow = qt * 128 + row;
      const size_t si = ((size_t)b * a.H + h) * a.T + qrow;
      const float nl = qrow < a.T ? -a.lse[si] * LOG2E : -INFINITY;
      const float delta = qrow < a.T ? a.delta[si] : 0.f;
      for (int j = 0; j <= qt; j++, g++) {
        const uint32_t ts = tmem + (g & 1) * 128 + hf * 64 + lane_addr, tdp = t_dp + hf * 64 + lane_addr;
        wait(&bar_s[g & 1], (g >> 1) & 1, 79);
        __syncwarp();
        tc::tc_fence_after();
        float p[64];
        {
          uint32_t r[2][32];
          tc::tmem_ld32(ts, r[0]);
          tc::tmem_ld32(ts + 32, r[1]);
          tc::tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 64; e++) p[e] = ex2_approx(fmaf(__uint_as_float(r[e >> 5][e & 31]), sl2, nl));
        }
        if (j == qt) {      // the diagonal block
#pragma unroll
          for (int e = 0; e < 64; e++)
            if (hf * 64 + e > row) p[e] = 0.f;
        }
        wait(bar_dp, g & 1, 80);
        __syncwarp();
        tc::tc_fence_after();
        uint32_t d[2][32];
        tc::tmem_ld32(tdp, d[0]);
        tc::tmem_ld32(tdp + 32, d[1]);
        tc::tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t dw[16];
#pragma unroll
          for (int x = 0; x < 16; x++) {
            const int e = c * 32 + 2 * x;
            dw[x] = pack_bf16(p[e] * (__uint_as_float(d[c][2 * x]) - delta), p[e + 1] * (__uint_as_float(d[c][2 * x + 1]) - delta));
          }
          tc::tmem_st16(ts + c * 16, dw);
        }
        tc::tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_ds);
      }
      wait(bar_done, li & 1, 81);
      __syncwarp();
      tc::tc_fence_after();
      const bool live = qrow < a.T && !*s_abort;
      bf16* dst = a.out + ((size_t)(b * a.T + (live ? qrow : 0))) * 3 * C + h * H128;
      store_pairs_rope<H128>(dst, t_dq + lane_addr, hf * 32, live, a.cosT, a.sinT, qrow, a.scale);
      tc::tc_fence_before();
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) tc::tmem_dealloc(tmem, 512);
}
