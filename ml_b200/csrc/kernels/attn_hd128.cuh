// Causal attention at head size 128, forward and backward.  Included by attn.cu behind attn_split.cuh (shares their helpers).
//
// At this head size the four products of a forward step over 256 queries x 128 keys take the tensor core as long as their
// exponentials take the special-function units (2048 cycles each), and in backward the products lead (2048 / 1536 cycles against
// 1024), so the kernels are built around never letting one wait for the other; tensor memory is the constraint (a 128 x 128
// fp32 tile is 128 of its 512 columns).  P and dS are written as bf16 pairs over the score columns they came from and are read
// from there as the A operand of the next product: no columns of their own, and no shared memory (but for the P^T of dK / dV).  MMAs are promised to run in
// the order of their issue only where accumulator and shape are the same, so a product that overwrites such columns is issued when
// the one that reads them has completed (its commit is waited for).
// All three kernels are persistent, one CTA per SM over a balanced table of items (attn_schedule); every wait is bounded and
// sticky: after one expiry the CTA's later waits return at once, its loader and MMA threads stop, and the element-wise warps walk on to
// the common end.  Loader and MMA threads come there when what they have issued is complete (attn_settle), whatever happened.
// (At the end itself, for all warps, that costs the dK / dV kernel registers: 353 us instead of 345.)
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
// is a chain; the two tiles run it out of phase, one on the tensor core while the other takes exponentials: they take turns.  Left
// alone they fall into step, and a step of both tiles takes 5400 cycles instead of 3700 (8 x 2048 tokens, 16 heads: 192 -> 161 us with the
// older maximum of the next lines).  P V starts when the first half of P is there.  160 registers leave a sub-partition with three of
// these warps room for one 32-register warp of a communication kernel.
// m is the maximum of all blocks so far, so that a row's largest probability is 1 and costs no rounding; O (in place) and l are rescaled
// whenever a row of the warp has a new one.  Kept from an earlier block until outgrown by 2^8 it takes 159 us instead of 180 (764 TFLOP/s
// over the causal half), but the largest probability is rounded like the others: 2.07e-3 off the 64-bit result instead of 2.04e-3 over
// 2048 tokens, and with scores of twice that spread 2.11e-3 instead of 1.86e-3.
__global__ void __maxnreg__(160) attn_fwd128_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_out,
                                                                   const AttnArgs a) {
  mlb_pdl_sync();
  using S = Fwd128Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_q = bars, *bar_qf = bars + 2, *bar_k = bars + 4, *bar_kf = bars + 6, *bar_v = bars + 8, *bar_vf = bars + 10, *bar_s = bars + 12,
           *bar_pa = bars + 14, *bar_pb = bars + 16, *bar_o = bars + 18;      // [2] each: per tile (q, s, p, o) or slot (k, v)
  volatile int* s_turn = (volatile int*)(bars + 20);      // [2][4]: blocks whose exponentials tile t's warp on sub-partition lg has taken
  uint64_t* bar_end = bars + 24;      // [2]: the MMA threads' last commits
  uint32_t* tmem_slot = (uint32_t*)(bars + 26);
  volatile int* s_abort = (volatile int*)(bars + 27);
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
      tc::mbar_init(&bar_pb[i], 4); tc::mbar_init(&bar_o[i], 1); tc::mbar_init(&bar_end[i], 1);
    }
    for (int i = 0; i < 8; i++) s_turn[i] = 0;
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
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) { return tc::mbar_wait_sticky(bar, phase, where, s_abort); };
  // item w = pair (heaviest first) of (sample, head); tile t of it has n(t) key blocks (none when the pair has no second tile)
  struct Item { int pair, b, h, nkb; };
  auto item_of = [&](int w) {
    const int bh = w % BH, pair = npair - 1 - w / BH;
    return Item{pair, bh / a.H, bh % a.H, min(2 * pair + 2, nq)};
  };
  auto blocks_of = [&](const Item& it, int t) { return 2 * it.pair + t < nq ? 2 * it.pair + t + 1 : 0; };

  if (warp == 9) {
    if (lane == 0) {
      int g = 0, cq[2] = {0, 0}, odd = 0;      // odd: a K without its V
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const Item it = item_of(w);
        auto load_q = [&](int t) {
          if (blocks_of(it, t) == 0 || !ok) return;
          if (cq[t] > 0 && !wait(&bar_qf[t], (cq[t] - 1) & 1, 50)) { ok = false; return; }
          cq[t]++;
          tc::mbar_expect_tx(&bar_q[t], T128_BYTES);
          split_load<2>(smem + S::Q + t * T128_BYTES, &tm, &bar_q[t], it.h * H128, (2 * it.pair + t) * 128, it.b, 2);
        };
        for (int j = 0; j < it.nkb; j++, g++) {
          const int sl = g & 1, ph = ((g >> 1) + 1) & 1;
          if (!ok || (g >= 2 && !wait(&bar_kf[sl], ph, 51))) { ok = false; break; }
          tc::mbar_expect_tx(&bar_k[sl], T128_BYTES);
          split_load<2>(smem + S::K + sl * T128_BYTES, &tm, &bar_k[sl], C + it.h * H128, j * 128, it.b, 2);
          if (j == 0) { load_q(0); load_q(1); }
          if (!ok || (g >= 2 && !wait(&bar_vf[sl], ph, 52))) { ok = false; odd = 1; break; }
          tc::mbar_expect_tx(&bar_v[sl], T128_BYTES);
          split_load<2>(smem + S::V + sl * T128_BYTES, &tm, &bar_v[sl], 2 * C + it.h * H128, j * 128, it.b, 2);
        }
      }
      for (int i = 0; i < 2; i++) {
        attn_settle(&bar_q[i], cq[i]);
        attn_settle(&bar_k[i], (g + odd + 1 - i) / 2);
        attn_settle(&bar_v[i], (g + 1 - i) / 2);
      }
    }
  } else if (warp == 8 || warp == 10) {
    if (tc::elect_one()) {
      const int t = warp == 8 ? 0 : 1;
      constexpr uint32_t idesc_s = tc::idesc_bf16(128, 128, 0, 0), idesc_o = tc::idesc_bf16(128, H128, 0, 1);
      const uint32_t t_s = tmem + t * 128, t_o = tmem + 256 + t * 128;
      const uint64_t dQ = desc_base_k(tc::smem_u32(smem + S::Q + t * T128_BYTES)), dK0 = desc_base_k(tc::smem_u32(smem + S::K)),
                     dV0 = desc_base_mn(tc::smem_u32(smem + S::V));
      int g = 0, gt = 0, cq = 0;
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const Item it = item_of(w);
        const int n = blocks_of(it, t);
        auto scores = [&](int j, int pv) {      // over the columns that the tile's latest P V (number pv - 1) reads P from
          const int sl = (g + j) & 1;
          if (!ok || !wait(&bar_k[sl], ((g + j) >> 1) & 1, 53) || (pv > 0 && !wait(&bar_o[t], (pv - 1) & 1, 82))) { ok = false; return; }
          tc::tc_fence_after();
          const uint64_t dK = dK0 + sl * T128_UNITS;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_s, dQ + off_k(ks, TILE_BYTES), dK + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(&bar_s[t]);
          tc::mma_commit(&bar_kf[sl]);
          if (j == n - 1) tc::mma_commit(&bar_qf[t]);
        };
        if (n > 0) {
          ok = wait(&bar_q[t], cq & 1, 54);
          cq++;
          scores(0, gt);
        }
        for (int j = 0; j < n; j++, gt++) {
          const int sl = (g + j) & 1;
          const uint64_t dV = dV0 + sl * T128_UNITS;
          if (!ok || !wait(&bar_v[sl], ((g + j) >> 1) & 1, 55) || !wait(&bar_pa[t], gt & 1, 56)) { ok = false; break; }
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 4; ks++) tc::mma_bf16_ts(t_o, t_s + ks * 8, dV + off_mn(ks), idesc_o, (j > 0 || ks > 0));
          if (!wait(&bar_pb[t], gt & 1, 57)) { ok = false; break; }
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 4; ks < 8; ks++) tc::mma_bf16_ts(t_o, t_s + ks * 8, dV + off_mn(ks), idesc_o, 1);
          tc::mma_commit(&bar_o[t]);
          tc::mma_commit(&bar_vf[sl]);
          if (j + 1 < n) scores(j + 1, gt + 1);
        }
        for (int j = n; ok && j < it.nkb; j++) {      // blocks only the other tile sees: released once they have landed
          const int sl = (g + j) & 1, ph = ((g + j) >> 1) & 1;
          if (!wait(&bar_k[sl], ph, 53)) { ok = false; break; }
          tc::mbar_arrive(&bar_kf[sl]);
          if (!wait(&bar_v[sl], ph, 55)) { ok = false; break; }
          tc::mbar_arrive(&bar_vf[sl]);
        }
        g += it.nkb;
      }
      tc::mma_commit(&bar_end[t]);
      attn_settle(&bar_end[t], 1);
    }
  } else {
    const int t = warp >> 2, lg = warp & 3, row = lg * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
    const uint32_t t_s = tmem + t * 128 + lane_addr, t_o = tmem + 256 + t * 128 + lane_addr;
    const float sl2 = a.scale * LOG2E;
    const uint64_t sl2x2 = pk2(sl2, sl2);
    uint8_t* stage = smem + S::OST + warp * 4096;
    int gt = 0, other = 0;      // blocks taken by this tile, and by the other tile in earlier items
    for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
      const Item it = item_of(w);
      const int n = blocks_of(it, t), n_other = blocks_of(it, t ^ 1);
      if (n == 0) { other += n_other; continue; }
      const int qt = 2 * it.pair + t, qrow = qt * 128 + row;
      float m = 0.f, l = 0.f;
      for (int j = 0; j < n; j++, gt++) {
        wait(&bar_s[t], gt & 1, 58);
        __syncwarp();
        tc::tc_fence_after();
        uint32_t r[4][32];
        tc::tmem_ld32x4_wait(t_s, r);
        if (j == n - 1) {      // the diagonal block
#pragma unroll
          for (int i = 0; i < 128; i++)
            if (i > row) r[i >> 5][i & 31] = 0xff800000u;
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // four chains: one of 64 dependent maxima takes ~500 cycles
#pragma unroll
        for (int i = 0; i < 32; i += 2)
#pragma unroll
          for (int c = 0; c < 4; c++) m4[c] = max3(m4[c], __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
        const float z = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl2;
        if (j == 0) {
          m = z;
        } else if (__any_sync(0xffffffffu, z > m)) {
          const float mn = fmaxf(m, z), alpha = m == mn ? 1.f : ex2_approx(m - mn);
          m = mn;
          l *= alpha;
          wait(&bar_o[t], (gt - 1) & 1, 59);
          __syncwarp();
          tc::tc_fence_after();
#pragma unroll
          for (int c = 0; c < 8; c++) {
            uint32_t o[16];
            tc::tmem_ld16_wait(t_o + c * 16, o);
#pragma unroll
            for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tc::tmem_st16(t_o + c * 16, o);
          }
          tc::tmem_st_wait();
        }
        // Turns: the two warps of a sub-partition take their exponentials one after the other (tile 0's block j, tile 1's block j, ...).
        // Left alone they fall into step, both on the special-function unit and then both waiting for the tensor core.
        // A counter and not an mbarrier, since one tile may be many blocks behind (a pair without a second tile); only the order hangs on
        // it, so a warp that has polled for long goes on.
        const int turn = other + min(j + t, n_other);      // blocks the other tile's warp is to have taken before
        for (int spin = 0; s_turn[(t ^ 1) * 4 + lg] < turn && spin < (1 << 16) && !*s_abort; spin++) { }
        __syncwarp();
        const float mu = m == -INFINITY ? 0.f : m;      // (nothing finite seen yet: exp2(-inf - 0) = 0)
        const uint64_t nm2 = pk2(-mu, -mu);
        uint64_t rs2 = pk2(0.f, 0.f), rs3 = rs2;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          uint32_t pw[16];
#pragma unroll
          for (int i = 0; i < 16; i++) {
            float z0, z1;
            upk2(fma2(pk2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), sl2x2, nm2), z0, z1);
            const float p0 = ex2_approx(z0), p1 = ex2_approx(z1);
            if (i & 1) rs3 = add2(rs3, pk2(p0, p1));
            else rs2 = add2(rs2, pk2(p0, p1));
            pw[i] = pack_bf16(p0, p1);
          }
          // the first half of P is handed over a quarter late, when its stores have long landed: waiting for them at once stalls the warp
          if (c == 2) {
            tc::tmem_st_wait();
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&bar_pa[t]);
          }
          tc::tmem_st16(t_s + c * 16, pw);
        }
        if (lane == 0) s_turn[t * 4 + lg] = gt + 1;
        tc::tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bar_pb[t]);
        rs2 = add2(rs2, rs3);
        float lo, hi;
        upk2(rs2, lo, hi);
        l += lo + hi;
      }
      other += n_other;
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
          tc::tmem_ld32_wait(t_o + half * 64 + c * 32, o);
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
  if (tid == 0) tc::report_given_up(s_abort);
  if (warp == 8) tc::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------ backward
// dK / dV of a 128-key tile, streaming query blocks.  TMEM: S^T, dP^T, dV, dK.  Two threads issue products, as in the kernels for head
// size 64, so that neither's waits hold up the other's products.  One takes  S^T(i) dP^T(i) S^T(i+1) ...,  the other  dV(i) dK(i) ...
// P^T goes to shared memory, so S^T(i+1) needs no more than that S^T(i) has been read, and the exponentials of block i+1 run under
// dK(i) and dP^T(i+1); over its scores it would make S^T(i+1) wait for dV(i) (tried: the same time).  dS^T stays over dP^T.  Sixteen element-wise
// warps, 32 keys by 32 of the block's 128 queries each, hide each other's TMEM and barrier latencies.  They read scores as fragments (two
// adjacent queries of each eight, for four keys), which reads a query's statistics a quarter as often from the shared memory that the
// products' operands come from.  The statistics are one warp's work (fetched by those who use them, each block waited 800 cycles for
// them).  Shared memory is full to the last 512 bytes: nothing is left to align its base with, which is checked instead.
// K, V and the first Q, dO of the next key tile are asked for as soon as their places are free, and its scores do not wait for this tile's
// epilogue, which sends dV and dK by TMA out of P's place: with loads behind the end of a tile and stores of 32 lines an instruction a change of
// tile was 12600 of 39500 cycles, now 7800.  A block takes 3500 cycles: its products 2048, its shared-memory traffic ~2900 (operands 1800,
// arriving tiles 512, P^T, statistics).  8 x 2048 tokens, 16 heads, both kernels: 655 -> 622 us.
struct BwdKV128Smem {
  static constexpr int K = 0;
  static constexpr int V = K + T128_BYTES;
  static constexpr int Q = V + T128_BYTES;               // 2 slots
  static constexpr int DO = Q + 2 * T128_BYTES;          // 2 slots
  static constexpr int P = DO + 2 * T128_BYTES;          // P^T of a block, two chunks of 64 queries
  static constexpr int STAT = P + T128_BYTES;            // 2 buffers x (lse * log2 e [128], delta [128])
  static constexpr int BAR = STAT + 2 * 1024;
  static constexpr int SCHED = BAR + 256;
  static constexpr int TOTAL = SCHED + 256;
};
// dQ of a 128-query tile, streaming key blocks.  TMEM: S in two buffers, dP, dQ; dS goes over the S it came from:
//   dP(j+1)  S(j+2)  dP(j+2) ...   by one thread,   dQ(j)  dQ(j+1) ...   by another
// keeps scores one block ahead, so the element-wise threads never wait for them.
// The products run through the CTA's query tiles without a break; dQ leaves by TMA out of dO's place, which is loaded for the next tile behind
// that.  A block takes ~2350 cycles, a change of tile 5700 (13000 with loads and stores at its end).
struct BwdQ128Smem {
  static constexpr int Q = 0;
  static constexpr int DO = Q + T128_BYTES;
  static constexpr int K = DO + T128_BYTES;              // 3 slots (S runs ahead of dQ, which reads K last)
  static constexpr int V = K + 3 * T128_BYTES;           // 2 slots
  static constexpr int BAR = V + 2 * T128_BYTES;
  static constexpr int SCHED = BAR + 256;
  static constexpr int TOTAL = SCHED + 256 + 1024;
};
constexpr int BWD128_E_WARPS = 16;      // element-wise warps: lane group w & 3, quarter of the 128 columns w >> 2
constexpr int BWD128_MMA_WARP = BWD128_E_WARPS, BWD128_LOAD_WARP = BWD128_E_WARPS + 1, BWD128_GRAD_WARP = BWD128_E_WARPS + 2,
              BWD128_STAT_WARP = BWD128_E_WARPS + 3;
constexpr int BWD128_THREADS = (BWD128_E_WARPS + 4) * 32;      // (five warps per sub-partition, as with two of the four)
// (split_col(ks): A-operand column of k-step ks of a bf16 tile whose 32-column quarters sit over their own fp32 columns)

// Epilogue of both: of an accumulator a warp takes columns [16 qd, + 16) and [64 + 16 qd, + 16) of its 32 rows, sixteen of RoPE's rotation pairs, as
// fragments, rotates them backward, and puts them as bf16 into a [128 x 128] tile in shared memory that leaves by TMA: no shuffles, and
// stores that touch 16 lines an instruction keep the load / store unit for thousands of cycles.
struct Rope128 { float2 c[2][4], s[2][4]; };      // [16 rows][2 j + v]: columns 8 j + fc, + 1 of row 8 v + fr
__device__ __forceinline__ void rope128(Rope128& r, const float* cosT, const float* sinT, int row0, int c0, int lane, int T) {
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int v = 0; v < 2; v++) {
      const size_t at = (size_t)min(row0 + h * 16 + v * 8 + (lane >> 2), T - 1) * (H128 / 2) + c0 + 2 * (lane & 3);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        r.c[h][2 * j + v] = __ldg(reinterpret_cast<const float2*>(cosT + at + j * 8));
        r.s[h][2 * j + v] = __ldg(reinterpret_cast<const float2*>(sinT + at + j * 8));
      }
    }
}
__device__ __forceinline__ void tile128_out(uint32_t tile, const uint32_t (&a)[2][8], const uint32_t (&b)[2][8], int lg, int c0, int lane, float f, bool rotate,
                                            const Rope128& r) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t wa[4], wb[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      float a0 = __uint_as_float(a[h][2 * m]) * f, a1 = __uint_as_float(b[h][2 * m]) * f;
      float b0 = __uint_as_float(a[h][2 * m + 1]) * f, b1 = __uint_as_float(b[h][2 * m + 1]) * f;
      if (rotate) {      // d0' = d0 c + d1 s, d1' = d1 c - d0 s
        const float2 c = r.c[h][m], s = r.s[h][m];
        const float d0 = a0, e0 = b0;
        a0 = d0 * c.x + a1 * s.x;
        a1 = a1 * c.x - d0 * s.x;
        b0 = e0 * c.y + b1 * s.y;
        b1 = b1 * c.y - e0 * s.y;
      }
      wa[m] = pack_bf16(a0, b0);
      wb[m] = pack_bf16(a1, b1);
    }
    // lane l has the address of row l % 8 of matrix l / 8: rows + 8 (l / 8 % 2), columns + 8 (l / 16)
    const int row = lg * 32 + h * 16 + (lane & 15), col = c0 + (lane >> 4) * 8;
    tc::stmatrix_x4(tile + sw_off(row, col), wa[0], wa[1], wa[2], wa[3]);
    tc::stmatrix_x4(tile + sw_off(row, col + 64), wb[0], wb[1], wb[2], wb[3]);
  }
}
// rows [32 lg, 32 lg + nlive) of such a tile to memory by the four warps that wrote them (thread 0 ... 127), for a part of a tile
__device__ __forceinline__ void tile128_rows(bf16* dst, long pitch, const uint8_t* tile, int lg, int nlive, int thread) {
#pragma unroll 1
  for (int r = thread >> 4; r < nlive; r += 8)
    *reinterpret_cast<uint4*>(dst + r * pitch + (thread & 15) * 8) = *reinterpret_cast<const uint4*>(tile + sw_off(lg * 32 + r, (thread & 15) * 8));
}

__global__ void __launch_bounds__(BWD128_THREADS, 1) attn_bwd_kv128_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do,
                                                                      const __grid_constant__ CUtensorMap tm_out, const AttnArgs a) {
  mlb_pdl_sync();
  using S = BwdKV128Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_k = bars, *bar_kf = bars + 1, *bar_q = bars + 2 /*[2]*/, *bar_qf = bars + 4 /*[2]*/, *bar_do = bars + 6 /*[2]*/, *bar_dof = bars + 8 /*[2]*/,
           *bar_s = bars + 10, *bar_dp = bars + 11, *bar_p = bars + 12, *bar_ds = bars + 13, *bar_done = bars + 14;
  uint64_t* bar_end = bars + 15;      // [2]: the MMA threads' last commits
  uint64_t *bar_sr = bars + 17 /* S^T read out */, *bar_st = bars + 18 /*[2] statistics there */, *bar_stf = bars + 20 /*[2] read */;
  uint64_t *bar_v = bars + 22, *bar_vf = bars + 23;
  uint32_t* tmem_slot = (uint32_t*)(bars + 24);
  volatile int* s_abort = (volatile int*)(bars + 25);
  if (attn_given_up()) return;
  if ((tc::smem_u32(smem) & 1023) != 0) {
    if (threadIdx.x == 0) mlb_set_error(MLB_ERR_BOUNDS, 0xA1);
    return;
  }
  const int nq = (a.T + 127) / 128, BH = a.B * a.H, C = a.H * H128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* srow = a.sched ? a.sched + (size_t)blockIdx.x * a.sched_stride : nullptr;
  int* s_sched = (int*)(smem + S::SCHED);
  if (srow && tid < 64) s_sched[tid] = tid < a.sched_stride ? __ldg(srow + tid) : -1;
  const ItemList items{srow, s_sched, (int)blockIdx.x, (int)gridDim.x, nq * BH};
  if (tid == 0) {
    for (int i = 0; i < 24; i++) tc::mbar_init(&bars[i], (i == 12 || i == 13 || i == 17 || i == 20 || i == 21) ? BWD128_E_WARPS : 1);
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
    tc::tma_prefetch_desc(&tm_do);
    tc::tma_prefetch_desc(&tm_out);
  }
  if (warp == BWD128_MMA_WARP) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t t_s = tmem, t_dp = tmem + 128, t_dv = tmem + 256, t_dk = tmem + 384;
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) { return tc::mbar_wait_sticky(bar, phase, where, s_abort); };
  // item w = key tile (heaviest, the first, first) of (sample, head)
  if (warp == BWD128_LOAD_WARP) {
    if (lane == 0) {
      // The next key tile's K is asked for when the last S^T of this one is there, its V when the last dP^T is: they arrive under the
      // rest of this tile's products and its epilogue
      int g = 0, nk = 0, nv = 0, odd = 0;      // odd: a block that is not counted
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const int kt = w / BH, bh = w % BH, b = bh / a.H, xh = (bh % a.H) * H128;
        for (int i = kt; i < nq; i++, g++) {
          const int sl = g & 1, ph = ((g >> 1) + 1) & 1;
          if (i == kt) {
            if (li > 0 && !wait(bar_kf, (li - 1) & 1, 61)) { ok = false; break; }
            nk++;
            tc::mbar_expect_tx(bar_k, T128_BYTES);
            split_load<2>(smem + S::K, &tm, bar_k, C + xh, kt * 128, b, 2);
          }
          if (g >= 2 && !wait(&bar_qf[sl], ph, 62)) { ok = false; break; }      // (dK comes after dV, and after the dP^T its dS^T was made of)
          tc::mbar_expect_tx(&bar_q[sl], T128_BYTES);
          split_load<2>(smem + S::Q + sl * T128_BYTES, &tm, &bar_q[sl], xh, i * 128, b, 2);
          tc::mbar_expect_tx(&bar_do[sl], T128_BYTES);
          split_load<2>(smem + S::DO + sl * T128_BYTES, &tm_do, &bar_do[sl], xh, i * 128, b, 2);
          if (i == kt) {
            if (li > 0 && !wait(bar_vf, (li - 1) & 1, 88)) { ok = false; odd = 1; break; }
            nv++;
            tc::mbar_expect_tx(bar_v, T128_BYTES);
            split_load<2>(smem + S::V, &tm, bar_v, 2 * C + xh, kt * 128, b, 2);
          }
        }
      }
      attn_settle(bar_k, nk);
      attn_settle(bar_v, nv);
      for (int i = 0; i < 2; i++) {
        attn_settle(&bar_q[i], (g + odd + 1 - i) / 2);
        attn_settle(&bar_do[i], (g + odd + 1 - i) / 2);
      }
    }
  } else if (warp == BWD128_MMA_WARP) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc_s = tc::idesc_bf16(128, 128, 0, 0);
      const uint64_t dK = desc_base_k(tc::smem_u32(smem + S::K)), dV = desc_base_k(tc::smem_u32(smem + S::V));
      const uint64_t dQ0 = desc_base_k(tc::smem_u32(smem + S::Q)), dO0 = desc_base_k(tc::smem_u32(smem + S::DO));
      int g = 0;
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const int n = nq - w / BH;
        ok = wait(bar_k, li & 1, 66);
        for (int i = 0; i < n; i++, g++) {
          const int sl = g & 1, ph = (g >> 1) & 1;
          // over the scores of the block before, once those have been read
          if (!ok || !wait(&bar_q[sl], ph, 64) || (g > 0 && !wait(bar_sr, (g - 1) & 1, 83))) { ok = false; break; }
          tc::tc_fence_after();
          const uint64_t dQ = dQ0 + sl * T128_UNITS, dO = dO0 + sl * T128_UNITS;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_s, dK + off_k(ks, TILE_BYTES), dQ + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(bar_s);
          if (i == n - 1) tc::mma_commit(bar_kf);
          if (i == 0) ok = wait(bar_v, li & 1, 89);
          // over dS^T of the block before, which its dK reads
          if (!ok || !wait(&bar_do[sl], ph, 65) || (g > 0 && !wait(&bar_qf[sl ^ 1], ((g - 1) >> 1) & 1, 84))) { ok = false; break; }
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_dp, dV + off_k(ks, TILE_BYTES), dO + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
          tc::mma_commit(bar_dp);
          if (i == n - 1) tc::mma_commit(bar_vf);
        }
      }
      tc::mma_commit(&bar_end[0]);
      attn_settle(&bar_end[0], 1);
    }
  } else if (warp == BWD128_GRAD_WARP) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc_g = tc::idesc_bf16(128, H128, 0, 1);
      const uint64_t aP = desc_base_k(tc::smem_u32(smem + S::P));
      const uint64_t gQ0 = desc_base_mn(tc::smem_u32(smem + S::Q)), gO0 = desc_base_mn(tc::smem_u32(smem + S::DO));
      int g = 0;
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const int n = nq - w / BH;
        for (int i = 0; i < n; i++, g++) {
          const int sl = g & 1;
          const uint64_t gQ = gQ0 + sl * T128_UNITS, gO = gO0 + sl * T128_UNITS;
          // (of an item's first block bar_p says too that the accumulators of the previous item have been read out; P^T is there without dP^T,
          // so that dO is has to be asked for)
          if (!wait(bar_p, g & 1, 67) || !wait(&bar_do[sl], (g >> 1) & 1, 93)) { ok = false; break; }
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_dv, aP + off_k(ks, TILE_BYTES), gO + off_mn(ks), idesc_g, (i > 0 || ks > 0));
          tc::mma_commit(&bar_dof[sl]);
          if (!wait(bar_ds, g & 1, 68)) { ok = false; break; }
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ts(t_dk, t_dp + split_col(ks), gQ + off_mn(ks), idesc_g, (i > 0 || ks > 0));
          tc::mma_commit(&bar_qf[sl]);
        }
        if (ok) tc::mma_commit(bar_done);
      }
      tc::mma_commit(&bar_end[1]);
      attn_settle(&bar_end[1], 1);
    }
  } else if (warp == BWD128_STAT_WARP) {
    // statistics of a block's queries, two blocks ahead at most; a query past the end has lse = +inf: p = 0
    int g = 0;
    bool ok = true;
    for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
      const size_t e = (size_t)(w % BH) * a.T;
      for (int i = w / BH; i < nq; i++, g++) {
        float nl[4], nd[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const int q = i * 128 + x * 32 + lane;
          nl[x] = q < a.T ? -a.lse[e + q] * LOG2E : -INFINITY;
          nd[x] = q < a.T ? -a.delta[e + q] : 0.f;
        }
        // (one answer for the warp: a lane whose wait has run out must not leave those behind whose wait has not)
        if (g >= 2 && !__all_sync(0xffffffffu, wait(&bar_stf[g & 1], ((g >> 1) + 1) & 1, 63))) { ok = false; break; }
        float* stat = (float*)(smem + S::STAT + (g & 1) * 1024);
#pragma unroll
        for (int x = 0; x < 4; x++) {
          stat[x * 32 + lane] = nl[x];
          stat[128 + x * 32 + lane] = nd[x];
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bar_st[g & 1]);
      }
    }
  } else {
    const int lg = warp & 3, qd = warp >> 2;
    const int fr = lane >> 2, fc = 2 * (lane & 3);      // this thread's row and column in a fragment's 8 x 8 matrices
    const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
    const uint32_t ts = t_s + qd * 32 + lane_addr, tdp = t_dp + qd * 32 + lane_addr;
    const float sl2 = a.scale * LOG2E;
    const uint64_t sl2x2 = pk2(sl2, sl2);
    const uint32_t p_tile = tc::smem_u32(smem + S::P);
    const uint32_t p_at = p_tile + sw_off(lg * 32 + (lane & 15), qd * 32 + (lane >> 4) * 8);      // stmatrix address of rows 0 ... 15, columns 0 ... 15
    const uint32_t p_at16 = p_tile + sw_off(lg * 32 + (lane & 15), qd * 32 + 16 + (lane >> 4) * 8);      // of columns 16 ... 31
    const bool sender = qd == 0 && lane == 0;      // of the 32 rows of four warps
    auto rows_read = [&]() {      // the rows that the sender's last store takes out of P's tile have been read: the four warps may write there again
      if (sender) tc::tma_wait_group_read<0>();
      named_bar_sync(1 + lg, 128);
    };
    int g = 0;
    for (int li = 0, w; (w = items.at(li)) >= 0; li++) {
      const int kt = w / BH, bh = w % BH, b = bh / a.H, h = bh % a.H;
      for (int i = kt; i < nq; i++, g++) {
        const float* st = (const float*)(smem + S::STAT + (g & 1) * 1024) + qd * 32 + fc;
        wait(&bar_st[g & 1], (g >> 1) & 1, 87);
        wait(bar_s, g & 1, 69);
        __syncwarp();
        tc::tc_fence_after();
        float p[2][16];
        uint32_t wp[2][8];
        {
          uint32_t r[2][16];
          tc::tmem_ld_frag_wait(ts, r);
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(bar_sr);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float2 nl = *reinterpret_cast<const float2*>(st + j * 8);
#pragma unroll
            for (int x = 0; x < 2; x++)
#pragma unroll
              for (int v = 0; v < 2; v++) {
                const int e = 4 * j + 2 * v;
                float z0, z1;
                upk2(fma2(pk2(__uint_as_float(r[x][e]), __uint_as_float(r[x][e + 1])), sl2x2, pk2(nl.x, nl.y)), z0, z1);
                p[x][e] = ex2_approx(z0);
                p[x][e + 1] = ex2_approx(z1);
              }
          }
        }
        if (i == kt && qd <= lg) {      // the diagonal block: no query before the key (8 x 8 matrices under, on and over the diagonal)
#pragma unroll
          for (int x = 0; x < 2; x++)
#pragma unroll
            for (int e = 0; e < 16; e++) {
              const int j = e >> 2, row8 = 2 * x + ((e >> 1) & 1);
              if (qd < lg || j < row8 || (j == row8 && fc + (e & 1) < fr)) p[x][e] = 0.f;
            }
        }
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
          for (int m = 0; m < 8; m++) wp[x][m] = pack_bf16(p[x][2 * m], p[x][2 * m + 1]);
        if (g > 0) wait(&bar_dof[(g - 1) & 1], ((g - 1) >> 1) & 1, 86);      // dV of the block before has read its P^T
        __syncwarp();
        if (i == kt && li > 0) rows_read();
#pragma unroll
        for (int x = 0; x < 2; x++) {
          tc::stmatrix_x4(p_at + x * 2048, wp[x][0], wp[x][1], wp[x][2], wp[x][3]);
          tc::stmatrix_x4(p_at16 + x * 2048, wp[x][4], wp[x][5], wp[x][6], wp[x][7]);
        }
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_p);
        wait(bar_dp, g & 1, 70);
        __syncwarp();
        tc::tc_fence_after();
        {
          uint32_t d[2][16];
          tc::tmem_ld_frag_wait(tdp, d);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float2 nd = *reinterpret_cast<const float2*>(st + 128 + j * 8);
#pragma unroll
            for (int x = 0; x < 2; x++)
#pragma unroll
              for (int v = 0; v < 2; v++) {
                const int e = 4 * j + 2 * v;
                float d0, d1;
                upk2(mul2(pk2(p[x][e], p[x][e + 1]), add2(pk2(__uint_as_float(d[x][e]), __uint_as_float(d[x][e + 1])), pk2(nd.x, nd.y))), d0, d1);
                wp[x][2 * j + v] = pack_bf16(d0, d1);
              }
          }
        }
        tc::tmem_st_frag(tdp, wp);
        tc::tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          tc::mbar_arrive(bar_ds);
          tc::mbar_arrive(&bar_stf[g & 1]);
        }
      }
      // ---- epilogue: dV, which is complete before dK, and then dK (softmax scale and RoPE's backward rotation applied), both through P's tile
      Rope128 rp;
      const int row0 = kt * 128 + lg * 32, nlive = a.T - row0;
      auto send = [&](int x) {
        x += h * H128;
        tc::fence_async_smem();
        named_bar_sync(1 + lg, 128);
        if (nlive < 32) {
          if (!*s_abort) tile128_rows(a.out + ((size_t)b * a.T + row0) * 3 * C + x, 3L * C, smem + S::P, lg, nlive, qd * 32 + lane);
        } else if (sender) {
          if (!*s_abort)
            for (int c = 0; c < 2; c++) tc::tma_store_2d(&tm_out, smem + S::P + c * TILE_BYTES + lg * 4096, x + c * 64, b * a.T + row0);
          tc::tma_commit_group();
        }
      };
      uint32_t ra[2][8], rb[2][8];
      wait(&bar_dof[(g - 1) & 1], ((g - 1) >> 1) & 1, 90);
      __syncwarp();
      tc::tc_fence_after();
      tc::tmem_ld_pairs_wait(t_dv + lane_addr + qd * 16, ra, t_dv + lane_addr + 64 + qd * 16, rb);
      tile128_out(p_tile, ra, rb, lg, qd * 16, lane, 1.f, false, rp);
      if (a.cosT) rope128(rp, a.cosT, a.sinT, row0, qd * 16, lane, a.T);      // (sooner there are no registers for them)
      send(2 * C);
      wait(bar_done, li & 1, 71);
      __syncwarp();
      tc::tc_fence_after();
      tc::tmem_ld_pairs_wait(t_dk + lane_addr + qd * 16, ra, t_dk + lane_addr + 64 + qd * 16, rb);
      tc::tc_fence_before();
      rows_read();
      tile128_out(p_tile, ra, rb, lg, qd * 16, lane, a.scale, a.cosT != nullptr, rp);
      send(C);
    }
    if (sender) tc::tma_wait_group<0>();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (tid == 0) tc::report_given_up(s_abort);
  if (warp == BWD128_MMA_WARP) tc::tmem_dealloc(tmem, 512);
}

__global__ void __launch_bounds__(BWD128_THREADS, 1) attn_bwd_q128_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do,
                                                                     const __grid_constant__ CUtensorMap tm_out, const AttnArgs a) {
  mlb_pdl_sync();
  using S = BwdQ128Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + S::BAR);
  uint64_t *bar_q = bars, *bar_qf = bars + 1, *bar_k = bars + 2 /*[3]*/, *bar_kf = bars + 5 /*[3]*/, *bar_v = bars + 8 /*[2]*/, *bar_vf = bars + 10 /*[2]*/,
           *bar_s = bars + 12 /*[2]*/, *bar_dp = bars + 14, *bar_done = bars + 15,
           *bar_ds = bars + 16 /*[2]: the thread that issues dQ may be a block behind*/;
  uint64_t* bar_end = bars + 18;      // [2]: the MMA threads' last commits
  uint64_t *bar_o = bars + 20 /* dO */, *bar_of = bars + 21 /* dQ has left dO's place */, *bar_out = bars + 22 /* dQ is there */;
  uint32_t* tmem_slot = (uint32_t*)(bars + 23);
  volatile int* s_abort = (volatile int*)(bars + 24);
  if (attn_given_up()) return;
  const int nq = (a.T + 127) / 128, BH = a.B * a.H, C = a.H * H128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* srow = a.sched ? a.sched + (size_t)blockIdx.x * a.sched_stride : nullptr;
  int* s_sched = (int*)(smem + S::SCHED);
  if (srow && tid < 64) s_sched[tid] = tid < a.sched_stride ? __ldg(srow + tid) : -1;
  const ItemList items{srow, s_sched, (int)blockIdx.x, (int)gridDim.x, nq * BH};
  if (tid == 0) {
    for (int i = 0; i < 23; i++) tc::mbar_init(&bars[i], (i == 16 || i == 17 || i == 22) ? BWD128_E_WARPS : 1);
    *s_abort = 0;
    tc::mbar_fence_init();
    tc::tma_prefetch_desc(&tm);
    tc::tma_prefetch_desc(&tm_do);
    tc::tma_prefetch_desc(&tm_out);
  }
  if (warp == BWD128_MMA_WARP) tc::tmem_alloc(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t t_dp = tmem + 256, t_dq = tmem + 384;      // S buffers at +0 and +128
  auto wait = [&](uint64_t* bar, uint32_t phase, int where) { return tc::mbar_wait_sticky(bar, phase, where, s_abort); };
  // item w = query tile (heaviest, the last, first) of (sample, head), with qt + 1 key blocks
  if (warp == BWD128_LOAD_WARP) {
    if (lane == 0) {
      // The next query tile's Q is asked for when the last scores of this one are there, its dO when dQ has left by its place
      // (behind the first two K: it comes last, and nothing waits for it alone)
      int g = 0, gv = 0, nx = 0, no = 0;
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const int qt = nq - 1 - w / BH, bh = w % BH, b = bh / a.H, xh = (bh % a.H) * H128;
        for (int j = 0; j <= qt; j++) {
          const int ks = g % 3, vs = gv & 1;
          if (j == 0) {
            if (li > 0 && !wait(bar_qf, (li - 1) & 1, 72)) { ok = false; break; }
            nx++;
            tc::mbar_expect_tx(bar_q, T128_BYTES);
            split_load<2>(smem + S::Q, &tm, bar_q, xh, qt * 128, b, 2);
          }
          if (g >= 3 && !wait(&bar_kf[ks], (g / 3 + 1) & 1, 73)) { ok = false; break; }
          g++;
          tc::mbar_expect_tx(&bar_k[ks], T128_BYTES);
          split_load<2>(smem + S::K + ks * T128_BYTES, &tm, &bar_k[ks], C + xh, j * 128, b, 2);
          if (j == min(1, qt)) {
            if (li > 0 && !wait(bar_of, (li - 1) & 1, 91)) { ok = false; break; }
            no++;
            tc::mbar_expect_tx(bar_o, T128_BYTES);
            split_load<2>(smem + S::DO, &tm_do, bar_o, xh, qt * 128, b, 2);
          }
          if (gv >= 2 && !wait(&bar_vf[vs], ((gv >> 1) + 1) & 1, 74)) { ok = false; break; }
          gv++;
          tc::mbar_expect_tx(&bar_v[vs], T128_BYTES);
          split_load<2>(smem + S::V + vs * T128_BYTES, &tm, &bar_v[vs], 2 * C + xh, j * 128, b, 2);
        }
      }
      attn_settle(bar_q, nx);
      attn_settle(bar_o, no);
      for (int i = 0; i < 3; i++) attn_settle(&bar_k[i], (g + 2 - i) / 3);
      for (int i = 0; i < 2; i++) attn_settle(&bar_v[i], (gv + 1 - i) / 2);
    }
  } else if (warp == BWD128_MMA_WARP) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc_s = tc::idesc_bf16(128, 128, 0, 0);
      const uint64_t dQ = desc_base_k(tc::smem_u32(smem + S::Q)), dO = desc_base_k(tc::smem_u32(smem + S::DO));
      const uint64_t dK0 = desc_base_k(tc::smem_u32(smem + S::K)), dV0 = desc_base_k(tc::smem_u32(smem + S::V));
      // a block of this CTA's sequence of items, which the products run through without a break: block j of n of item li
      struct Cursor { int li, j, n; };
      auto blocks = [&](int li) { const int w = items.at(li); return w < 0 ? 0 : nq - w / BH; };      // 0: past the last item
      auto next = [&](Cursor c) {
        if (c.n > 0 && ++c.j == c.n) { c.li++; c.j = 0; c.n = blocks(c.li); }
        return c;
      };
      bool ok = true;
      auto scores = [&](int gb, const Cursor& c) {      // over dS of block gb - 2, which its dQ reads
        const int sl = gb % 3;
        if (!ok || (c.j == 0 && !wait(bar_q, c.li & 1, 77)) || !wait(&bar_k[sl], (gb / 3) & 1, 75) ||
            (gb > 1 && !wait(&bar_kf[(gb - 2) % 3], ((gb - 2) / 3) & 1, 85))) { ok = false; return; }
        tc::tc_fence_after();
        const uint64_t dK = dK0 + sl * T128_UNITS;
        const uint32_t t_s = tmem + (gb & 1) * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_s, dQ + off_k(ks, TILE_BYTES), dK + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
        tc::mma_commit(&bar_s[gb & 1]);
        if (c.j + 1 == c.n) tc::mma_commit(bar_qf);
      };
      auto dprobs = [&](int gb, const Cursor& c) {
        if (!ok || (c.j == 0 && !wait(bar_o, c.li & 1, 92)) || !wait(&bar_v[gb & 1], (gb >> 1) & 1, 76)) { ok = false; return; }
        tc::tc_fence_after();
        const uint64_t dV = dV0 + (gb & 1) * T128_UNITS;
#pragma unroll
        for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ss(t_dp, dO + off_k(ks, TILE_BYTES), dV + off_k(ks, TILE_BYTES), idesc_s, ks > 0);
        tc::mma_commit(bar_dp);
        tc::mma_commit(&bar_vf[gb & 1]);
      };
      Cursor c0{0, 0, blocks(0)}, c1 = next(c0), c2 = next(c1);
      if (c0.n > 0) scores(0, c0);
      if (c1.n > 0) scores(1, c1);
      if (c0.n > 0) dprobs(0, c0);
      for (int g = 0; ok && c0.n > 0; g++) {
        if (!wait(&bar_ds[g & 1], (g >> 1) & 1, 78)) break;      // dP of this block read
        if (c1.n > 0) dprobs(g + 1, c1);
        if (c2.n > 0) scores(g + 2, c2);
        c0 = c1; c1 = c2; c2 = next(c2);
      }
      tc::mma_commit(&bar_end[0]);
      attn_settle(&bar_end[0], 1);
    }
  } else if (warp == BWD128_GRAD_WARP) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc_g = tc::idesc_bf16(128, H128, 0, 1);
      const uint64_t gK0 = desc_base_mn(tc::smem_u32(smem + S::K));
      int g = 0, kr = 0;      // kr = g % 3
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const int n = nq - w / BH;
        for (int j = 0; j < n; j++, g++) {
          if (!wait(&bar_ds[g & 1], (g >> 1) & 1, 68)) { ok = false; break; }      // dS(j) stored (of an item's first block: the previous dQ read out)
          tc::tc_fence_after();
          const uint64_t gK = gK0 + kr * T128_UNITS;
          const uint32_t t_ds = tmem + (g & 1) * 128;
#pragma unroll
          for (int ks = 0; ks < 8; ks++) tc::mma_bf16_ts(t_dq, t_ds + split_col(ks), gK + off_mn(ks), idesc_g, (j > 0 || ks > 0));
          tc::mma_commit(&bar_kf[kr]);
          kr = kr == 2 ? 0 : kr + 1;
          if (j + 1 == n) tc::mma_commit(bar_done);
        }
      }
      tc::mma_commit(&bar_end[1]);
      attn_settle(&bar_end[1], 1);
    }
  } else if (warp == BWD128_STAT_WARP) {
    // dQ tiles on their way out
    if (lane == 0) {
      bool ok = true;
      for (int li = 0, w; ok && (w = items.at(li)) >= 0; li++) {
        const int qt = nq - 1 - w / BH, bh = w % BH, b = bh / a.H, x = (bh % a.H) * H128;
        ok = wait(bar_out, li & 1, 94);
        if (!ok) break;
        for (int lg = 0; lg < 4; lg++)      // (the tile comes here after a wait that ran out, too)
          if (!*s_abort && a.T - (qt * 128 + lg * 32) >= 32)
            for (int c = 0; c < 2; c++) tc::tma_store_2d(&tm_out, smem + S::DO + c * TILE_BYTES + lg * 4096, x + c * 64, b * a.T + qt * 128 + lg * 32);
        tc::tma_commit_group();
        tc::tma_wait_group_read<0>();
        tc::mbar_arrive(bar_of);
      }
      tc::tma_wait_group<0>();
    }
  } else if (warp < BWD128_E_WARPS) {
    const int lg = warp & 3, qd = warp >> 2, row = lg * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(lg * 32) << 16;
    const float sl2 = a.scale * LOG2E;
    int g = 0;
    float next_nl = 0.f, next_delta = 0.f;      // this thread's query of the next item (fetched at the start of the one before it)
    auto fetch = [&](int w) {
      const int q = (nq - 1 - w / BH) * 128 + row;
      const size_t e = (size_t)(w % BH) * a.T + q;
      next_nl = q < a.T ? -a.lse[e] * LOG2E : -INFINITY;
      next_delta = q < a.T ? a.delta[e] : 0.f;
    };
    int w = items.at(0);
    if (w >= 0) fetch(w);
    for (int li = 0; w >= 0; li++) {
      const int qt = nq - 1 - w / BH, bh = w % BH, b = bh / a.H, h = bh % a.H;
      const float nl = next_nl, delta = next_delta;
      w = items.at(li + 1);
      if (w >= 0) fetch(w);
      for (int j = 0; j <= qt; j++, g++) {
        const uint32_t ts = tmem + (g & 1) * 128 + qd * 32 + lane_addr, tdp = t_dp + qd * 32 + lane_addr;
        wait(&bar_s[g & 1], (g >> 1) & 1, 79);
        __syncwarp();
        tc::tc_fence_after();
        float p[32];
        {
          uint32_t r[32];
          tc::tmem_ld32_wait(ts, r);
#pragma unroll
          for (int e = 0; e < 32; e++) p[e] = ex2_approx(fmaf(__uint_as_float(r[e]), sl2, nl));
        }
        if (j == qt) {      // the diagonal block
#pragma unroll
          for (int e = 0; e < 32; e++)
            if (qd * 32 + e > row) p[e] = 0.f;
        }
        wait(bar_dp, g & 1, 80);
        __syncwarp();
        tc::tc_fence_after();
        uint32_t d[32], dw[16];
        tc::tmem_ld32_wait(tdp, d);
#pragma unroll
        for (int x = 0; x < 16; x++)
          dw[x] = pack_bf16(p[2 * x] * (__uint_as_float(d[2 * x]) - delta), p[2 * x + 1] * (__uint_as_float(d[2 * x + 1]) - delta));
        tc::tmem_st16(ts, dw);
        tc::tmem_st_wait();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bar_ds[g & 1]);
      }
      // ---- epilogue, through dO's tile, which every dP has read
      Rope128 rp;
      const int row0 = qt * 128 + lg * 32, nlive = a.T - row0;
      if (a.cosT) rope128(rp, a.cosT, a.sinT, row0, qd * 16, lane, a.T);
      uint32_t ra[2][8], rb[2][8];
      wait(bar_done, li & 1, 81);
      __syncwarp();
      tc::tc_fence_after();
      tc::tmem_ld_pairs_wait(t_dq + lane_addr + qd * 16, ra, t_dq + lane_addr + 64 + qd * 16, rb);
      tc::tc_fence_before();
      tile128_out(tc::smem_u32(smem + S::DO), ra, rb, lg, qd * 16, lane, a.scale, a.cosT != nullptr, rp);
      if (nlive < 32) {
        named_bar_sync(1 + lg, 128);
        if (!*s_abort) tile128_rows(a.out + ((size_t)b * a.T + row0) * 3 * C + h * H128, 3L * C, smem + S::DO, lg, nlive, qd * 32 + lane);
      }
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar_out);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (tid == 0) tc::report_given_up(s_abort);
  if (warp == BWD128_MMA_WARP) tc::tmem_dealloc(tmem, 512);
}
