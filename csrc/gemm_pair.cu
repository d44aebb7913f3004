// Quantised linear layers for passes of more than 64 tokens: pairs of CTAs on 256 weight rows, persistent.
//
//   Y[t, n] = sum_k X[t, k] * W[n, k]       W: INT4 or INT8 chunks of 128 x 128 (repack.cu), dequantised to fp16 on the way
//
// What bounded the one-CTA kernel (gemm_w4.cu, 128 rows x 256 tokens a CTA) here: its tensor pipe was busy 55 % of the time
// (75 k cycles a tile, 41 k of them MMA, 14B gate/up).  A tile's prologue and epilogue stood in the open, and 128 K columns
// of 256 tokens plus a chunk are 72 KB for 1024 cycles of MMA - more than the L2 gives every SM at once (60 B per cycle).
// Hence
//   - cta_group::2: one tcgen05.mma works on the 256 rows of two CTAs.  Each loads its own 128 rows and HALF of the tokens'
//     activations, which halves the activation traffic (40 B per cycle and SM);
//   - one pair per two SMs takes unit after unit (a unit: 256 rows x nt tokens x a range of K).  While the last MMAs of
//     a unit run the dequantising warps fill the four operand slots for the next one, and only then empty the accumulator:
//     the pipe stands still for the TMEM reads alone, the stores run under the next unit's MMAs;
//   - nt is a run-time multiple of 32 up to 256, so that 160 tokens do not pay for 256 and unit counts can be fitted to
//     the 74 pairs (plan_pair below).
//
// Roles of a CTA (608 threads): warp 0 streams weight chunks (bulk copies), warp 18 the activation stages (tiled TMA, its
// half of the tokens, counted in at the leader's barrier), warps 2-17 dequantise chunks into TMEM (four groups of four warps,
// group g takes every fourth chunk) and run the epilogues, warp 1 of the LEADER (cluster rank 0) issues
// the MMAs of both CTAs.  Its commits reach both CTAs (multicast arrive); nothing is loaded with multicast.
//
// Barriers: w_full / w_empty (own CTA), x_full (leader: bytes of both), a_ready (leader: 4 warps of each CTA), done (both: the
// MMAs of the chunk in slot s are complete - frees the operand slot and the activation stage of the same index; nobody gets two uses of a
// slot ahead, so one parity tells them apart), acc_full
// (both), acc_empty (leader: 16 warps of each CTA have read their part).  The weight ring's depth is a multiple of four, so
// that a slot is always read by the same group.
//
// Measured (B200, cold L2, one-CTA kernel before -> this one): 14B gate/up 2048 tokens 524 -> 385 us (1506 TFLOP/s, 0.90 of the
// measured cuBLAS burst peak), down 279 -> 181 us (1599), o 131 -> 78 us, QKV 154 -> 115 us; 7B gate/up 77 tokens 50 -> 38 us, INT8
// 1500 tokens (expanded to fp16 first before) 411 + 74 -> 295 us.
#include "gemm_common.cuh"

namespace zse {

constexpr int kPairThreads = 608;
constexpr int kPairMaxSlots = 7;                 // operand slots in TMEM = activation stages
constexpr int kPairMaxSW = 16;
constexpr int kPairW8Chunk = 16640;              // 128 x 128 int8 + 128 scales
constexpr int kPairXch = 16384;                  // gate/up exchange of eight warp pairs
constexpr int kPairSmemMax = 232448;
constexpr int kPairTmem = 512;                   // columns: the accumulator first, the operand slots (64 each) last

struct PairBars {
  uint64_t w_full[kPairMaxSW], w_empty[kPairMaxSW];
  uint64_t x_full[kPairMaxSlots], a_ready[kPairMaxSlots], done[kPairMaxSlots];
  uint64_t acc_full, acc_empty;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(PairBars) <= 512, "barriers fit their place");

struct PairArgs {
  const uint8_t* w;        // chunks [n_tiles][k_stages]
  const __half* bias;      // [N] or null (kEpiF16)
  void* out;
  int M, N, ldo;
  int k_stages, spp, ks;   // K stages of 128, per split, splits (fp32 planes)
  int n_tiles, n_pairs;    // 128-row tiles, pairs of them
  int nt, m_tiles, m_group;
  int sw;                  // depth of the weight ring
  int slots;               // operand slots and activation stages
  Status* status;
  GatherWait gather;       // flags not null: x is a gathered buffer, wait for the row blocks of a unit's tokens
};

struct PairUnit {
  int n, m, z, s0, n_k;
};
// Units in an order that keeps m_group token tiles (about 2048 tokens) in L2 while the weights stream past them once.
__device__ __forceinline__ PairUnit pair_unit(const PairArgs& a, int i) {
  PairUnit u;
  const int per_z = a.n_pairs * a.m_tiles;
  u.z = i / per_z;
  int r = i - u.z * per_z;
  const int mg = r / (a.n_pairs * a.m_group);
  r -= mg * a.n_pairs * a.m_group;
  const int gm = min(a.m_group, a.m_tiles - mg * a.m_group);
  u.n = r / gm;
  u.m = mg * a.m_group + r % gm;
  u.s0 = u.z * a.spp;
  u.n_k = min(a.k_stages, u.s0 + a.spp) - u.s0;
  return u;
}

__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for arrivals that may come from the other CTA of the pair (same contract as mbar_wait).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, Status* st,
                                                  unsigned where, unsigned detail) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  uint64_t t0 = 0;
  unsigned spins = 0;
  while (!mbar_try_wait_cluster(bar, parity)) {
    if ((++spins & 0xFF) == 0) {
      if (*abort_flag) return false;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > kWaitLimitNs) {
        report(st, kWaitTimeout, where, detail);
        *abort_flag = 1;
        __threadfence_block();
        return false;
      }
    }
  }
  return true;
}
// Tiled load into this CTA's shared memory whose bytes are counted at a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(cluster_bar)
      : "memory");
}
__device__ __forceinline__ void umma_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {          // arrives at this offset in both CTAs
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(uint16_t(3))
      : "memory");
}
__device__ __forceinline__ void pair_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// All-gather in the prologue: rows [t0, t1) were written into this GPU's memory by their owners (other GPUs, plain or
// multicast stores); a row block is complete when its flag holds the pass epoch.  One thread waits (bounded), then orders those
// writes before the TMA loads it is about to issue (async proxy).
__device__ __forceinline__ bool pair_gather_wait(const GatherWait& g, int t0, int t1, volatile int* abort_flag, Status* st) {
  const uint32_t want = *reinterpret_cast<const volatile uint32_t*>(g.epoch);
  auto flag = [&](int b) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(g.flags + b) : "memory");
    return v;
  };
  bool ok = true;
  for (int b = t0 / kSpRowBlock; b * kSpRowBlock < t1 && ok; ++b) {
    SpinClock clk;
    while (flag(b) != want) {
      if (clk.expired(0x3F) || ((clk.spins & 0x3F) == 0 && *abort_flag)) {
        report(st, kPeerTimeout, 36, unsigned(b));
        *abort_flag = 1;
        ok = false;
        break;
      }
    }
  }
  asm volatile("fence.proxy.async;" ::: "memory");
  return ok;
}

// A 32-bit word of eight nibbles -> four half2 (order fixed by repack.cu: adjacent pairs come out of one mask).
__device__ __forceinline__ void pair_dequant_w4(uint32_t w, __half2 s2, __half2 z2, uint32_t* out4) {
  const __half2 k1024 = __half2half2(__ushort_as_half(0x6400));
  const __half2 k16th = __half2half2(__ushort_as_half(0x2C00));   // 1/16
  const __half2 kNeg64 = __half2half2(__ushort_as_half(0xD400));  // -64
  const uint32_t w8 = w >> 8;
  uint32_t t[4];
  asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xEA;" : "=r"(t[0]) : "r"(w));
  asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xEA;" : "=r"(t[1]) : "r"(w));
  asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xEA;" : "=r"(t[2]) : "r"(w8));
  asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xEA;" : "=r"(t[3]) : "r"(w8));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 h = *reinterpret_cast<__half2*>(&t[i]);
    const __half2 q = (i & 1) ? __hfma2(h, k16th, kNeg64) : __hsub2(h, k1024);
    const __half2 e = __hfma2(q, s2, z2);
    out4[i] = *reinterpret_cast<const uint32_t*>(&e);
  }
}
// Sixteen int8 -> eight half2: a byte b under the exponent of 1024 is 1024 + (b + 128); minus 1152 leaves b exactly.
__device__ __forceinline__ void pair_dequant_w8(const uint4& w, __half2 s2, uint32_t* out8) {
  const __half2 k1152 = __half2half2(__ushort_as_half(0x6480));
  const uint32_t in[4] = {w.x ^ 0x80808080u, w.y ^ 0x80808080u, w.z ^ 0x80808080u, w.w ^ 0x80808080u};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t lo = __byte_perm(in[i], 0x64646464u, 0x4140), hi = __byte_perm(in[i], 0x64646464u, 0x4342);
    const __half2 x = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&lo), k1152), s2);
    const __half2 y = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&hi), k1152), s2);
    out8[2 * i] = *reinterpret_cast<const uint32_t*>(&x);
    out8[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&y);
  }
}

// The accumulator of one unit: 16-column chunks g, g + 4, ... belong to warp group g, which takes two of them at a time (all
// four at once did not fit 96 registers, and spilled values missed what little L1 the rings leave) and hands the accumulator
// back before it works on the last two.  `live` is false once a wait of this warp ran out: it then takes part in the barriers
// only.
template <int EPI>
__device__ __forceinline__ void pair_epilogue(const PairArgs& a, int tile, int t0, int z, uint32_t taddr, int g, int q,
                                              int lane, uint32_t empty_bar, float* xch, bool live) {
  if (live) tc_fence_after_sync();
#pragma unroll 1
  for (int b = 0; b < 2; ++b) {
    uint32_t v[2][16];
    const int ca = (g + 8 * b) * 16;                           // first columns of the two chunks: ca, ca + 64
    if (live) {
      if (ca < a.nt) ZSE_TMEM_LD_X16(v[0], taddr + ca);
      if (ca + 64 < a.nt) ZSE_TMEM_LD_X16(v[1], taddr + ca + 64);
      tc_wait_ld();
      if (b == (a.nt > 128)) {                                 // nothing of this group's columns is left to read
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(empty_bar);
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int c0 = ca + 64 * c;
      if (c0 < a.nt) {
        if (EPI == kEpiSwiGLU) {
          // rows 0..63 of a tile are gate, 64..127 the up rows of the same outputs: the two warps that hold them swap
          // half of their columns and finish eight each
          float* give = xch + ((q & 1) + 2 * g) * 512 + (q < 2 ? 0 : 256) + lane;
          const float* take = xch + ((q & 1) + 2 * g) * 512 + (q < 2 ? 256 : 0) + lane;
          const int bar_id = 1 + (q & 1) + 2 * g;
          if (live) {
#pragma unroll
            for (int i = 0; i < 8; ++i) give[i * 32] = __uint_as_float(q < 2 ? v[c][8 + i] : v[c][i]);
          }
          asm volatile("bar.sync %0, 64;" ::"r"(bar_id) : "memory");
          const int n = tile * 64 + (q & 1) * 32 + lane;
          const int t = t0 + c0 + (q < 2 ? 0 : 8);
          if (live && tile < a.n_tiles && n < a.N / 2) {
            __half* out = reinterpret_cast<__half*>(a.out) + size_t(t) * a.ldo + n;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float other = take[i * 32];
              const float gate = q < 2 ? __uint_as_float(v[c][i]) : other;
              const float up = q < 2 ? other : __uint_as_float(v[c][8 + i]);
              if (t + i < a.M) *out = __float2half_rn(clamp_f16(silu_f(gate) * up));
              out += a.ldo;
            }
          }
          asm volatile("bar.sync %0, 64;" ::"r"(bar_id) : "memory");
        } else {
          const int n = tile * kTileN + q * 32 + lane;
          if (live && tile < a.n_tiles && n < a.N) {
            const float bias = EPI == kEpiF16 && a.bias != nullptr ? __half2float(a.bias[n]) : 0.f;
            const int t = t0 + c0;
            if (EPI == kEpiF16) {
              __half* out = reinterpret_cast<__half*>(a.out) + size_t(t) * a.ldo + n;
#pragma unroll
              for (int i = 0; i < 16; ++i, out += a.ldo)
                if (t + i < a.M) *out = __float2half_rn(clamp_f16(__uint_as_float(v[c][i]) + bias));
            } else {
              float* out = reinterpret_cast<float*>(a.out) + (size_t(z) * a.M + t) * a.ldo + n;
#pragma unroll
              for (int i = 0; i < 16; ++i, out += a.ldo)
                if (t + i < a.M) *out = __uint_as_float(v[c][i]);
            }
          }
        }
      }
    }
  }
}

template <int EPI, bool W8>
__global__ void __launch_bounds__(kPairThreads, 1) __cluster_dims__(2, 1, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const PairArgs a) {
  constexpr int kChunk = W8 ? kPairW8Chunk : kW4ChunkBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int x_sub = a.nt * 64;                                 // bytes of 64 K columns of this CTA's nt / 2 tokens
  const int x_stage = 2 * x_sub;
  uint8_t* w_ring = smem + a.slots * x_stage;
  float* xch = reinterpret_cast<float*>(w_ring + a.sw * kChunk);
  PairBars* bars = reinterpret_cast<PairBars*>(reinterpret_cast<uint8_t*>(xch) + kPairXch);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t crank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const int pair = blockIdx.x >> 1, n_workers = gridDim.x >> 1;
  const int n_units = a.n_pairs * a.m_tiles * a.ks;
  if (threadIdx.x == 0) {
    for (int i = 0; i < a.sw; ++i) {
      mbar_init(&bars->w_full[i], 1);
      mbar_init(&bars->w_empty[i], 4);
    }
    for (int i = 0; i < a.slots; ++i) {
      mbar_init(&bars->x_full[i], 1);
      mbar_init(&bars->a_ready[i], 8);
      mbar_init(&bars->done[i], 1);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->acc_empty, 32);
    bars->abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmap_x);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  pair_cluster_sync();                                         // both CTAs' barriers exist before anybody signals them
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  pdl_launch_dependents();                                     // (the TMEM is ours: a dependent cannot take it first)

  if (warp == 0) {
    // ------------------------------------------------------------------ weight chunks of this CTA's 128 rows
    if (lane == 0) {
      int s = 0, c = 0;
      uint32_t ph = 1;
      bool live = true;
      for (int i = pair; i < n_units && live; i += n_workers) {
        const PairUnit u = pair_unit(a, i);
        const int tile = min(u.n * 2 + int(crank), a.n_tiles - 1);       // the missing half of an odd pair is computed, not stored
        const uint8_t* src = a.w + (size_t(tile) * a.k_stages + u.s0) * kChunk;
        for (int k = 0; k < u.n_k; ++k, ++c, src += kChunk) {
          if (c >= a.sw && !mbar_wait(&bars->w_empty[s], ph, abort_flag, a.status, 41, c)) {
            live = false;
            break;
          }
          mbar_arrive_expect_tx(&bars->w_full[s], kChunk);
          bulk_g2s(w_ring + s * kChunk, src, kChunk, &bars->w_full[s]);
          if (++s == a.sw) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 18) {
    // ------------------------------------------------------------------ activations: this CTA's half of the tokens
    if (lane == 0) {
      int c = 0, s = 0;
      uint32_t ph = 1;
      bool live = true;
      uint64_t arrived = 0;                                    // token tiles (the first 64) whose rows have been seen
      pdl_wait();                                              // they come from the previous kernel
      const uint32_t ring = smem_u32(smem);
      for (int i = pair; i < n_units && live; i += n_workers) {
        const PairUnit u = pair_unit(a, i);
        const int row = u.m * a.nt + int(crank) * (a.nt / 2);
        if (a.gather.flags != nullptr && (u.m > 63 || ((arrived >> u.m) & 1) == 0)) {
          if (!pair_gather_wait(a.gather, row, min(row + a.nt / 2, a.M), abort_flag, a.status)) break;
          if (u.m <= 63) arrived |= 1ull << u.m;
        }
        for (int k = 0; k < u.n_k; ++k, ++c) {
          // the MMAs of the chunk that had this stage before are complete: it may be refilled
          if (c >= a.slots && !mbar_wait(&bars->done[s], ph, abort_flag, a.status, 42, c)) {
            live = false;
            break;
          }
          const uint32_t full = map_to_rank(smem_u32(&bars->x_full[s]), 0);
          if (crank == 0) mbar_arrive_expect_tx(&bars->x_full[s], 2 * x_stage);
          const uint32_t dst = ring + s * x_stage;
          const int k0 = (u.s0 + k) * kW4StageK;
          tma_load_2d_pair(dst, &tmap_x, k0, row, full);
          tma_load_2d_pair(dst + x_sub, &tmap_x, k0 + 64, row, full);
          if (++s == a.slots) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMAs of both CTAs
    // The whole warp walks the loop and one elected lane issues (see elect_one): 260 cycles a chunk, 650 with a single lane.
    if (crank == 0) {
      const uint32_t idesc = (1u << 4) | (uint32_t(a.nt >> 3) << 17) | (uint32_t(256 >> 4) << 24);
      const uint64_t desc0 = make_desc_sw128(smem_u32(smem));
      int c = 0, s = 0, j = 0;
      uint32_t ph = 0;
      bool live = true;
      for (int i = pair; i < n_units && live; i += n_workers, ++j) {
        const PairUnit u = pair_unit(a, i);
        live = j == 0 || __all_sync(0xffffffffu, mbar_wait_cluster(&bars->acc_empty, (j - 1) & 1, abort_flag, a.status, 43, j));
        for (int k = 0; k < u.n_k && live; ++k, ++c) {
          live = __all_sync(0xffffffffu, mbar_wait_cluster(&bars->x_full[s], ph, abort_flag, a.status, 44, c) &&
                                             mbar_wait_cluster(&bars->a_ready[s], ph, abort_flag, a.status, 45, c));
          if (!live) break;
          tc_fence_after_sync();
          const uint64_t bd = desc0 + uint64_t((s * x_stage) >> 4);
          const uint32_t at = tmem + kPairTmem - (a.slots - s) * 64;
          if (elect_one()) {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj)
              umma_ts_pair(tmem, at + jj * 8, bd + uint64_t((jj >> 2) * (x_sub >> 4) + (jj & 3) * 2), idesc, (k | jj) != 0);
            tc_commit_pair(&bars->done[s]);
            if (k == u.n_k - 1) tc_commit_pair(&bars->acc_full);
          }
          __syncwarp();
          if (++s == a.slots) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dequantisation and epilogues
    const int q = warp & 3, g = (warp - 2) >> 2;               // TMEM lane quarter, group
    const int row = q * 32 + lane;
    const uint32_t slot0 = tmem + (uint32_t(q * 32) << 16) + kPairTmem - a.slots * 64;
    const uint32_t ready_bar = map_to_rank(smem_u32(&bars->a_ready[0]), 0);
    const uint32_t empty_bar = map_to_rank(smem_u32(&bars->acc_empty), 0);
    int sw = g, slot = g;
    uint32_t wph = 0, sph = 1;                                 // parities: of the weights' arrival, of the slot's last use
    bool live = true, stores = false;
    int first = 0;                                             // chunk number of the unit's first chunk
    int j = 0;                                                 // units of this pair seen
    int next = g;                                              // this group's next chunk
    int epi = pair;                                            // unit whose epilogue comes next, and its number
    int epi_j = 0;
    auto finish = [&]() {
      if (!stores) {
        pdl_wait();                                            // the output may still be read by the previous kernel
        stores = true;
      }
      live = live && mbar_wait(&bars->acc_full, epi_j & 1, abort_flag, a.status, 48, epi_j);
      const PairUnit e = pair_unit(a, epi);
      pair_epilogue<EPI>(a, e.n * 2 + int(crank), e.m * a.nt, e.z, tmem + (uint32_t(q * 32) << 16), g, q, lane, empty_bar,
                         xch, live);
      epi += n_workers;
      ++epi_j;
    };
    for (int i = pair; i < n_units; i += n_workers, ++j) {
      const PairUnit u = pair_unit(a, i);
      for (; next < first + u.n_k; next += 4) {
        live = live && mbar_wait(&bars->w_full[sw], wph, abort_flag, a.status, 46, next);
        if (live) {
          const uint8_t* chunk = w_ring + sw * kChunk + row * 16;
          __half2 s2, z2;
          if (W8) {
            s2 = __half2half2(*reinterpret_cast<const __half*>(w_ring + sw * kChunk + 16384 + row * 2));
          } else {
            const __half2 sz = *reinterpret_cast<const __half2*>(w_ring + sw * kChunk + 8192 + row * 4);
            s2 = __half2half2(__low2half(sz)), z2 = __half2half2(__high2half(sz));
          }
          uint32_t o[2][16];                                   // 32 K columns ahead of the wait for the operand slot
          auto quarter = [&](int hh, uint32_t* to) {
            if constexpr (W8) {
#pragma unroll
              for (int p = 0; p < 2; ++p)
                pair_dequant_w8(*reinterpret_cast<const uint4*>(chunk + (hh * 2 + p) * 2048), s2, to + p * 8);
            } else {
              const uint4 w4 = *reinterpret_cast<const uint4*>(chunk + hh * 2048);
              pair_dequant_w4(w4.x, s2, z2, to + 0);
              pair_dequant_w4(w4.y, s2, z2, to + 4);
              pair_dequant_w4(w4.z, s2, z2, to + 8);
              pair_dequant_w4(w4.w, s2, z2, to + 12);
            }
          };
          quarter(0, o[0]);
          if (next >= a.slots) live = mbar_wait(&bars->done[slot], sph, abort_flag, a.status, 47, next);
          if (live) {
            tc_fence_after_sync();
            const uint32_t dst = slot0 + slot * 64;
            ZSE_TMEM_ST_X16(dst, o[0]);
            quarter(1, o[1]);
            ZSE_TMEM_ST_X16(dst + 16, o[1]);
            quarter(2, o[0]);
            ZSE_TMEM_ST_X16(dst + 32, o[0]);
            quarter(3, o[1]);
            ZSE_TMEM_ST_X16(dst + 48, o[1]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->w_empty[sw]);    // the chunk has been read: its slot may be refilled
            tc_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(ready_bar + slot * 8);
          }
        }
        sw += 4;
        if (sw >= a.sw) { sw -= a.sw; wph ^= 1; }
        slot += 4;
        if (slot >= a.slots) { slot -= a.slots; sph ^= 1; }
        // the first chunk of this unit lies in its slot: now the accumulators of the units before it
        while (epi_j < j) finish();
      }
      first += u.n_k;
    }
    while (epi_j < j) finish();
  }
  __syncthreads();
  if (*abort_flag) {                                           // copies in flight must land before the CTA may leave
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) {
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  pair_cluster_sync();                                         // nobody leaves while the other CTA may still signal it
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ---- plan ------------------------------------------------------------------------------------------------------------------
// Tokens per unit and K splits.  A unit costs spp chunks (8 MMAs of nt / 2 cycles on a pair and what surrounds them, but not
// less than a chunk takes to arrive and be dequantised) and a fixed part for the hand-over of the accumulator; all pairs work in
// rounds.
// More token tiles than necessary can be right when they fill the last round better; K splits (planes, where the consumer
// adds them) fill the machine when there are fewer units than pairs, at the price of writing and reading a plane each.
struct PairPlan {
  int nt, m_tiles, ks;
};
static PairPlan plan_pair(int M, int N, int K, bool planes_ok, int n_tiles, int sm_count, int want_split) {
  const int workers = max(1, sm_count / 2);
  const int n_pairs = (n_tiles + 1) / 2, k_stages = K / kW4StageK;
  PairPlan best{256, (M + 255) / 256, 1};
  double best_cost = -1;
  const int mt0 = (M + 255) / 256;
  for (int mt = mt0; mt <= mt0 + 3; ++mt) {
    const int nt = min(256, ((M + mt - 1) / mt + 31) / 32 * 32);
    const int m_tiles = (M + nt - 1) / nt;
    const int max_ks = planes_ok ? min(8, k_stages) : 1;
    for (int ks = 1; ks <= max_ks; ++ks) {
      if (planes_ok && want_split > 0 && ks != min(want_split, max_ks)) continue;
      const int spp = (k_stages + ks - 1) / ks;
      const long units = long(n_pairs) * m_tiles * ks;
      const long rounds = (units + workers - 1) / workers;
      const double chunk = max(6.6 * nt, 950.0);               // cycles, from timed layers of 72 to 512 tokens
      double cost = double(rounds) * (spp * chunk + 3000.0);
      cost += double(ks - 1) * double(M) * N * 8.0 / 4000.0;
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best = PairPlan{nt, m_tiles, ks};
      }
    }
  }
  const int spp = (k_stages + best.ks - 1) / best.ks;
  best.ks = (k_stages + spp - 1) / spp;                        // no empty split
  return best;
}

static int pair_sm_count() {
  static int sms[kMaxDevices] = {};
  const int d = current_device_slot();
  if (sms[d] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || n <= 1) n = 148;
    sms[d] = n;
  }
  return sms[d];
}

static int pair_n_tiles(int N, int epilogue) {
  return epilogue == kEpiSwiGLU ? (N / 2 + 63) / 64 : (N + kTileN - 1) / kTileN;
}

template <int EPI, bool W8>
static int launch_pair(const CUtensorMap& tx, const PairArgs& a, int smem, cudaStream_t st) {
  auto kern = gemm_pair_kernel<EPI, W8>;
  static bool attr_done[kMaxDevices] = {};
  const int dev = current_device_slot();
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemMax) != cudaSuccess)
      return ZSE_ERR_LAUNCH;
    attr_done[dev] = true;
  }
  const int units = a.n_pairs * a.m_tiles * a.ks;
  return launch_pdl(kern, dim3(2 * min(pair_sm_count() / 2, units)), dim3(kPairThreads), size_t(smem), st, tx, a) ==
                 cudaSuccess
             ? 0
             : ZSE_ERR_LAUNCH;
}

int gemm_pair_planes(int M, int N, int K, int want_split) {
  return plan_pair(M, N, K, true, pair_n_tiles(N, kEpiPartialF32), pair_sm_count(), want_split).ks;
}

void gemm_pair_plan(int M, int N, int K, int epilogue, int want_split, int sm_count, int* tokens, int* splits) {
  const PairPlan p = plan_pair(M, N, K, epilogue == kEpiPartialF32, pair_n_tiles(N, epilogue), sm_count, want_split);
  *tokens = p.nt;
  *splits = p.ks;
}

int gemm_pair_run(bool w8, const void* w_tiled, const void* x, int x_rows_cap, const void* bias, void* out, int M, int N,
                  int K, int ldo, int epilogue, int want_split, const GatherWait* gather, Status* status, cudaStream_t st) {
  if (M <= 0) return 0;
  if (K % kW4StageK != 0 || N <= 0 || K <= 0) return ZSE_ERR_SHAPE;
  const int n_tiles = pair_n_tiles(N, epilogue);
  const PairPlan p = plan_pair(M, N, K, epilogue == kEpiPartialF32, n_tiles, pair_sm_count(), want_split);
  const int k_stages = K / kW4StageK;
  const int chunk = w8 ? kPairW8Chunk : kW4ChunkBytes;
  const int slots = min(kPairMaxSlots, (kPairTmem - p.nt) / 64);
  const int fixed = slots * p.nt * 128 + kPairXch + 512 + 1024;
  const int sw = min(kPairMaxSW, (kPairSmemMax - fixed) / chunk / 4 * 4);
  CUtensorMap tx;
  if (int rc = get_tmap(x, uint64_t(max(x_rows_cap, M)), uint64_t(K), uint32_t(p.nt / 2), &tx)) return rc;
  const int groups = (p.m_tiles * p.nt + 2047) / 2048;         // token tiles in equal groups of about 2048 tokens
  PairArgs a{reinterpret_cast<const uint8_t*>(w_tiled), reinterpret_cast<const __half*>(bias), out, M, N, ldo, k_stages,
             (k_stages + p.ks - 1) / p.ks, p.ks, n_tiles, (n_tiles + 1) / 2, p.nt, p.m_tiles,
             (p.m_tiles + groups - 1) / groups, sw, slots, status,
             gather != nullptr ? *gather : GatherWait{nullptr, nullptr}};
  const int smem = fixed + sw * chunk;
  switch (epilogue) {
    case kEpiF16: return w8 ? launch_pair<kEpiF16, true>(tx, a, smem, st) : launch_pair<kEpiF16, false>(tx, a, smem, st);
    case kEpiSwiGLU:
      return w8 ? launch_pair<kEpiSwiGLU, true>(tx, a, smem, st) : launch_pair<kEpiSwiGLU, false>(tx, a, smem, st);
    case kEpiPartialF32:
      return w8 ? launch_pair<kEpiPartialF32, true>(tx, a, smem, st) : launch_pair<kEpiPartialF32, false>(tx, a, smem, st);
    default: return ZSE_ERR_SHAPE;
  }
}

}  // namespace zse

using namespace zse;

// Linear layer on INT8 chunks for passes of more than 64 tokens (epilogues fp16, SwiGLU, fp32 planes); k_split as in
// zse_gemm_w4, planes written: zse_gemm_w8_splits.  (Reference: tiled_dequant_matmul_int8,
// zse-engine/zse_engine/orchestrator/kernels.py:1195-1249.)
extern "C" int zse_gemm_w8(const void* w_tiled, const void* x, int x_rows_cap, const void* bias, void* out, int M, int N,
                           int K, int ldo, int epilogue, int k_split, void* status, void* stream) {
  return gemm_pair_run(true, w_tiled, x, x_rows_cap, bias, out, M, N, K, ldo, epilogue, k_split, nullptr,
                       reinterpret_cast<Status*>(status), reinterpret_cast<cudaStream_t>(stream));
}
extern "C" int zse_gemm_w8_splits(int M, int N, int K, int k_split) {
  if (M <= 0 || K % kW4StageK != 0 || K <= 0) return 1;
  return gemm_pair_planes(M, N, K, k_split);
}
