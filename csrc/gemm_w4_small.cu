// INT4 group-128 weights x up to 8 tokens: a stream of weights through registers and mma.sync.
//
//   Y[t, n] = sum_k X[t, k] * (nibble[n, k] * scale[n, k/128] + zero[n, k/128])
//
// What bounds it is how fast the SMs can take the weights in.  The tcgen05 kernels (gemm_w4.cu, gemm_w4_dec.cu) expand every
// nibble to fp16 (13 instructions for eight of them), write the result to TMEM and then pay per MMA instruction whatever
// the number of tokens is.  Here
//   - a warp loads the chunks straight from global memory into the A fragments of mma.m16n8k16: lane (g, t) reads the 16
//     bytes = 32 K columns of part t of rows g and g + 8, and as the order of K inside a product is free, each lane's own
//     32 columns serve as its K slots (the lane's B fragments are then 64 contiguous bytes of its token's activations);
//   - nibbles are not converted: masked with 0x000f000f a word is a pair of fp16 subnormals q * 2^-24, with 0x00f000f0 a pair
//     16 q * 2^-24, both exact in the tensor cores.  Five instructions for eight nibbles; the two masks have an accumulator
//     each.  Once per group of 128 the sums meet scale and minimum in fp32:
//         y += scale * (2^24 lo + 2^20 hi) + zero * sum_k x,   sum_k x from one more MMA with a matrix of ones,
//     so weights are never rounded to fp16 as they are in the other kernels;
//   - an item is half a 128-row tile: rows 32h..32h+31 and 64+32h..64+32h+31, which holds both rows of every gate/up pair and
//     of every rotation pair of a 128-wide head.  The warps of a CTA share an item's K groups, each with its next group's
//     weights and activations in flight (70 KB an SM); their sums meet in shared memory, always in the same order.
// Staging the activations as fragments in shared memory first was slower (gate/up of the 7B shape 27.6 us against 23.3: the
// copy and its barrier stand before the first product), and so was not fetching them ahead (26.6).  Started alone from a
// cold L2 that is 3.1 TB/s, launch included; back to back with weights from memory 3.7 TB/s at 7168 x 14336 and 4.7 at 8192 x 28672
// (one token, 14.9 and 26.6 us).  It issues 1.8 instructions per cycle: what is left is latency at the ends of items and issue.
//
// Epilogues: fp16 (+bias), SwiGLU, fp32 planes (K ranges, the consumer adds them), fused QKV (bias, rotate-half RoPE, K/V rows
// into the paged cache).  Replaces for these passes the scalar GEMV kernels of the reference
// (zse-engine/zse_engine/orchestrator/kernels.py:1129-1192,1906-2003).
#include "gemm_common.cuh"

namespace zse {

constexpr int kSmallThreads = 512;               // one CTA of so many an SM, or two of half as many (128 registers a thread)
constexpr int kSmallPitch = 68;                  // floats per token column of 64 rows: conflict-free stores of fragments

struct SmallArgs {
  const uint8_t* w;        // chunks [n_tiles][k_stages][8704]
  const __half* x;         // [M, K]
  const __half* bias;
  void* out;
  int M, N, K, ldo;
  int k_stages, spp, n_half, items;              // K groups, per split; half tiles; half tiles x splits
  SmallRope rope;
};

__device__ __forceinline__ uint4 small_ldg(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t small_ldg1(const void* p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
// D = A B, the first product of a sum
__device__ __forceinline__ void small_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                           uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void small_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A sum that came out infinite or NaN, again with weights as the other kernels have them (fp16 of scale * q + minimum): scale *
// sum(q x) + minimum * sum(x) is inf - inf, or 0 * inf, where an infinite activation times the weight is infinite.  Sums of finite
// activations are finite (products of fp16 numbers, fp32), so nobody else comes here.  One row of a tile, K groups from `chunk` on.
__device__ __forceinline__ float small_not_finite(const uint8_t* chunk, int row, int groups, const __half* x) {
  float y = 0.f;
#pragma unroll 1
  for (int k = 0; k < groups; ++k, chunk += kW4ChunkBytes) {
    const __half2 sz = *reinterpret_cast<const __half2*>(chunk + 8192 + row * 4);
#pragma unroll 1
    for (int i = 0; i < 16; ++i, x += 8) {                     // eight columns a word
      const uint32_t u = *reinterpret_cast<const uint32_t*>(chunk + (i >> 2) * 2048 + row * 16 + (i & 3) * 4);
      for (int c = 0; c < 8; ++c) {
        const int q = (u >> ((c >> 1) * 4 + (c & 1) * 16)) & 15;
        y = fmaf(__half2float(__hfma(__int2half_rn(q), __low2half(sz), __high2half(sz))), __half2float(x[c]), y);
      }
    }
  }
  return y;
}

template <int EPI>
__global__ void __launch_bounds__(kSmallThreads, 1) gemm_w4_small_kernel(const SmallArgs a) {
  extern __shared__ float red[];                               // [warps][8 columns][kSmallPitch]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  pdl_launch_dependents();
  constexpr bool kPairs = EPI == kEpiSwiGLU || EPI == kEpiQkvRope;
  constexpr float kMaxFloat = 3.402823466e38f;
  __shared__ uint32_t odd_tokens;                              // tokens with a sum that is not finite
  if (threadIdx.x == 0) odd_tokens = 0;
  // rows j and 32 + j of a half tile, the two of a gate/up or rotation pair
  auto store2 = [&](int item, int tok, int j, float va, float vb) {
    const int tile = item >> 1, h32 = (item & 1) * 32;         // (these epilogues have no K splits: an item is a half tile)
    if (EPI == kEpiSwiGLU) {
      const int n = tile * 64 + h32 + j;
      if (n < a.N / 2)
        reinterpret_cast<__half*>(a.out)[size_t(tok) * a.ldo + n] = __float2half_rn(clamp_f16(silu_f(va) * vb));
      return;
    }
    // a tile is a head of 128: q heads, k heads, v heads; dims d and d + 64 rotate together
    const SmallRope& rp = a.rope;
    const int d = h32 + j;
    if (a.bias != nullptr) {
      va += __half2float(a.bias[tile * 128 + d]);
      vb += __half2float(a.bias[tile * 128 + 64 + d]);
    }
    if (tile < rp.nh + rp.nkv) {
      const int pos = min(max(rp.positions[tok], 0), rp.max_position - 1);
      const float2 cs = rp.cos_sin[size_t(pos) * 64 + d];
      const float ra = va * cs.x - vb * cs.y, rb = vb * cs.x + va * cs.y;
      va = ra, vb = rb;
    }
    __half* dst = nullptr;
    if (tile < rp.nh) {
      dst = reinterpret_cast<__half*>(a.out) + size_t(tok) * a.ldo + tile * 128;
    } else {
      const long long slot = rp.slots[tok];
      if (slot >= 0) {
        const bool is_v = tile >= rp.nh + rp.nkv;
        const int kvh = tile - rp.nh - (is_v ? rp.nkv : 0);
        const long long blk = slot / rp.block_size, off = slot % rp.block_size;
        dst = rp.kv_layer + (((blk * 2 + (is_v ? 1 : 0)) * rp.nkv + kvh) * rp.block_size + off) * 128;
      }
    }
    if (dst != nullptr) {
      dst[d] = __float2half_rn(clamp_f16(va));
      dst[64 + d] = __float2half_rn(clamp_f16(vb));
    }
  };
  auto store1 = [&](int item, int tok, int row, float s) {
    const int z = item / a.n_half, half = item - z * a.n_half;
    const int n = (half >> 1) * 128 + (half & 1) * 32 + (row < 32 ? row : row + 32);
    if (n >= a.N) return;
    if (EPI == kEpiF16)
      reinterpret_cast<__half*>(a.out)[size_t(tok) * a.ldo + n] =
          __float2half_rn(clamp_f16(s + (a.bias != nullptr ? __half2float(a.bias[n]) : 0.f)));
    else
      reinterpret_cast<float*>(a.out)[(size_t(z) * a.M + tok) * a.ldo + n] = s;
  };

  uint4 w[8];                                                  // [16-row block][row g, row g + 8] of the group in flight
  uint32_t sz[8];
  int f_item = blockIdx.x, f_k = 0, f_end = 0;                 // what is fetched next
  const uint8_t *src = nullptr, *ssz = nullptr;                // its nibbles and scales, from this lane's place on
  // first group of this warp in the next item (from f_item on) that has one for it
  auto seek = [&]() {
    for (; f_item < a.items; f_item += gridDim.x) {
      const int z = f_item / a.n_half, half = f_item - z * a.n_half;
      f_k = z * a.spp + warp;
      f_end = min(a.k_stages, (z + 1) * a.spp);
      if (f_k < f_end) {
        const uint8_t* chunk = a.w + (size_t(half >> 1) * a.k_stages + f_k) * kW4ChunkBytes;
        src = chunk + t * 2048 + ((half & 1) * 32 + g) * 16;
        ssz = chunk + 8192 + ((half & 1) * 32 + g) * 4;
        break;
      }
    }
  };
  auto fetch = [&](int st) {                                   // rows (st & 1) * 16 + (st >> 1) * 64 of the half tile
    const uint8_t* p = src + ((st >> 1) * 64 + (st & 1) * 16) * 16;
    w[2 * st] = small_ldg(p);
    w[2 * st + 1] = small_ldg(p + 128);
  };
  auto fetch_scales = [&]() {
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      const uint8_t* p = ssz + ((st >> 1) * 64 + (st & 1) * 16) * 4;
      sz[2 * st] = small_ldg1(p);
      sz[2 * st + 1] = small_ldg1(p + 32);
    }
  };
  seek();
  if (f_item < a.items) {                                      // weights are constant: they may come before the wait
#pragma unroll
    for (int st = 0; st < 4; ++st) fetch(st);
    fetch_scales();
  }
  pdl_wait();

  const __half* xrow = a.x + size_t(min(g, a.M - 1)) * a.K + t * 32;    // (columns of tokens that are not there are not stored)
  uint4 nx[4];                                                 // activations of the group in flight: 64 bytes of a token
  auto fetch_x = [&]() {
#pragma unroll
    for (int p = 0; p < 4; ++p) nx[p] = *reinterpret_cast<const uint4*>(xrow + f_k * 128 + p * 8);
  };
  if (f_item < a.items) fetch_x();
  for (int item = blockIdx.x; item < a.items; item += gridDim.x) {
    float y[4][4];
#pragma unroll
    for (int st = 0; st < 4; ++st)
#pragma unroll
      for (int i = 0; i < 4; ++i) y[st][i] = 0.f;
    while (f_item == item) {
      uint4 b[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) b[p] = nx[p];
      // ---- what comes next
      f_k += warps;
      src += size_t(warps) * kW4ChunkBytes;
      ssz += size_t(warps) * kW4ChunkBytes;
      if (f_k >= f_end) {
        f_item += gridDim.x;
        seek();
      }
      const bool more = f_item < a.items;
      if (more) fetch_x();
      float sum[4];
      constexpr uint32_t one = 0x3c003c00u;
      small_mma0(sum, one, one, one, one, b[0].x, b[0].z);
      small_mma(sum, one, one, one, one, b[0].y, b[0].w);
#pragma unroll
      for (int p = 1; p < 4; ++p) {
        small_mma(sum, one, one, one, one, b[p].x, b[p].z);
        small_mma(sum, one, one, one, one, b[p].y, b[p].w);
      }
#pragma unroll
      for (int st = 0; st < 4; ++st) {
        float lo[4], hi[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const uint32_t u = p == 0 ? w[2 * st].x : p == 1 ? w[2 * st].y : p == 2 ? w[2 * st].z : w[2 * st].w;
          const uint32_t v =
              p == 0 ? w[2 * st + 1].x : p == 1 ? w[2 * st + 1].y : p == 2 ? w[2 * st + 1].z : w[2 * st + 1].w;
          const uint32_t u8 = u >> 8, v8 = v >> 8;
          constexpr uint32_t ml = 0x000f000fu, mh = 0x00f000f0u;
          if (p == 0) {
            small_mma0(lo, u & ml, v & ml, u8 & ml, v8 & ml, b[p].x, b[p].z);
            small_mma0(hi, u & mh, v & mh, u8 & mh, v8 & mh, b[p].y, b[p].w);
          } else {
            small_mma(lo, u & ml, v & ml, u8 & ml, v8 & ml, b[p].x, b[p].z);
            small_mma(hi, u & mh, v & mh, u8 & mh, v8 & mh, b[p].y, b[p].w);
          }
        }
        const float2 p0 = __half22float2(*reinterpret_cast<const __half2*>(&sz[2 * st]));
        const float2 p1 = __half22float2(*reinterpret_cast<const __half2*>(&sz[2 * st + 1]));
        const float l0 = p0.x * 16777216.f, l1 = p1.x * 16777216.f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          y[st][i] = fmaf(l0, fmaf(hi[i], 0.0625f, lo[i]), fmaf(p0.y, sum[i], y[st][i]));
          y[st][2 + i] = fmaf(l1, fmaf(hi[2 + i], 0.0625f, lo[2 + i]), fmaf(p1.y, sum[i], y[st][2 + i]));
        }
        if (more) fetch(st);                                   // into the registers that were just used up
      }
      if (more) fetch_scales();
    }
    // ---- add the warps' sums
    float* mine = red + warp * 8 * kSmallPitch;
#pragma unroll
    for (int st = 0; st < 4; ++st)
#pragma unroll
      for (int i = 0; i < 4; ++i) mine[(2 * t + (i & 1)) * kSmallPitch + st * 16 + g + (i >> 1) * 8] = y[st][i];
    __syncthreads();
    auto total = [&](int col, int row) {
      float s = 0.f;
      for (int i = 0; i < warps; ++i) s += red[(i * 8 + col) * kSmallPitch + row];
      return s;
    };
    // sums of a thread's outputs (rows j and 32 + j together where the epilogue needs both) that are not finite are noted
    // for the end, so that the loop carries no registers for them
    if (kPairs) {
      for (int e = threadIdx.x; e < a.M * 32; e += blockDim.x) {
        const int tok = e >> 5, j = e & 31;
        const float va = total(tok, j), vb = total(tok, 32 + j);
        if (!(fabsf(va) + fabsf(vb) <= kMaxFloat)) atomicOr(&odd_tokens, 1u << tok);
        store2(item, tok, j, va, vb);
      }
    } else {
      for (int e = threadIdx.x; e < a.M * 64; e += blockDim.x) {
        const int tok = e >> 6, row = e & 63;
        const float s = total(tok, row);
        if (!(fabsf(s) <= kMaxFloat)) atomicOr(&odd_tokens, 1u << tok);
        store1(item, tok, row, s);
      }
    }
    __syncthreads();
  }
  if (odd_tokens == 0) return;
#pragma unroll 1
  for (int item = blockIdx.x; item < a.items; item += gridDim.x) {
    const int z = item / a.n_half, half = item - z * a.n_half, k0 = z * a.spp, groups = min(a.k_stages, k0 + a.spp) - k0;
    const uint8_t* chunk = a.w + (size_t(half >> 1) * a.k_stages + k0) * kW4ChunkBytes;
    constexpr int rows = kPairs ? 32 : 64;
#pragma unroll 1
    for (int e = threadIdx.x; e < a.M * rows; e += blockDim.x) {
      const int tok = e / rows, row = e % rows;
      if (((odd_tokens >> tok) & 1) == 0) continue;
      const __half* x = a.x + size_t(tok) * a.K + k0 * kW4StageK;
      const int r = (half & 1) * 32 + (row < 32 ? row : row + 32);
      const float va = small_not_finite(chunk, r, groups, x);
      if (kPairs) {
        const float vb = small_not_finite(chunk, r + 64, groups, x);
        if (!(fabsf(va) + fabsf(vb) <= kMaxFloat)) store2(item, tok, row, va, vb);
      } else if (!(fabsf(va) <= kMaxFloat)) {
        store1(item, tok, row, va);
      }
    }
  }
}

// ---- host side -------------------------------------------------------------------------------------------------------------
static int small_sms() {
  static int sms[kMaxDevices] = {};
  const int d = current_device_slot();
  if (sms[d] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || n <= 0) n = 148;
    sms[d] = n;
  }
  return sms[d];
}

static int small_tiles(int N, int epilogue) {
  return epilogue == kEpiSwiGLU ? (N / 2 + 63) / 64 : (N + kTileN - 1) / kTileN;
}

// K splits: half tiles alone leave SMs without work in narrow layers, so where planes are allowed K is cut until there are
// about two CTAs an SM, but into no fewer than six groups.
int gemm_w4_small_planes(int N, int K, int want_split) {
  const int n_half = 2 * small_tiles(N, kEpiPartialF32), k_stages = K / kW4StageK;
  int ks = want_split > 0 ? want_split : 2 * small_sms() / n_half;
  ks = max(1, min(ks, min(8, want_split > 0 ? k_stages : max(1, k_stages / 6))));
  const int spp = (k_stages + ks - 1) / ks;
  return (k_stages + spp - 1) / spp;                           // no empty split
}

// Epilogues that need the whole sum have no K splits here, so the time of a narrow layer goes with its depth alone (1.7 us and 0.9 a
// thousand columns), while a cluster along K (gemm_w4.cu) or the split plan of gemm_w4_dec.cu has more CTAs for it.  Measured (B200,
// weights from memory, 4 tokens; here | cluster | split plan, us): 8 tiles of 4096: 5.5 | 6.2 | 6.0, of 8192: 9.0 | 7.9 | 8.6;
// 16 of 5632: 7.3 | 7.6 | 8.2, of 8192: 9.0 | 8.6 | 9.5, of 16384: 16.0 | 12.7 | 15.1; 28 of 4096 (Gemma-2 9B o_proj): 5.7 | 7.5 | 7.8, of
// 10240: 11.1 | 11.2 | 11.9, of 14336 (down_proj): 14.6 | 13.4 | 14.7; 32 of 14336: 14.6 | 14.1 | 17.5; 36 of 21504: 20.9 | 28 | 24; 40
// of 13824: 14.5 | 19.2 | 17.4.  More than 32 tiles have no room for clusters of eight at once.
bool gemm_w4_small_takes(int M, int N, int K, int epilogue, bool split_plan) {
  if (g_w4_mode != 0 || M < 1 || M > 8 || K <= 0 || K % kW4StageK != 0) return false;
  if (epilogue == kEpiPartialF32) return true;
  const int tiles = small_tiles(N, epilogue), k_stages = K / kW4StageK;
  return split_plan ? tiles > 28 || k_stages <= 33 + 3 * tiles : tiles > 32 || k_stages * (57 - tiles) <= 2400;
}

// These CTAs start while the attention kernel and others with most of an SM's shared memory still run, and fetch their weights
// meanwhile.  That needs an SM whose split between shared memory and L1 suits both: left to the driver's choice the launch waits
// until SMs are empty.  Anything from 25 to 75 % avoids it (100 % does not), and the L1 serves the activations of 8 tokens: 7168 x 14336,
// fp16, 16.3 us at 25 % and 17.1 at 50.  7B steps, driver's choice -> 25 %: one sequence of 517 tokens 1820 -> 1710 us, of 4000
// 1950 -> 1808, 8 of 517 2090 -> 1872.
constexpr int kSmallCarveout = 25;

template <int EPI>
static int launch_small(const SmallArgs& a, cudaStream_t st) {
  static bool attr_done[kMaxDevices] = {};
  const int dev = current_device_slot();
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(gemm_w4_small_kernel<EPI>, cudaFuncAttributePreferredSharedMemoryCarveout, kSmallCarveout) !=
        cudaSuccess)
      return ZSE_ERR_LAUNCH;
    attr_done[dev] = true;
  }
  const int sms = small_sms();
  const bool two = a.items > sms;
  const int threads = two ? kSmallThreads / 2 : kSmallThreads;
  return launch_pdl(gemm_w4_small_kernel<EPI>, dim3(min(a.items, two ? 2 * sms : sms)), dim3(threads),
                    size_t(threads / 32) * 8 * kSmallPitch * 4, st, a) == cudaSuccess
             ? 0
             : ZSE_ERR_LAUNCH;
}

int gemm_w4_small_run(const void* w_tiled, const void* x, const void* bias, void* out, int M, int N, int K, int ldo,
                      int epilogue, int want_split, const SmallRope* rope, cudaStream_t st) {
  if (M < 1 || M > 8 || K <= 0 || K % kW4StageK != 0 || N <= 0) return ZSE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w_tiled) & 15)) return ZSE_ERR_ALIGN;
  const int k_stages = K / kW4StageK, n_half = 2 * small_tiles(N, epilogue);
  const int ks = epilogue == kEpiPartialF32 ? gemm_w4_small_planes(N, K, want_split) : 1;
  SmallArgs a{reinterpret_cast<const uint8_t*>(w_tiled), reinterpret_cast<const __half*>(x),
              reinterpret_cast<const __half*>(bias), out, M, N, K, ldo, k_stages, (k_stages + ks - 1) / ks, n_half,
              n_half * ks, rope != nullptr ? *rope : SmallRope{}};
  switch (epilogue) {
    case kEpiF16: return launch_small<kEpiF16>(a, st);
    case kEpiSwiGLU: return launch_small<kEpiSwiGLU>(a, st);
    case kEpiPartialF32: return launch_small<kEpiPartialF32>(a, st);
    case kEpiQkvRope: return launch_small<kEpiQkvRope>(a, st);
    default: return ZSE_ERR_SHAPE;
  }
}

}  // namespace zse
