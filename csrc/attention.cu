// Attention over the paged fp16 KV cache.
//
// Cache layout per layer: [num_blocks][2 (K, V)][nkv][block_size][hd]; block_size is a multiple of 16, so a
// 16-token tile of one kv head is a contiguous hd*32-byte run.  Block id -1 in a block table is a hole left by
// eviction and is skipped, as in the reference (zse-engine/zse_engine/orchestrator/kernels.py:571,653).
//
// attn_decode_kernel  - one query token per sequence.  K and V are read once per kv head for all G = nh/nkv query heads (the
//                       reference reads them once per query head, kernels.py:524-671).  One grid of as many CTAs as fit; each
//                       takes an equal run of 16-token tiles over all sequences and kv heads, its four warps
//                       stream tiles through private 3-stage cp.async rings that run on from one item into the next (no CTA
//                       barriers in the main loop), keep an online softmax in registers and give it to shared memory at the end
//                       of an item, where all threads add it up.
// attn_prefill_kernel - causal attention of a chunk of query tokens against everything already in the cache
//                       (earlier chunks included), flash-attention style: 64 query rows per CTA, 64-token KV tiles,
//                       online softmax.  Serves prefill, chunked prefill and speculative verification
//                       (replaces kernels.py:859-957, which only sees the current pass).
#include "api.h"
#include "common.cuh"

namespace zse {

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

constexpr int kDecWarps = 4;
constexpr float kLog2e = 1.4426950408889634f;

// Shared-memory tile: `rows` rows of HD halfs; 16-byte chunk c of row r lives at chunk (c ^ (r & 7)).
template <int HD>
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
  return uint32_t(row * (HD * 2) + ((chunk ^ (row & 7)) << 4));
}

// ---- decode: how the work is cut -------------------------------------------------------------------------------------------
// All 16-token tiles of all (sequence, kv head) items stand in one line, sequence by sequence.  With num_splits > 2 every CTA
// takes the same number of them, `per`, whatever items they belong to; an item that lies in several CTAs is merged from scratch
// by attn_combine_kernel (at most num_splits - 1 pieces: `per` is raised for that if one sequence is very long).  The last of a
// head's num_splits records in scratch says how many pieces there are.  That leaves nothing for two pieces, so with num_splits = 2
// every item is cut in two halves; with 1 items stay whole.
constexpr int kDecStages = 3;                                     // of a warp's ring
// Where a warp's O goes when its item is merged: to a place of its own, or to the slot of its last tile, which lets one more CTA
// onto an SM where there would be no room for it (HD = 64; NB = 2), but no warp may fetch on before all have read it (2 % where the
// CTAs are the same).
template <int HD, int NB>
constexpr bool kOwnPlace = NB == 1 && HD >= 128;
__device__ __forceinline__ int seq_tiles(int len, int window) {
  return ((len + 15) >> 4) - ((window > 0 ? max(0, len - window) : 0) >> 4);
}
__device__ __forceinline__ int tiles_per_cta(int total, int longest, int ctas, int num_splits) {
  return max(kDecWarps, max((total + ctas - 1) / ctas, (longest + num_splits - 3) / (num_splits - 2)));
}
__device__ __forceinline__ int* piece_count(float* scratch, int row, int num_splits, int hd) {
  return reinterpret_cast<int*>(scratch + (size_t(row + 1) * num_splits - 1) * (hd + 2));
}
// 2^x in one instruction: scores below the maximum, so the range handling of exp2f() is not needed
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// EXT adds what the Gemma family needs: scores soft-capped as cap*tanh(s/cap) and a sliding window (only the last
// `window` tokens are seen).  The cache is addressed through strides (block, K->V), so a layer may be a view into a
// pool with wider rows.  NB: blocks of eight query heads per kv head.
//
// Tokens are the 16 rows of the products and query heads their 8 columns (S^T = K Q^T, O^T = V^T P^T; the probabilities change
// sides with movmatrix).  With heads as the rows, half of every product, every exponential and half of the accumulators were for
// heads that do not exist (groups of 2 to 8): 385 instructions a tile and 164 registers.
//
// With few sequences a launch is all start and end, and in a layer the instructions come from the L2 every time.  So everything but
// the tile itself is kept short: one form of the cursors for any number of sequences (in lanes, no shared memory), loops that
// stay loops, and one merge by all threads instead of two rounds between warps (60 KB of instructions before, 35 now).  One 7B
// sequence of 517 / 4000 tokens: 8.5 -> 7.5 / 12.9 -> 11.0 us with the merge of the pieces; 17 of 100 to 3000: 18.6 -> 16.9 us;
// 14B, 64 of 128 to 2300: 69.6 -> 59.2 us cut, 57.1 -> 55.2 whole.
template <int HD, bool EXT, int NB>
__global__ void __launch_bounds__(kDecWarps * 32)
attn_decode_kernel(const __half* __restrict__ q, int ldq, const __half* __restrict__ kv, const int* __restrict__ bt,
                   int max_blocks, const int* __restrict__ seq_lens, __half* __restrict__ out, int ldo,
                   float* __restrict__ scratch, int num_seqs, int nh, int nkv, int block_size, int block_shift,
                   int num_splits, float scale_log2, long long blk_stride, long long half_stride, float softcap, int window) {
  constexpr int kTileBytes = 16 * HD * 2;              // one 16-token K (or V) tile
  constexpr int kChunksPerRow = HD / 8;
  constexpr int kSteps = HD / 16;
  constexpr int kHeads = 8 * NB;
  constexpr int kSlotBytes = 2 * kTileBytes;           // K and V
  constexpr bool kOwn = kOwnPlace<HD, NB>;
  constexpr int kPitch = kOwn ? HD + 4 : HD;           // floats per head of a warp's O
  constexpr int kGiven = kHeads * kPitch;
  static_assert(kOwn || kGiven * 4 <= kSlotBytes, "O fits a slot");
  extern __shared__ __align__(128) uint8_t smem[];
  struct Given {                                       // behind the rings, per warp: m, l, where O is
    float m[kHeads], l[kHeads];
    int slot;
  };
  Given* given = reinterpret_cast<Given*>(smem + kDecWarps * kDecStages * kSlotBytes);
  float* own = reinterpret_cast<float*>(given + kDecWarps);
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  const int G = nh / nkv;
  auto tiles_of = [&](int i) { return seq_tiles(seq_lens[i], EXT ? window : 0); };
  const bool fixed = num_splits < 3;                   // CTA i has item i, or one half of item i / 2
  int p_begin = blockIdx.x, p_end = p_begin + 1, per = 1;
  if (!fixed) {
    int total = 0, longest = 0;
    for (int i = lane; i < num_seqs; i += 32) {
      const int n = tiles_of(i);
      total += n * nkv;
      longest = max(longest, n);
    }
    total = __reduce_add_sync(0xffffffffu, total);
    longest = __reduce_max_sync(0xffffffffu, longest);
    per = tiles_per_cta(total, longest, gridDim.x, num_splits);
    p_begin = min(total, int(blockIdx.x) * per);
    p_end = min(total, p_begin + per);
  }

  // 32 neighbouring sequences in the lanes of a warp: tiles of sequence base + lane, and the position behind its last item.  No
  // shared memory and no barriers; a cursor only moves forward.
  struct Window {
    int base, n, behind, end;
  };
  auto move_to = [&](Window& w, int p) {               // to the window that position p lies in
    while (p >= w.end) {
      w.base += 32;
      w.n = w.base + lane < num_seqs ? tiles_of(w.base + lane) : 0;
      w.behind = w.n * nkv;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, w.behind, o);
        if (lane >= o) w.behind += u;
      }
      w.behind += w.end;
      w.end = __shfl_sync(0xffffffffu, w.behind, 31);
    }
  };
  struct Seg {
    int seq, kvh, first, n, tiles;                     // tiles first .. first + n - 1 of `tiles` of the item
  };
  // the segment at position p (p < p_end), and the position behind it; the whole warp calls it
  auto segment = [&](int p, Window& w, Seg& sg) {
    if (fixed) {
      const int item = p >> (num_splits - 1);
      sg.seq = unsigned(item) / unsigned(nkv), sg.kvh = item - sg.seq * nkv;
      sg.tiles = tiles_of(sg.seq);
      const int part = (sg.tiles + num_splits - 1) >> (num_splits - 1);
      sg.first = num_splits == 2 && (p & 1) ? part : 0;
      sg.n = min(part, sg.tiles - sg.first);
      return p + 1;
    }
    move_to(w, p);
    const int at = __popc(__ballot_sync(0xffffffffu, w.behind <= p));
    sg.seq = w.base + at;
    sg.tiles = __shfl_sync(0xffffffffu, w.n, at);
    const int in = p - (__shfl_sync(0xffffffffu, w.behind, at) - sg.tiles * nkv);
    sg.kvh = unsigned(in) / unsigned(sg.tiles);
    sg.first = in - sg.kvh * sg.tiles;
    sg.n = min(sg.tiles - sg.first, p_end - p);
    return p + sg.n;
  };

  // ---- this warp's tiles, one after the other over all segments: what is fetched next
  uint8_t* ring = smem + warp * (kDecStages * kSlotBytes);
  Window fw{-32, 0, 0, 0};
  if (p_begin < p_end && !fixed) move_to(fw, p_begin);
  Window cw = fw;
  Seg fs{};
  int fp = p_begin, fi = 0, f_tile0 = 0;
  uint32_t holes = 0;                                  // bit = ring slot whose tile lies in a dropped block
  auto issue = [&](int slot) {                         // next tile -> ring slot; always commits a group
    while (fi >= fs.n && fp < p_end) {                 // on to a segment with a tile for this warp
      fp = segment(fp, fw, fs);
      fi = warp;
      f_tile0 = (EXT && window > 0 ? max(0, seq_lens[fs.seq] - window) >> 4 : 0) + fs.first;
    }
    holes &= ~(1u << slot);
    if (fi < fs.n) {
      const int tile = f_tile0 + fi;
      const int bi = block_shift >= 0 ? tile >> block_shift : tile / (block_size >> 4);
      const int in = tile - bi * (block_size >> 4);
      const int blk = bt[size_t(fs.seq) * max_blocks + bi];
      if (blk >= 0) {
        const __half* ksrc = kv + size_t(blk) * blk_stride + (size_t(fs.kvh) * block_size + in * 16) * HD + lane * 8;
        const __half* vsrc = ksrc + half_stride;
        uint8_t* kd = ring + slot * kSlotBytes;
#pragma unroll
        for (int j = 0; j < kTileBytes / 512; ++j) {
          const int idx = j * 32 + lane;
          const uint32_t off = tile_off<HD>(idx / kChunksPerRow, idx % kChunksPerRow);
          cp_async16(kd + off, ksrc + j * 256);
          cp_async16(kd + kTileBytes + off, vsrc + j * 256);
        }
      } else {
        holes |= 1u << slot;
      }
      fi += kDecWarps;
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int i = 0; i < kDecStages - 1; ++i) issue(i);

  int slot = 0;
  for (int p = p_begin; p < p_end;) {
    Seg sg;
    const int here = p;
    p = segment(p, cw, sg);
    if (sg.n == 0 && num_splits == 1) continue;        // (an empty sequence; an empty half still has a record)
    const int len = seq_lens[sg.seq];
    const int first_tok = EXT && window > 0 ? max(0, len - window) : 0;
    uint32_t qb[NB][kSteps][2];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int h = nb * 8 + g;
      const __half* src = q + size_t(sg.seq) * ldq + size_t(sg.kvh * G + h) * HD + t2;
#pragma unroll
      for (int kk = 0; kk < kSteps; ++kk) {
        qb[nb][kk][0] = h < G ? *reinterpret_cast<const uint32_t*>(src + kk * 16) : 0u;
        qb[nb][kk][1] = h < G ? *reinterpret_cast<const uint32_t*>(src + kk * 16 + 8) : 0u;
      }
    }
    float o[NB][kSteps][4], m[NB][2], l[NB][2];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      m[nb][0] = m[nb][1] = -INFINITY;
      l[nb][0] = l[nb][1] = 0.f;
#pragma unroll
      for (int d = 0; d < kSteps; ++d) o[nb][d][0] = o[nb][d][1] = o[nb][d][2] = o[nb][d][3] = 0.f;
    }
    for (int i = warp; i < sg.n; i += kDecWarps) {
      cp_async_wait<kDecStages - 2>();
      __syncwarp();
      const bool hole = (holes >> slot) & 1u;
      issue(slot == 0 ? kDecStages - 1 : slot - 1);    // the slot of the tile before this one
      const uint32_t kbase = smem_u32(ring + slot * kSlotBytes), vbase = kbase + kTileBytes;
      slot = slot + 1 == kDecStages ? 0 : slot + 1;
      if (hole) continue;
      const int tok = ((first_tok >> 4) + sg.first + i) << 4;
      const int mm = lane >> 3, rr = lane & 7;
      float s[NB][2][4];                               // even and odd K steps apart: two chains
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[nb][0][e] = s[nb][1][e] = 0.f;
#pragma unroll
      for (int kk = 0; kk < kSteps; ++kk) {
        uint32_t a[4];
        ldsm_x4(kbase + tile_off<HD>((mm & 1) * 8 + rr, kk * 2 + (mm >> 1)), a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) mma16816(s[nb][kk & 1], a, qb[nb][kk][0], qb[nb][kk][1]);
      }
      const bool dead0 = tok + g >= len || (EXT && tok + g < first_tok);
      const bool dead1 = tok + g + 8 >= len || (EXT && tok + g + 8 < first_tok);
      uint32_t pb[NB][2];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[e] = (s[nb][0][e] + s[nb][1][e]) * scale_log2;
          if constexpr (EXT) {
            if (softcap > 0.f) v[e] = softcap * kLog2e * tanhf(v[e] * (1.f / (kLog2e * softcap)));
          }
          if (e < 2 ? dead0 : dead1) v[e] = -INFINITY;
        }
        float x0 = fmaxf(v[0], v[2]), x1 = fmaxf(v[1], v[3]);       // heads t2, t2 + 1
#pragma unroll
        for (int sh = 4; sh < 32; sh <<= 1) {
          x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, sh));
          x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, sh));
        }
        const float n0 = fmaxf(m[nb][0], x0), n1 = fmaxf(m[nb][1], x1);
        if (__any_sync(0xffffffffu, n0 > m[nb][0] || n1 > m[nb][1])) {
          const float a0 = m[nb][0] == -INFINITY ? 0.f : ex2_approx(m[nb][0] - n0);
          const float a1 = m[nb][1] == -INFINITY ? 0.f : ex2_approx(m[nb][1] - n1);
          l[nb][0] *= a0;
          l[nb][1] *= a1;
#pragma unroll
          for (int d = 0; d < kSteps; ++d) {
            o[nb][d][0] *= a0; o[nb][d][1] *= a1; o[nb][d][2] *= a0; o[nb][d][3] *= a1;
          }
          m[nb][0] = n0;
          m[nb][1] = n1;
        }
        const float b0 = m[nb][0] == -INFINITY ? 0.f : m[nb][0], b1 = m[nb][1] == -INFINITY ? 0.f : m[nb][1];
        const float p00 = ex2_approx(v[0] - b0), p01 = ex2_approx(v[1] - b1), p10 = ex2_approx(v[2] - b0),
                    p11 = ex2_approx(v[3] - b1);
        l[nb][0] += p00 + p10;
        l[nb][1] += p01 + p11;
        pb[nb][0] = transpose_8x8(pack_h2(p00, p01));  // tokens 0..7: [token][head] -> [head][token], the B operand
        pb[nb][1] = transpose_8x8(pack_h2(p10, p11));
      }
#pragma unroll
      for (int d = 0; d < kSteps; ++d) {
        uint32_t a[4];
        ldsm_x4_t(vbase + tile_off<HD>((mm >> 1) * 8 + rr, d * 2 + (mm & 1)), a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) mma16816(o[nb][d], a, pb[nb][0], pb[nb][1]);
      }
    }
    // ---- the four warps give what they have, all threads add it up
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int sh = 4; sh < 32; sh <<= 1) l[nb][e] += __shfl_xor_sync(0xffffffffu, l[nb][e], sh);
    // (conflict-free: heads four banks apart, or bits 3 and 4 of a column turned by the head)
    const int mine = slot == 0 ? kDecStages - 1 : slot - 1;      // the slot of the last tile
    if (kOwn) __syncthreads(); else __syncwarp();                // (own places: the item before has been read)
    float* to = kOwn ? own + warp * kGiven : reinterpret_cast<float*>(ring + mine * kSlotBytes);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int h = nb * 8 + t2 + e, turn = kOwn ? 0 : (h & 6) << 2;
#pragma unroll
        for (int d = 0; d < kSteps; ++d) {
          to[h * kPitch + ((d * 16 + g) ^ turn)] = o[nb][d][e];
          to[h * kPitch + ((d * 16 + g + 8) ^ turn)] = o[nb][d][2 + e];
        }
        if (g == 0) {
          given[warp].m[h] = m[nb][e];
          given[warp].l[h] = l[nb][e];
        }
      }
    if (!kOwn && lane == 0) given[warp].slot = mine;
    __syncthreads();
    const int start = here - sg.first;                           // position of the item's first tile
    const int pieces = fixed ? num_splits : (start + sg.tiles - 1) / per - start / per + 1;
    const bool alone = pieces == 1;
    const int piece = fixed ? int(blockIdx.x) & 1 : int(blockIdx.x) - start / per;
    if (!fixed && sg.first == 0 && threadIdx.x < G)
      *piece_count(scratch, sg.seq * nh + sg.kvh * G + threadIdx.x, num_splits, HD) = pieces;
    constexpr int kPart = HD / 4;                                // a thread: four elements this far apart
#pragma unroll 1
    for (int idx = threadIdx.x; idx < G * kPart; idx += kDecWarps * 32) {
      const int h = idx / kPart, d = idx % kPart, head = sg.kvh * G + h;
      float mw[kDecWarps], M = -INFINITY, L = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) M = fmaxf(M, mw[w] = given[w].m[h]);
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) {
        const float* src =
            (kOwn ? own + w * kGiven : reinterpret_cast<const float*>(smem + (w * kDecStages + given[w].slot) * kSlotBytes)) +
            h * kPitch;
        const float f = mw[w] == -INFINITY ? 0.f : ex2_approx(mw[w] - M);
        L += given[w].l[h] * f;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] += src[(d + k * kPart) ^ (kOwn ? 0 : (h & 6) << 2)] * f;
      }
      if (alone) {
        __half* dst = out + size_t(sg.seq) * ldo + size_t(head) * HD + d;
        const float inv = L > 0.f ? 1.f / L : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) dst[k * kPart] = __float2half_rn(L > 0.f ? acc[k] * inv : 0.f);
      } else {
        float* dst = scratch + (size_t(sg.seq * nh + head) * num_splits + piece) * (HD + 2);
#pragma unroll
        for (int k = 0; k < 4; ++k) dst[d + k * kPart] = acc[k];
        if (d == 0) {
          dst[HD] = M;
          dst[HD + 1] = L;
        }
      }
    }
    if (!kOwn) __syncthreads();
  }
  cp_async_wait<0>();
  for (int i = blockIdx.x; i < num_seqs; i += gridDim.x)         // sequences of nothing: zeros
    if (tiles_of(i) == 0) {
      for (int d = threadIdx.x; d < nh * HD; d += blockDim.x) out[size_t(i) * ldo + d] = __float2half_rn(0.f);
      if (!fixed)
        for (int h = threadIdx.x; h < nh; h += blockDim.x) *piece_count(scratch, i * nh + h, num_splits, HD) = 1;
    }
}

// Items that attn_decode_kernel cut in pieces (num_splits > 1).  grid (nh, sequences), HD threads.
template <int HD>
__global__ void attn_combine_kernel(float* __restrict__ scratch, __half* __restrict__ out, int ldo, int nh, int num_splits) {
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.x, seq = blockIdx.y, d = threadIdx.x;
  const float* src = scratch + size_t(seq * nh + head) * num_splits * (HD + 2);
  // what a few pieces need is read beside their number, not behind it (places that exist, whatever they hold); lane s has the
  // maximum and the sum of piece s
  const int lane = threadIdx.x & 31, some = max(2, num_splits - 1);
  const int pieces = num_splits == 2 ? 2 : *piece_count(scratch, seq * nh + head, num_splits, HD);
  float m = lane < some ? src[lane * (HD + 2) + HD] : -INFINITY, l = lane < some ? src[lane * (HD + 2) + HD + 1] : 0.f;
  float o[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) o[s] = s < some ? src[s * (HD + 2) + d] : 0.f;
  if (pieces == 1) return;                             // its CTA stored it
  __half* dst = out + size_t(seq) * ldo + size_t(head) * HD + d;
  if (pieces > 32) {
    float M = -INFINITY, L = 0.f, acc = 0.f;
    for (int s = 0; s < pieces; ++s) M = fmaxf(M, src[s * (HD + 2) + HD]);
    for (int s = 0; s < pieces; ++s) {
      const float ms = src[s * (HD + 2) + HD], f = ms == -INFINITY ? 0.f : ex2_approx(ms - M);
      L += src[s * (HD + 2) + HD + 1] * f;
      acc += src[s * (HD + 2) + d] * f;
    }
    *dst = __float2half_rn(L > 0.f ? acc / L : 0.f);
    return;
  }
  m = lane < pieces ? m : -INFINITY;
  float M = m;
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, sh));
  const float f = m == -INFINITY ? 0.f : ex2_approx(m - M);
  float L = lane < pieces ? l * f : 0.f;
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) L += __shfl_xor_sync(0xffffffffu, L, sh);
  float acc = 0.f;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const float fs = __shfl_sync(0xffffffffu, f, s);
    if (s < pieces) acc += o[s] * fs;
  }
#pragma unroll 4
  for (int s = 4; s < pieces; ++s) acc += src[s * (HD + 2) + d] * __shfl_sync(0xffffffffu, f, s);
  *dst = __float2half_rn(L > 0.f ? acc / L : 0.f);
}

// ---- prefill / chunked prefill / verify ----------------------------------------------------------------
constexpr int kPfWarps = 4;          // 16 query rows each -> 64 query rows per CTA
constexpr int kPfKvTile = 64;

template <int HD, bool EXT>
__global__ void __launch_bounds__(kPfWarps * 32)
attn_prefill_kernel(const __half* __restrict__ q, int ldq, const __half* __restrict__ kv, const int* __restrict__ bt,
                    int max_blocks, const int* __restrict__ cu_q, const int* __restrict__ q_pos0,
                    __half* __restrict__ out, int ldo, int nh, int nkv, int block_size, float scale_log2,
                    long long blk_stride, long long half_stride, float softcap, int window) {
  constexpr int kChunksPerRow = HD / 8;
  constexpr int kKSteps = HD / 16;
  constexpr int kNTilesO = HD / 8;
  constexpr int kTileBytes = kPfKvTile * HD * 2;
  extern __shared__ __align__(128) uint8_t smem[];       // [2 stages][K tile, V tile]
  const int qt = blockIdx.x, head = blockIdx.y, seq = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_begin = cu_q[seq], q_len = cu_q[seq + 1] - q_begin;
  if (qt * 64 >= q_len) return;
  const int pos0 = q_pos0[seq];
  const int kvh = head / (nh / nkv);
  const int* my_bt = bt + size_t(seq) * max_blocks;
  const size_t kv_head_stride = size_t(block_size) * HD;

  // this warp's 16 query rows
  const int r0 = qt * 64 + warp * 16 + (lane >> 2), r1 = r0 + 8;       // row index inside the sequence's chunk
  uint32_t qa[kKSteps][4];
  {
    const int c = (lane & 3) * 2;
    const __half* q0 = q + size_t(q_begin + r0) * ldq + size_t(head) * HD;
    const __half* q1 = q + size_t(q_begin + r1) * ldq + size_t(head) * HD;
#pragma unroll
    for (int kk = 0; kk < kKSteps; ++kk) {
      qa[kk][0] = r0 < q_len ? *reinterpret_cast<const uint32_t*>(q0 + kk * 16 + c) : 0u;
      qa[kk][1] = r1 < q_len ? *reinterpret_cast<const uint32_t*>(q1 + kk * 16 + c) : 0u;
      qa[kk][2] = r0 < q_len ? *reinterpret_cast<const uint32_t*>(q0 + kk * 16 + 8 + c) : 0u;
      qa[kk][3] = r1 < q_len ? *reinterpret_cast<const uint32_t*>(q1 + kk * 16 + 8 + c) : 0u;
    }
  }
  // keys visible to the last query row of this CTA
  const int last_row = min(q_len, qt * 64 + 64) - 1;
  const int kv_len = pos0 + last_row + 1;
  const int n_tiles = (kv_len + kPfKvTile - 1) / kPfKvTile;

  auto issue = [&](int t) {
    if (t < n_tiles) {
      uint8_t* kd = smem + (t & 1) * 2 * kTileBytes;
      uint8_t* vd = kd + kTileBytes;
      // 64 rows x kChunksPerRow chunks, split over 128 threads
      for (int idx = threadIdx.x; idx < kPfKvTile * kChunksPerRow; idx += kPfWarps * 32) {
        const int row = idx / kChunksPerRow, ch = idx % kChunksPerRow;
        const int tok = t * kPfKvTile + row;
        const int blk = tok < kv_len ? my_bt[tok / block_size] : -1;
        if (blk >= 0) {
          const __half* ksrc = kv + size_t(blk) * blk_stride + size_t(kvh) * kv_head_stride +
                               size_t(tok % block_size) * HD + ch * 8;
          cp_async16(kd + tile_off<HD>(row, ch), ksrc);
          cp_async16(vd + tile_off<HD>(row, ch), ksrc + half_stride);
        } else {
          *reinterpret_cast<uint4*>(kd + tile_off<HD>(row, ch)) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(vd + tile_off<HD>(row, ch)) = make_uint4(0, 0, 0, 0);
        }
      }
    }
    cp_async_commit();
  };

  float o[kNTilesO][4];
#pragma unroll
  for (int n = 0; n < kNTilesO; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  const int p0 = pos0 + r0, p1 = pos0 + r1;              // absolute positions of the two rows

  // first tile any row of this CTA can see (its first row's window start)
  const int t_begin = (EXT && window > 0) ? max(0, pos0 + qt * 64 - window + 1) / kPfKvTile : 0;
  issue(t_begin);
  for (int t = t_begin; t < n_tiles; ++t) {
    issue(t + 1);
    cp_async_wait<1>();
    __syncthreads();
    const uint32_t kbase = smem_u32(smem + (t & 1) * 2 * kTileBytes);
    const uint32_t vbase = kbase + kTileBytes;
    const int tok0 = t * kPfKvTile;
    // skip tiles entirely in the future of this warp's rows (warp-uniform)
    const int warp_last_pos = pos0 + qt * 64 + warp * 16 + 15;
    if (tok0 <= warp_last_pos) {
      float s[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
      {
        const int m = lane >> 3, rr = lane & 7;
#pragma unroll
        for (int kk = 0; kk < kKSteps; ++kk) {
#pragma unroll
          for (int jp = 0; jp < 4; ++jp) {                 // pairs of 8-token n-tiles
            const int row = jp * 16 + (m >> 1) * 8 + rr;
            uint32_t b0, b1, b2, b3;
            ldsm_x4(kbase + tile_off<HD>(row, kk * 2 + (m & 1)), b0, b1, b2, b3);
            mma16816(s[2 * jp], qa[kk], b0, b1);
            mma16816(s[2 * jp + 1], qa[kk], b2, b3);
          }
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // an 8-token group never straddles a block (block_size is a multiple of 16)
        const bool hole = my_bt[min(tok0 + j * 8, kv_len - 1) / block_size] < 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int tk = tok0 + j * 8 + (lane & 3) * 2 + (e & 1);
          const int pos = e < 2 ? p0 : p1;
          float v = s[j][e] * scale_log2;
          if constexpr (EXT) {
            if (softcap > 0.f) v = softcap * kLog2e * tanhf(v * (1.f / (kLog2e * softcap)));
            if (window > 0 && tk <= pos - window) v = -INFINITY;
          }
          if (tk > pos || hole) v = -INFINITY;
          s[j][e] = v;
          if (e < 2) mx0 = fmaxf(mx0, v); else mx1 = fmaxf(mx1, v);
        }
      }
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
      const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
      const float a0 = (m0 == -INFINITY) ? 0.f : exp2f(m0 - n0), a1 = (m1 == -INFINITY) ? 0.f : exp2f(m1 - n1);
      l0 *= a0;
      l1 *= a1;
#pragma unroll
      for (int n = 0; n < kNTilesO; ++n) {
        o[n][0] *= a0; o[n][1] *= a0; o[n][2] *= a1; o[n][3] *= a1;
      }
      m0 = n0;
      m1 = n1;
      const float b0f = m0 == -INFINITY ? 0.f : m0, b1f = m1 == -INFINITY ? 0.f : m1;   // fully masked rows
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {                     // 16 tokens per PV k-step
        uint32_t pa[4];
        const float p00 = exp2f(s[2 * ks][0] - b0f), p01 = exp2f(s[2 * ks][1] - b0f);
        const float p02 = exp2f(s[2 * ks][2] - b1f), p03 = exp2f(s[2 * ks][3] - b1f);
        const float p10 = exp2f(s[2 * ks + 1][0] - b0f), p11 = exp2f(s[2 * ks + 1][1] - b0f);
        const float p12 = exp2f(s[2 * ks + 1][2] - b1f), p13 = exp2f(s[2 * ks + 1][3] - b1f);
        l0 += p00 + p01 + p10 + p11;
        l1 += p02 + p03 + p12 + p13;
        pa[0] = pack_h2(p00, p01);
        pa[1] = pack_h2(p02, p03);
        pa[2] = pack_h2(p10, p11);
        pa[3] = pack_h2(p12, p13);
        const int m = lane >> 3, rr = lane & 7;
        const int row = ks * 16 + (m & 1) * 8 + rr;
#pragma unroll
        for (int p = 0; p < kNTilesO / 2; ++p) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(vbase + tile_off<HD>(row, p * 2 + (m >> 1)), b0, b1, b2, b3);
          mma16816(o[2 * p], pa, b0, b1);
          mma16816(o[2 * p + 1], pa, b2, b3);
        }
      }
    }
    __syncthreads();                                       // tile buffer may be refilled
  }
  cp_async_wait<0>();
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
  l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const float i0 = l0 > 0.f ? 1.f / l0 : 0.f, i1 = l1 > 0.f ? 1.f / l1 : 0.f;
  const int c = (lane & 3) * 2;
#pragma unroll
  for (int n = 0; n < kNTilesO; ++n) {
    if (r0 < q_len)
      *reinterpret_cast<uint32_t*>(out + size_t(q_begin + r0) * ldo + size_t(head) * HD + n * 8 + c) =
          pack_h2(o[n][0] * i0, o[n][1] * i0);
    if (r1 < q_len)
      *reinterpret_cast<uint32_t*>(out + size_t(q_begin + r1) * ldo + size_t(head) * HD + n * 8 + c) =
          pack_h2(o[n][2] * i1, o[n][3] * i1);
  }
}

}  // namespace zse

using namespace zse;

extern "C" int64_t zse_attn_decode_scratch_floats(int num_seqs, int nh, int hd, int max_splits) {
  return int64_t(num_seqs) * nh * max_splits * (hd + 2);
}

// Shared memory of the decode kernel: rings, and what its warps give besides O.
template <int HD, int NB>
constexpr int kDecodeSmem =
    kDecWarps * (kDecStages * 2 * 16 * HD * 2 + (2 * 8 * NB + 1) * 4 + (kOwnPlace<HD, NB> ? 8 * NB * (HD + 4) * 4 : 0));
// CTAs that an SM holds: shared memory decides (228 KB, 1 KB of each CTA's is the system's; 255 registers a thread leave room for two)
template <int HD, int NB>
constexpr int kDecodeCtasPerSm = 228 * 1024 / (kDecodeSmem<HD, NB> + 1024);
static_assert(kDecodeCtasPerSm<64, 1> == 4 && kDecodeCtasPerSm<64, 2> == 4 && kDecodeCtasPerSm<128, 1> == 2 &&
              kDecodeCtasPerSm<128, 2> == 2 && kDecodeCtasPerSm<256, 1> == 1 && kDecodeCtasPerSm<256, 2> == 1);

// The attribute is raised once per device (host work: not a stream operation).
template <int HD, bool EXT, int NB>
static int prepare_decode() {
  static bool attr[kMaxDevices] = {};
  const int dev_slot = current_device_slot();
  if (!attr[dev_slot]) {
    if (cudaFuncSetAttribute(attn_decode_kernel<HD, EXT, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kDecodeSmem<HD, NB>) != cudaSuccess)
      return ZSE_ERR_LAUNCH;
    attr[dev_slot] = true;
  }
  return 0;
}

static int decode_sms() {
  static int sms[kMaxDevices] = {};
  const int d = current_device_slot();
  if (sms[d] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || n <= 0) n = 148;
    sms[d] = n;
  }
  return sms[d];
}

template <int HD, bool EXT, int NB>
static int launch_decode(const void* q, int ldq, const void* kv, const void* bt, int max_blocks, const void* lens,
                         void* out, int ldo, void* scratch, int num_seqs, int nh, int nkv, int block_size, int splits,
                         float scale, long long blk_stride, long long half_stride, float softcap, int window,
                         cudaStream_t st) {
  if (int rc = prepare_decode<HD, EXT, NB>()) return rc;
  const int tpb = block_size / 16;
  int shift = 0;
  while ((1 << shift) < tpb) ++shift;
  if ((1 << shift) != tpb) shift = -1;
  // cut: as many CTAs as the chip holds at once, each with the same share of the tiles (with few sequences most of the chip is left
  // to the next kernel)
  const int fit = decode_sms() * kDecodeCtasPerSm<HD, NB>;
  const int ctas = splits >= 3 ? min(fit, num_seqs * nkv * (splits - 1)) : num_seqs * nkv * splits;
  if (launch_pdl(attn_decode_kernel<HD, EXT, NB>, dim3(ctas), dim3(kDecWarps * 32), size_t(kDecodeSmem<HD, NB>), st,
                 reinterpret_cast<const __half*>(q), ldq, reinterpret_cast<const __half*>(kv), reinterpret_cast<const int*>(bt),
                 max_blocks, reinterpret_cast<const int*>(lens), reinterpret_cast<__half*>(out), ldo,
                 reinterpret_cast<float*>(scratch), num_seqs, nh, nkv, block_size, shift, splits, scale * kLog2e, blk_stride,
                 half_stride, softcap, window) != cudaSuccess)
    return ZSE_ERR_LAUNCH;
  if (splits > 1) {
    if (launch_pdl(attn_combine_kernel<HD>, dim3(nh, num_seqs), dim3(HD), 0, st, reinterpret_cast<float*>(scratch),
                   reinterpret_cast<__half*>(out), ldo, nh, splits) != cudaSuccess)
      return ZSE_ERR_LAUNCH;
  }
  return 0;
}

extern "C" int zse_attn_decode_ext(const void* q, int ldq, const void* kv_layer, int64_t blk_stride,
                                   int64_t half_stride, const void* block_tables, int max_blocks, const void* seq_lens,
                                   void* out, int ldo, void* scratch, int num_seqs, int nh, int nkv, int hd,
                                   int block_size, int num_splits, float scale, float softcap, int window,
                                   void* stream) {
  if (num_seqs <= 0) return 0;
  if (nh % nkv || nh / nkv > 16 || block_size % 16 || num_splits < 1 || softcap < 0.f || window < 0)
    return ZSE_ERR_SHAPE;
  if (num_splits > 1 && scratch == nullptr) return ZSE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(kv_layer) & 15) || (blk_stride & 7) || (half_stride & 7)) return ZSE_ERR_ALIGN;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool ext = softcap > 0.f || window > 0;
#define ZSE_DEC_NB(HD_, EXT_, NB_)                                                                                       \
  return launch_decode<HD_, EXT_, NB_>(q, ldq, kv_layer, block_tables, max_blocks, seq_lens, out, ldo, scratch, num_seqs, \
                                       nh, nkv, block_size, num_splits, scale, blk_stride, half_stride, softcap, window, st)
#define ZSE_DEC(HD_, EXT_)                          \
  {                                                 \
    if (nh / nkv <= 8) ZSE_DEC_NB(HD_, EXT_, 1);    \
    ZSE_DEC_NB(HD_, EXT_, 2);                       \
  }
  if (hd == 128) { if (ext) ZSE_DEC(128, true) ZSE_DEC(128, false) }
  if (hd == 64) { if (ext) ZSE_DEC(64, true) ZSE_DEC(64, false) }
  if (hd == 256) ZSE_DEC(256, true)
#undef ZSE_DEC
#undef ZSE_DEC_NB
  return ZSE_ERR_SHAPE;
}

extern "C" int zse_attn_decode(const void* q, int ldq, const void* kv_layer, const void* block_tables, int max_blocks,
                               const void* seq_lens, void* out, int ldo, void* scratch, int num_seqs, int nh, int nkv,
                               int hd, int block_size, int num_splits, float scale, void* stream) {
  const int64_t half = int64_t(nkv) * block_size * hd;
  return zse_attn_decode_ext(q, ldq, kv_layer, 2 * half, half, block_tables, max_blocks, seq_lens, out, ldo, scratch,
                             num_seqs, nh, nkv, hd, block_size, num_splits, scale, 0.f, 0, stream);
}

template <int HD, bool EXT>
static int launch_prefill(const void* q, int ldq, const void* kv, const void* bt, int max_blocks, const void* cu_q,
                          const void* pos0, void* out, int ldo, int num_seqs, int max_q_len, int nh, int nkv,
                          int block_size, float scale, long long blk_stride, long long half_stride, float softcap,
                          int window, cudaStream_t st) {
  constexpr int smem = 2 * 2 * kPfKvTile * HD * 2;
  static bool attr[kMaxDevices] = {};
  const int dev_slot = current_device_slot();
  if (!attr[dev_slot]) {
    if (cudaFuncSetAttribute(attn_prefill_kernel<HD, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess)
      return ZSE_ERR_LAUNCH;
    attr[dev_slot] = true;
  }
  dim3 grid((max_q_len + 63) / 64, nh, num_seqs);
  attn_prefill_kernel<HD, EXT><<<grid, kPfWarps * 32, smem, st>>>(
      reinterpret_cast<const __half*>(q), ldq, reinterpret_cast<const __half*>(kv), reinterpret_cast<const int*>(bt),
      max_blocks, reinterpret_cast<const int*>(cu_q), reinterpret_cast<const int*>(pos0),
      reinterpret_cast<__half*>(out), ldo, nh, nkv, block_size, scale * kLog2e, blk_stride, half_stride, softcap,
      window);
  return cudaGetLastError() == cudaSuccess ? 0 : ZSE_ERR_LAUNCH;
}

extern "C" int zse_attn_prefill_ext(const void* q, int ldq, const void* kv_layer, int64_t blk_stride,
                                    int64_t half_stride, const void* block_tables, int max_blocks, const void* cu_q,
                                    const void* q_pos0, void* out, int ldo, int num_seqs, int max_q_len, int nh,
                                    int nkv, int hd, int block_size, float scale, float softcap, int window,
                                    void* stream) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  if (nh % nkv || block_size % 16 || softcap < 0.f || window < 0) return ZSE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(kv_layer) & 15) || (blk_stride & 7) || (half_stride & 7)) return ZSE_ERR_ALIGN;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool ext = softcap > 0.f || window > 0;
#define ZSE_PF(HD_, EXT_)                                                                                            \
  return launch_prefill<HD_, EXT_>(q, ldq, kv_layer, block_tables, max_blocks, cu_q, q_pos0, out, ldo, num_seqs,     \
                                   max_q_len, nh, nkv, block_size, scale, blk_stride, half_stride, softcap, window, st)
  if (hd == 128) { if (ext) ZSE_PF(128, true); ZSE_PF(128, false); }
  if (hd == 64) { if (ext) ZSE_PF(64, true); ZSE_PF(64, false); }
  if (hd == 256) ZSE_PF(256, true);
#undef ZSE_PF
  return ZSE_ERR_SHAPE;
}

extern "C" int zse_attn_prefill(const void* q, int ldq, const void* kv_layer, const void* block_tables, int max_blocks,
                                const void* cu_q, const void* q_pos0, void* out, int ldo, int num_seqs, int max_q_len,
                                int nh, int nkv, int hd, int block_size, float scale, void* stream) {
  const int64_t half = int64_t(nkv) * block_size * hd;
  return zse_attn_prefill_ext(q, ldq, kv_layer, 2 * half, half, block_tables, max_blocks, cu_q, q_pos0, out, ldo,
                              num_seqs, max_q_len, nh, nkv, hd, block_size, scale, 0.f, 0, stream);
}

// ---- decode attention with library-owned scratch (attn_decode_static.h) -------------------------------------------
#include "attn_decode_static.h"

static __device__ __align__(256) float g_attn_static_scratch[ZSE_ATTN_STATIC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxStaticDevices = 64;
float* g_static_scratch_ptr[kMaxStaticDevices] = {};

// address of the scratch array on the current device, looked up once per device; nullptr with *err set on failure
float* static_scratch(int* err) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxStaticDevices) {
    *err = ZSE_ERR_DRIVER;
    return nullptr;
  }
  if (g_static_scratch_ptr[dev] == nullptr) {
    float* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_attn_static_scratch) != cudaSuccess || p == nullptr) {
      (void)cudaGetLastError();
      *err = ZSE_ERR_DRIVER;
      return nullptr;
    }
    g_static_scratch_ptr[dev] = p;
  }
  *err = 0;
  return g_static_scratch_ptr[dev];
}
}  // namespace

extern "C" int64_t zse_attn_decode_static_max_floats(void) { return ZSE_ATTN_STATIC_SCRATCH_FLOATS; }

extern "C" int zse_attn_decode_static_setup(void) {
  // everything the first call on a device would otherwise do on the host: the address of the scratch array and the
  // shared-memory attribute of the kernels zse_attn_decode_static can reach (head_dim 64 / 128 / 256)
  int err = 0;
  static_scratch(&err);
  if (err) return err;
  if (int rc = prepare_decode<128, false, 1>()) return rc;
  if (int rc = prepare_decode<128, false, 2>()) return rc;
  if (int rc = prepare_decode<64, false, 1>()) return rc;
  if (int rc = prepare_decode<64, false, 2>()) return rc;
  if (int rc = prepare_decode<256, true, 1>()) return rc;
  return prepare_decode<256, true, 2>();
}

extern "C" int zse_attn_decode_static(const void* q, int ldq, const void* kv_layer, const void* block_tables,
                                      int max_blocks, const void* seq_lens, void* out, int ldo, int num_seqs, int nh,
                                      int nkv, int hd, int block_size, int num_splits, float scale, void* stream) {
  if (num_seqs <= 0) return 0;
  if (num_splits < 1 || nh <= 0 || hd <= 0) return ZSE_ERR_SHAPE;
  if (num_splits > 1 &&
      zse_attn_decode_scratch_floats(num_seqs, nh, hd, num_splits) > int64_t(ZSE_ATTN_STATIC_SCRATCH_FLOATS))
    return ZSE_ERR_LIMIT;
  float* scratch = nullptr;
  if (num_splits > 1) {                       // one split needs no scratch: no lookup, nothing that can fail
    int err = 0;
    scratch = static_scratch(&err);
    if (scratch == nullptr) return err;
  }
  return zse_attn_decode(q, ldq, kv_layer, block_tables, max_blocks, seq_lens, out, ldo, scratch, num_seqs, nh, nkv,
                         hd, block_size, num_splits, scale, stream);
}
