// Attention with grouped-query heads: decode (one new query token per sequence over the paged KV cache) and causal prefill.
#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>

#include "b2_common.cuh"

namespace {

// ---------------------------------------------------------------------------
// paged_decode_kernel
//
// Bound: HBM.  Every K and V row of every context is read once (512 bytes per token and KV head) and used for the
// G = nq / nkv query heads of its group; nothing else of size moves.
//
// One warp brings the tiles (64 tokens of one (sequence, KV head): 16 KB of K, 16 KB of V) into a 3-stage ring by TMA and runs
// ahead over the borders between heads and sequences, so that two CTAs per SM keep up to 190 KB in flight; four warps take 16
// tokens each from a landed tile (ldmatrix, mma.sync.m16n8k16 with the rows past the group's heads empty: the tensor pipe is
// idle most of the time anyway) and keep their own running maximum and sum.  The rows of a context's last tile come in groups of
// 16, so that little is read past its end.
//
// Work split: the tiles of the whole batch, in the order (sequence, head, position), are dealt in contiguous equal ranges
// to the CTAs - the contexts' lengths are read on the device, so a captured graph stays balanced for any batch.  A
// (sequence, head) that spans several CTAs is combined by whichever of them finishes last; a CTA holds at most two such
// parts and settles both at its end.  Settling takes 3-4 us (a fence, an atomic and the parts' way through L2), as long as
// walking 8 tiles: where every (sequence, head) can have a CTA of its own and the longest is no further than that above
// the even share, they are dealt whole.  One sequence of 300 tokens 5.9 -> 4.8 us, 37 of 40..700 tokens 16.5 -> 13.1.
// ---------------------------------------------------------------------------
constexpr int ATT_WARPS = 4, ATT_THREADS = (ATT_WARPS + 1) * 32;  // the last warp is the producer
constexpr int ATT_TILE = 64;          // tokens per tile
constexpr int ATT_HD = 128;           // head dimension
// Query heads per KV head.  (Wider groups: paged_decode_wide_kernel below.)
constexpr int ATT_MAX_GROUP = 2;
constexpr int ATT_CTAS_PER_SM = 2;
constexpr int ATT_STAGES = 3;
constexpr int ATT_HALF_BYTES = ATT_TILE * 128;          // 64 tokens x 64 dimensions: one swizzled box
constexpr int ATT_STAGE_BYTES = 4 * ATT_HALF_BYTES;     // K dimensions 0..63, 64..127, V the same
constexpr int ATT_SLOT = ATT_MAX_GROUP * ATT_HD + 2 * ATT_MAX_GROUP;  // floats of one partial result: O, then the maxima and sums
constexpr int ATT_MAX_SEQS = 1024;
constexpr int ATT_COMBINE_TILES = 8;  // what combining the parts of an item costs, in tiles
static_assert(ATT_CTAS_PER_SM * 2 * ATT_SLOT == B2_ATTN_WS_FLOATS_PER_SM, "the context allocates two slots per CTA");

struct AttnArgs {
  const uint16_t* q;
  int64_t q_stride;
  const int32_t* tables;
  int64_t bt_stride;
  const int32_t* lens;
  uint16_t* out;
  float* ws;       // [2 * CTAs][ATT_SLOT]
  int* counters;   // [sequences * KV heads], zero between launches
  B2Status* status;
  int bt_width, block_size, num_blocks, n_seqs, nkv, group;
  int stages;  // wide groups: tiles of the ring
  uint32_t flip;     // wide groups: the sign bits of a pair of bf16 where the scale is negative
  float scale_log2;  // softmax scale * log2(e); wide groups: its size
};

__device__ __forceinline__ void consumers_meet() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// The tiles [pos, end) of a CTA as segments that lie inside one (sequence, head).
struct AttnWalk {
  const int* first_tile;  // [n_seqs + 1] tiles per KV head before each sequence
  int nkv, pos, end, b;
  // the current segment
  int head, tiles, t0, t1;
  __device__ __forceinline__ AttnWalk(const int* ft, int n_seqs, int heads, int begin, int stop) : first_tile(ft), nkv(heads), pos(begin), end(stop), b(0) {
    int hi = n_seqs - 1;
    while (b < hi) {  // the sequence the first tile belongs to
      const int mid = (b + hi + 1) >> 1;
      if (first_tile[mid] * nkv <= pos) b = mid;
      else hi = mid - 1;
    }
  }
  __device__ __forceinline__ bool next() {
    if (pos >= end) return false;
    while (first_tile[b + 1] * nkv <= pos) ++b;
    tiles = first_tile[b + 1] - first_tile[b];
    const int in_seq = pos - first_tile[b] * nkv;
    head = in_seq / tiles;
    t0 = in_seq - head * tiles;
    t1 = min(tiles, t0 + end - pos);
    pos += t1 - t0;
    return true;
  }
  __device__ __forceinline__ int item_begin() const { return pos - t1; }
};

__global__ void __launch_bounds__(ATT_THREADS, ATT_CTAS_PER_SM)
paged_decode_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmK16,
                    const __grid_constant__ CUtensorMap tmV16, const AttnArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float* s_o = reinterpret_cast<float*>(smem + ATT_STAGES * ATT_STAGE_BYTES);  // [warp][head of the group][ATT_HD]
  int* first_tile = reinterpret_cast<int*>(s_o + ATT_WARPS * a.group * ATT_HD);
  int* s_len = first_tile + a.n_seqs + 1;
  __shared__ float s_m[ATT_WARPS][ATT_MAX_GROUP], s_l[ATT_WARPS][ATT_MAX_GROUP];
  __shared__ __align__(8) uint64_t s_bars[2 * ATT_STAGES];
  __shared__ int s_abort, s_last[2], s_most, s_live;
  volatile int* abort_flag = &s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar_full = b2::smem_u32(s_bars), bar_empty = bar_full + ATT_STAGES * 8;
  if (tid == 0) {
    b2::tma_prefetch_desc(&tmK);
    b2::tma_prefetch_desc(&tmV);
    for (int i = 0; i < ATT_STAGES; ++i) {
      b2::mbar_init(bar_full + i * 8, 1);
      b2::mbar_init(bar_empty + i * 8, ATT_WARPS);
    }
    s_abort = 0;
    b2::mbar_fence_init();
  }
  b2::pdl_launch_dependents();

  // ---- tiles per sequence, prefix-summed by one warp.  Lengths and tables are not results of the kernels just before this
  // one (see the header), so this runs while those are ending; the query and the cache are read after the dependency wait. ----
  const int max_len = a.bt_width * a.block_size;
  if (warp == 0) {
    const int per = (a.n_seqs + 31) / 32, s0 = lane * per;
    int mine = 0, most = 0, live = 0;
#pragma unroll 4
    for (int i = 0; i < per; ++i)
      if (s0 + i < a.n_seqs) {
        const int len = max(0, min(__ldg(a.lens + s0 + i), max_len));
        const int t = (len + ATT_TILE - 1) / ATT_TILE;
        s_len[s0 + i] = len;
        first_tile[s0 + i + 1] = t;
        mine += t;
        most = max(most, t);
        if (t > 0) live = s0 + i + 1;
      }
    most = __reduce_max_sync(0xffffffffu, most);
    live = __reduce_max_sync(0xffffffffu, live);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    int at = incl - mine;
    if (lane == 0) {
      first_tile[0] = 0;
      s_most = most;
      s_live = live;
    }
    for (int i = 0; i < per; ++i)
      if (s0 + i < a.n_seqs) first_tile[s0 + i + 1] = at += first_tile[s0 + i + 1];
  }
  __syncthreads();
  // rows without a context (a graph's padded ones) have no tiles; their output is zero
  if (warp < ATT_WARPS)
    for (int b = blockIdx.x; b < a.n_seqs; b += gridDim.x)
      if (s_len[b] == 0) {
        b2::pdl_wait();
        const int row = a.nkv * a.group * ATT_HD;
        for (int i = tid * 8; i < row; i += ATT_WARPS * 32 * 8) *reinterpret_cast<uint4*>(a.out + static_cast<int64_t>(b) * row + i) = make_uint4(0, 0, 0, 0);
      }
  const int total = first_tile[a.n_seqs] * a.nkv;
  if (total == 0) return;
  // (parts of an item are fewer, and no CTA has more tiles, when as many CTAs as need be take the same number of them)
  const int cta = blockIdx.x, items = s_live * a.nkv, cap = static_cast<int>(gridDim.x);
  const int per = (total + cap - 1) / cap;
  const int spread = per <= 8 ? (total + per - 1) / per : cap;
  const bool by_item = items <= cap && s_most <= total / spread + ATT_COMBINE_TILES;
  const int ctas = by_item ? items : spread;
  if (cta >= ctas) return;
  const int base = total / ctas, rem = total % ctas;
  auto begin_of = [&](int i) {
    if (!by_item) return i * base + min(i, rem);
    const int b = i / a.nkv, first = first_tile[b];
    return b >= s_live ? total : first * a.nkv + (i - b * a.nkv) * (first_tile[b + 1] - first);
  };
  auto cta_of = [&](int t) { const int big = rem * (base + 1); return t < big ? t / (base + 1) : rem + (t - big) / base; };
  AttnWalk walk(first_tile, a.n_seqs, a.nkv, begin_of(cta), begin_of(cta + 1));
  int stage = 0;
  uint32_t phase = 0;

  if (warp == ATT_WARPS) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      bool ok = true, waited = false;
      while (ok && walk.next()) {
        const int32_t* table = a.tables + static_cast<int64_t>(walk.b) * a.bt_stride;
        const int len = s_len[walk.b], x = walk.head * ATT_HD;
        int blk_no = -1, blk = 0;
        for (int t = walk.t0; t < walk.t1; ++t) {
          const int tok = t * ATT_TILE, left = len - tok;
          if (tok / a.block_size != blk_no) {
            blk_no = tok / a.block_size;
            blk = min(max(0, __ldg(table + blk_no)), a.num_blocks - 1);  // stay inside the cache whatever the table holds
          }
          if (!waited) b2::pdl_wait();
          waited = true;
          const int y = blk * a.block_size + tok - blk_no * a.block_size;
          if (!b2::mbar_wait(bar_empty + stage * 8, phase ^ 1, abort_flag, 1000000000ull, B2_WAIT_SMEM_EMPTY)) { ok = false; break; }
          const uint32_t fb = bar_full + stage * 8, dst = b2::smem_u32(smem) + stage * ATT_STAGE_BYTES;
          if (left >= ATT_TILE) {
            b2::mbar_arrive_expect_tx(fb, ATT_STAGE_BYTES);
            b2::tma_load_2d(dst, &tmK, fb, x, y, b2::kEvictFirst);
            b2::tma_load_2d(dst + ATT_HALF_BYTES, &tmK, fb, x + 64, y, b2::kEvictFirst);
            b2::tma_load_2d(dst + 2 * ATT_HALF_BYTES, &tmV, fb, x, y, b2::kEvictFirst);
            b2::tma_load_2d(dst + 3 * ATT_HALF_BYTES, &tmV, fb, x + 64, y, b2::kEvictFirst);
          } else {
            const int groups = (left + 15) >> 4;
            b2::mbar_arrive_expect_tx(fb, groups * (ATT_STAGE_BYTES / 4));
            for (int i = 0; i < groups; ++i) {
              const uint32_t d = dst + i * 16 * 128;
              b2::tma_load_2d(d, &tmK16, fb, x, y + i * 16, b2::kEvictFirst);
              b2::tma_load_2d(d + ATT_HALF_BYTES, &tmK16, fb, x + 64, y + i * 16, b2::kEvictFirst);
              b2::tma_load_2d(d + 2 * ATT_HALF_BYTES, &tmV16, fb, x, y + i * 16, b2::kEvictFirst);
              b2::tma_load_2d(d + 3 * ATT_HALF_BYTES, &tmV16, fb, x + 64, y + i * 16, b2::kEvictFirst);
            }
          }
          if (++stage == ATT_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  const int g = lane >> 2, c = lane & 3;  // row (query head of the group) and column pair of the fragments
  // this lane's row of the four 8x8 matrices of an ldmatrix: K as (tokens, dims) pairs, V transposed
  const int k_tok = ((lane >> 4) << 3) + (lane & 7), k_chunk = (lane >> 3) & 1;
  const int v_tok = (((lane >> 3) & 1) << 3) + (lane & 7), v_chunk = lane >> 4;
  b2::pdl_wait();
  int open_item[2] = {-1, -1}, open_c0[2], open_n[2];  // parts written to the workspace: [0] an item begun elsewhere, [1] one begun here
  while (walk.next()) {
    const int b = walk.b, head = walk.head, len = s_len[b];
    const uint16_t* qrow = a.q + static_cast<int64_t>(b) * a.q_stride + (head * a.group + g) * ATT_HD;
    uint32_t qf[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int i = 0; i < 2; ++i) qf[k][i] = g < a.group ? *reinterpret_cast<const uint32_t*>(qrow + k * 16 + i * 8 + c * 2) : 0u;
    float o[16][2];
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j][0] = o[j][1] = 0.f;
    float m = -INFINITY, l = 0.f;

    for (int t = walk.t0; t < walk.t1; ++t) {
      const int left = len - t * ATT_TILE - warp * 16;  // tokens of this warp's 16 that exist
      if (!b2::mbar_wait(bar_full + stage * 8, phase, abort_flag, 1000000000ull, B2_WAIT_SMEM_FULL)) break;
      if (left > 0) {
        const uint32_t k_row = b2::smem_u32(smem) + stage * ATT_STAGE_BYTES + (warp * 16 + k_tok) * 128;
        float s[2][2] = {};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          uint32_t kf[4];
          b2::ldmatrix_x4(kf, k_row + (k >> 2) * ATT_HALF_BYTES + ((((k & 3) * 2 + k_chunk) ^ (k_tok & 7)) << 4));
          b2::mma_rows8(s[0][0], s[0][1], qf[k][0], qf[k][1], kf[0], kf[1]);
          b2::mma_rows8(s[1][0], s[1][1], qf[k][0], qf[k][1], kf[2], kf[3]);
        }
        float mx = m;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            s[i][e] = i * 8 + c * 2 + e < left ? s[i][e] * a.scale_log2 : -INFINITY;
            mx = fmaxf(mx, s[i][e]);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        if (__any_sync(0xffffffffu, mx > m)) {
          const float f = exp2f(m - mx);  // mx is finite: at least one token exists
          m = mx;
          l *= f;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            o[j][0] *= f;
            o[j][1] *= f;
          }
        }
        float p[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            p[i][e] = b2::ex2(s[i][e] - m);
            l += p[i][e];
          }
        const uint32_t p0 = b2::pack_bf16(p[0][0], p[0][1]), p1 = b2::pack_bf16(p[1][0], p[1][1]);
        const uint32_t v_row = b2::smem_u32(smem) + stage * ATT_STAGE_BYTES + 2 * ATT_HALF_BYTES + (warp * 16 + v_tok) * 128;
        // rows past the context's end may hold anything: they count as zero
        uint32_t keep[2] = {0xffffffffu, 0xffffffffu};
        if (left < 16) {
#pragma unroll
          for (int i = 0; i < 2; ++i) keep[i] = (i * 8 + c * 2 < left ? 0xffffu : 0u) | (i * 8 + c * 2 + 1 < left ? 0xffff0000u : 0u);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t vf[4];
          b2::ldmatrix_x4_trans(vf, v_row + (j >> 2) * ATT_HALF_BYTES + ((((j & 3) * 2 + v_chunk) ^ (v_tok & 7)) << 4));
          b2::mma_rows8(o[2 * j][0], o[2 * j][1], p0, p1, vf[0] & keep[0], vf[1] & keep[1]);
          b2::mma_rows8(o[2 * j + 1][0], o[2 * j + 1][1], p0, p1, vf[2] & keep[0], vf[3] & keep[1]);
        }
      }
      __syncwarp();
      if (lane == 0) b2::mbar_arrive(bar_empty + stage * 8);
      if (++stage == ATT_STAGES) { stage = 0; phase ^= 1; }
    }

    // ---- the four warps' parts meet in shared memory ----
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    consumers_meet();  // the previous segment's parts have been read
    if (g < a.group) {
      if (c == 0) {
        s_m[warp][g] = m;
        s_l[warp][g] = l;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) *reinterpret_cast<float2*>(s_o + (warp * a.group + g) * ATT_HD + j * 8 + c * 2) = make_float2(o[j][0], o[j][1]);
    }
    consumers_meet();
    const bool whole = walk.t0 == 0 && walk.t1 == walk.tiles;
    const int which = walk.t0 == 0 ? 1 : 0;
    float* slot = a.ws + (static_cast<int64_t>(cta) * 2 + which) * ATT_SLOT;
    uint16_t* out = a.out + (static_cast<int64_t>(b) * a.nkv + head) * a.group * ATT_HD;
    for (int i = tid; i < a.group * (ATT_HD / 4); i += ATT_WARPS * 32) {
      const int r = i >> 5, d = (i & 31) * 4;
      float mx = s_m[0][r];
#pragma unroll
      for (int w = 1; w < ATT_WARPS; ++w) mx = fmaxf(mx, s_m[w][r]);
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < ATT_WARPS; ++w) {
        const float f = mx == -INFINITY ? 0.f : exp2f(s_m[w][r] - mx);
        const float4 x = *reinterpret_cast<const float4*>(s_o + (w * a.group + r) * ATT_HD + d);
        acc.x += f * x.x; acc.y += f * x.y; acc.z += f * x.z; acc.w += f * x.w;
        sum += f * s_l[w][r];
      }
      if (whole) {
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
        *reinterpret_cast<uint2*>(out + r * ATT_HD + d) = make_uint2(b2::pack_bf16(acc.x * inv, acc.y * inv), b2::pack_bf16(acc.z * inv, acc.w * inv));
      } else {
        *reinterpret_cast<float4*>(slot + r * ATT_HD + d) = acc;
        if (d == 0) {
          slot[ATT_MAX_GROUP * ATT_HD + r] = mx;
          slot[ATT_MAX_GROUP * ATT_HD + ATT_MAX_GROUP + r] = sum;
        }
      }
    }
    if (!whole) {
      const int begin = walk.item_begin();
      open_item[which] = b * a.nkv + head;
      open_c0[which] = cta_of(begin);
      open_n[which] = cta_of(begin + walk.tiles - 1) - open_c0[which] + 1;
    }
  }

  // ---- parts of items that other CTAs share: whoever arrives last combines them ----
  if (open_item[0] >= 0 || open_item[1] >= 0) {
    __threadfence();
    consumers_meet();
    if (tid < 2) {
      const int item = tid == 0 ? open_item[0] : open_item[1], n = tid == 0 ? open_n[0] : open_n[1];
      s_last[tid] = 0;
      if (item >= 0 && atomicAdd(a.counters + item, 1) == n - 1) {
        a.counters[item] = 0;
        s_last[tid] = 1;
      }
    }
    consumers_meet();
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      if (!s_last[which]) continue;
      __threadfence();
      const int item = open_item[which], n = open_n[which];
      // the first CTA holds the item's beginning (its slot 1), the others a later part (their slot 0)
      const float* first = a.ws + static_cast<int64_t>(open_c0[which]) * 2 * ATT_SLOT;
      auto part = [&](int k) { return first + (k == 0 ? 1 : 2 * k) * ATT_SLOT; };
      uint16_t* out = a.out + static_cast<int64_t>(item) * a.group * ATT_HD;
      if (n <= 8) {  // a few parts: every thread reads all of them
        for (int i = tid; i < a.group * (ATT_HD / 4); i += ATT_WARPS * 32) {
          const int r = i >> 5, d = (i & 31) * 4;
          float pm[8], ps[8], mx = -INFINITY, sum = 0.f;
          uint4 x[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < n) {
              pm[k] = b2::ld_cg_f32(part(k) + ATT_MAX_GROUP * ATT_HD + r);
              ps[k] = b2::ld_cg_f32(part(k) + ATT_MAX_GROUP * ATT_HD + ATT_MAX_GROUP + r);
              x[k] = b2::ld_cg_v4(part(k) + r * ATT_HD + d);
            }
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < n) mx = fmaxf(mx, pm[k]);
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < n) {
              const float f = mx == -INFINITY ? 0.f : exp2f(pm[k] - mx);
              acc.x += f * __uint_as_float(x[k].x); acc.y += f * __uint_as_float(x[k].y);
              acc.z += f * __uint_as_float(x[k].z); acc.w += f * __uint_as_float(x[k].w);
              sum += f * ps[k];
            }
          const float inv = sum > 0.f ? 1.f / sum : 0.f;
          *reinterpret_cast<uint2*>(out + r * ATT_HD + d) = make_uint2(b2::pack_bf16(acc.x * inv, acc.y * inv), b2::pack_bf16(acc.z * inv, acc.w * inv));
        }
        continue;
      }
      // weights of the parts, one warp per head: n <= 2 * 148 parts, 512 places per head in s_o
      consumers_meet();
      for (int r = warp; r < a.group; r += ATT_WARPS) {
        float mx = -INFINITY, sum = 0.f;
        for (int k = lane; k < n; k += 32) mx = fmaxf(mx, b2::ld_cg_f32(part(k) + ATT_MAX_GROUP * ATT_HD + r));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        for (int k = lane; k < n; k += 32) {
          const float f = mx == -INFINITY ? 0.f : exp2f(b2::ld_cg_f32(part(k) + ATT_MAX_GROUP * ATT_HD + r) - mx);
          s_o[r * (ATT_WARPS * ATT_HD) + k] = f;
          sum += f * b2::ld_cg_f32(part(k) + ATT_MAX_GROUP * ATT_HD + ATT_MAX_GROUP + r);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) s_m[0][r] = sum > 0.f ? 1.f / sum : 0.f;
      }
      consumers_meet();
      for (int i = tid; i < a.group * (ATT_HD / 4); i += ATT_WARPS * 32) {
        const int r = i >> 5, d = (i & 31) * 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int k = 0; k < n; ++k) {
          const float f = s_o[r * (ATT_WARPS * ATT_HD) + k];
          const uint4 x = b2::ld_cg_v4(part(k) + r * ATT_HD + d);
          acc.x += f * __uint_as_float(x.x); acc.y += f * __uint_as_float(x.y);
          acc.z += f * __uint_as_float(x.z); acc.w += f * __uint_as_float(x.w);
        }
        const float inv = s_m[0][r];
        *reinterpret_cast<uint2*>(out + r * ATT_HD + d) = make_uint2(b2::pack_bf16(acc.x * inv, acc.y * inv), b2::pack_bf16(acc.z * inv, acc.w * inv));
      }
    }
  }
  const int aborted = *abort_flag;
  if (aborted) {
    for (int i = 0; i < 100; ++i) __nanosleep(2000);  // copies in flight land before the CTA leaves
    if (tid == 0) b2::report_timeout(a.status, aborted);
  }
}

// ---------------------------------------------------------------------------
// paged_decode_wide_kernel
//
// Decode attention with 3 to 8 query heads per KV head.  Bound: HBM, as above.
//
// The models with wide groups are deep and wide enough that another rounding of the probabilities grows to 3 % of their hidden
// state, and so this kernel fixes what each probability is rounded against: a context is walked from its end in blocks of 128
// tokens, each rounded to bf16 against the maximum of that block and those walked before, and every output element is one unbroken
// chain of tensor-core sums.  That leaves one CTA per (sequence, KV head) and shares its work out inside it: for the scores a
// warp takes 16 tokens of each tile of 64, the maxima meet in shared memory, and for the product a warp takes 32 of the 128
// dimensions and all tokens, with the probabilities from shared memory; every thread adds up the columns of its fragments in
// their order.  Where flash-attn does not cut contexts the results are its own but for 0 to 3 elements in a million of random data.
//
// 64 contexts of 1056 tokens, 32 / 8 heads: 66.7 us in flash-attn, 45.2 here (6.1 TB/s); 96 of 70..700 47.0 and 28.8, 32 of 1056
// 34.9 and 23.7.  Not for narrow groups, although batches of about equal contexts would gain where there are three CTAs an SM and more (64 of 1056
// tokens, 16 / 8 heads, 48.7 and 43.7 us, 512 of 30..270 68 and 54): the other kernel's warps round against maxima of their own, which is
// nearer to float64 (2.12e-3 and 2.23e-3; 2.05e-3 and 2.18e-3 for contexts of 100..1024), and its even ranges take a long context apart, which is walked
// alone here (63 contexts of 100 tokens and one of 4000 15.6 and 57.7 us, one of 32000 34 and 418).
//
// Four CTAs per SM with a ring of three 16 KB tiles (64 tokens of K or of V) each, or fewer with longer rings where there are no
// more to be had: 190 KB per SM in flight.  With no more than two CTAs for an SM (FEW) a block's product runs side by side with the next
// block's scores: nothing else fills the gaps in a warp's chains of eight tensor-core sums.  A block takes 1.0 us instead of 1.8: 16 contexts
// of 1056 tokens 19.5 -> 13.4 us (16.1 by the producer's whole warp and the longer ring alone), of 100..3000 42 -> 26, 32 of 1056 26.1 -> 23.7.
// ---------------------------------------------------------------------------
constexpr int WD_MAX_GROUP = 8;
constexpr int WD_MAX_STAGES = 12;
constexpr int WD_CTAS_PER_SM = 4;
constexpr int WD_BLOCK = 2 * ATT_TILE;                    // tokens that share a maximum
constexpr int WD_STAGE_BYTES = 2 * ATT_HALF_BYTES;        // dimensions 0..63, 64..127
constexpr int WD_P_PITCH = WD_BLOCK + 8;                  // floats: rows start 8 banks apart, so that the 8-byte accesses of half a warp meet in none
// The fewest (sequence, KV head) pairs that are served (16 contexts of 1056 tokens and 8 KV heads 38.8 us in the library, 13.4 here, of 100..3000 tokens
// 59 and 26).  Up to 1.6 pairs an SM the library cuts long contexts into parts, each rounded for itself, and is a little nearer to float64; a
// context of one CTA walks at 70 GB/s with one CTA for an SM, at 50 with two, at 40 beyond, however long it is.  Attention.attend leaves those batches to the library.
constexpr int WD_MIN_ITEMS = 128;
constexpr uint32_t wide_smem(int stages) { return 1024 + stages * WD_STAGE_BYTES; }
static_assert(wide_smem(WD_MAX_STAGES) + 6 * 1024 <= 228 * 1024 && 2 * (wide_smem(6) + 6 * 1024) <= 228 * 1024 && 3 * (wide_smem(4) + 6 * 1024) <= 228 * 1024 && 4 * (wide_smem(3) + 6 * 1024) <= 228 * 1024, "CTAs per SM (6 KB: static, reserved)");

template <bool FEW>
__global__ void __launch_bounds__(ATT_THREADS, FEW ? 2 : WD_CTAS_PER_SM)
paged_decode_wide_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmK16,
                         const __grid_constant__ CUtensorMap tmV16, const AttnArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ __align__(16) float s_p[WD_MAX_GROUP][WD_P_PITCH];
  __shared__ float s_m[ATT_WARPS][WD_MAX_GROUP];
  __shared__ __align__(8) uint64_t s_bars[2 * WD_MAX_STAGES];
  __shared__ int s_abort;
  volatile int* abort_flag = &s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ring = b2::smem_u32(smem), bar_full = b2::smem_u32(s_bars), bar_empty = bar_full + WD_MAX_STAGES * 8;
  if (threadIdx.x == 0) {
    b2::tma_prefetch_desc(&tmK);
    b2::tma_prefetch_desc(&tmV);
    for (int i = 0; i < a.stages; ++i) {
      b2::mbar_init(bar_full + i * 8, 1);
      b2::mbar_init(bar_empty + i * 8, ATT_WARPS);
    }
    s_abort = 0;
    b2::mbar_fence_init();
  }
  __syncthreads();
  b2::pdl_launch_dependents();
  const int b = blockIdx.x / a.nkv, head = blockIdx.x - b * a.nkv;
  const int len = b2::uniform(max(0, min(__ldg(a.lens + b), a.bt_width * a.block_size)));
  const int blocks = (len + WD_BLOCK - 1) / WD_BLOCK;
  uint16_t* out = a.out + static_cast<int64_t>(blockIdx.x) * a.group * ATT_HD;
  int stage = 0;
  uint32_t phase = 0;

  if (b2::uniform(warp) == ATT_WARPS) {  // (uniform for everyone, it costs the other warps registers that they spill)
    // ---------------- TMA producer: the whole warp walks, one thread issues (see b2_gemm_tile.cu) ----------------
    const int32_t* table = a.tables + static_cast<int64_t>(b) * a.bt_stride;
    const int x = head * ATT_HD;
    bool ok = true;
    b2::pdl_wait();
    for (int j = blocks - 1; ok && j >= 0; --j) {
      int y[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int tok = max(0, min(j * WD_BLOCK + t * ATT_TILE, len - 1)), no = tok / a.block_size;
        y[t] = b2::uniform(min(max(0, __ldg(table + no)), a.num_blocks - 1)) * a.block_size + tok - no * a.block_size;  // inside the cache whatever the table holds
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // K, K, V, V
        const int left = len - j * WD_BLOCK - (i & 1) * ATT_TILE;
        if (left <= 0) continue;
        ok = __all_sync(0xffffffffu, b2::mbar_wait(bar_empty + stage * 8, phase ^ 1, abort_flag, 1000000000ull, B2_WAIT_SMEM_EMPTY)) != 0;
        if (!ok) break;
        const uint32_t fb = bar_full + stage * 8, dst = ring + stage * WD_STAGE_BYTES;
        const int row = y[i & 1];
        if (b2::elect_one()) {
          if (left >= ATT_TILE) {
            const CUtensorMap* m = i < 2 ? &tmK : &tmV;
            b2::mbar_arrive_expect_tx(fb, WD_STAGE_BYTES);
            b2::tma_load_2d(dst, m, fb, x, row, b2::kEvictFirst);
            b2::tma_load_2d(dst + ATT_HALF_BYTES, m, fb, x + 64, row, b2::kEvictFirst);
          } else {
            const CUtensorMap* m = i < 2 ? &tmK16 : &tmV16;
            const int groups = (left + 15) >> 4;
            b2::mbar_arrive_expect_tx(fb, groups * (WD_STAGE_BYTES / 4));
            for (int r = 0; r < groups; ++r) {
              b2::tma_load_2d(dst + r * 16 * 128, m, fb, x, row + r * 16, b2::kEvictFirst);
              b2::tma_load_2d(dst + r * 16 * 128 + ATT_HALF_BYTES, m, fb, x + 64, row + r * 16, b2::kEvictFirst);
            }
          }
        }
        __syncwarp();
        if (++stage == a.stages) { stage = 0; phase ^= 1; }
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  const int g = lane >> 2, c = lane & 3;  // row (query head of the group) and column pair of the fragments
  const int k_tok = ((lane >> 4) << 3) + (lane & 7), k_chunk = (lane >> 3) & 1;
  const int v_tok = (((lane >> 3) & 1) << 3) + (lane & 7), v_chunk = lane >> 4;
  b2::pdl_wait();
  uint32_t qf[8][2];
  {
    const uint16_t* qrow = a.q + static_cast<int64_t>(b) * a.q_stride + (head * a.group + g) * ATT_HD;
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int i = 0; i < 2; ++i) qf[k][i] = g < a.group ? *reinterpret_cast<const uint32_t*>(qrow + k * 16 + i * 8 + c * 2) ^ a.flip : 0u;
  }
  float o[4][2] = {};  // this warp's 32 dimensions
  float m = -INFINITY, l = 0.f;
  // (A wait that runs out leaves its flag, the waits after it end at once, and the walk goes on to its end: every warp meets every barrier.)
  auto landed = [&]() { b2::mbar_wait(bar_full + stage * 8, phase, abort_flag, 1000000000ull, B2_WAIT_SMEM_FULL); };
  auto advance = [&]() {
    const int was = stage;
    if (++stage == a.stages) { stage = 0; phase ^= 1; }
    return was;
  };
  auto release = [&](int st) {
    __syncwarp();
    if (lane == 0) b2::mbar_arrive(bar_empty + st * 8);
  };
  auto k_row = [&]() { return ring + stage * WD_STAGE_BYTES + (warp * 16 + k_tok) * 128; };
  auto v_row = [&]() { return ring + stage * WD_STAGE_BYTES + (warp >> 1) * ATT_HALF_BYTES + v_tok * 128; };
  // 16 dimensions of the scores of this warp's 16 tokens of a tile
  auto keys = [&](uint32_t row, int k, float (&d)[2][2]) {
    uint32_t kf[4];
    b2::ldmatrix_x4(kf, row + (k >> 2) * ATT_HALF_BYTES + ((((k & 3) * 2 + k_chunk) ^ (k_tok & 7)) << 4));
    b2::mma_rows8(d[0][0], d[0][1], qf[k][0], qf[k][1], kf[0], kf[1]);
    b2::mma_rows8(d[1][0], d[1][1], qf[k][0], qf[k][1], kf[2], kf[3]);
  };
  // 16 tokens of the product: the probabilities' fragments, their sum (every warp reads all of them: each holds the whole sum), the values;
  // rows past the context's end may hold anything and count as zero
  auto values = [&](uint32_t row, int t, int k, uint32_t keep0, uint32_t keep1) {
    const float* pr = &s_p[g][t * ATT_TILE + k * 16 + c * 2];
    const float2 x = *reinterpret_cast<const float2*>(pr), y = *reinterpret_cast<const float2*>(pr + 8);
    l = l + x.x + x.y + y.x + y.y;
    const uint32_t p0 = b2::pack_bf16(x.x, x.y), p1 = b2::pack_bf16(y.x, y.y);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t vf[4];
      b2::ldmatrix_x4_trans(vf, row + k * 16 * 128 + (((((warp & 1) * 2 + i) * 2 + v_chunk) ^ (v_tok & 7)) << 4));
      b2::mma_rows8(o[2 * i][0], o[2 * i][1], p0, p1, vf[0] & keep0, vf[1] & keep1);
      b2::mma_rows8(o[2 * i + 1][0], o[2 * i + 1][1], p0, p1, vf[2] & keep0, vf[3] & keep1);
    }
  };
  float s[2][2][2];  // scores of this warp's tokens
  auto scores = [&](int there) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      s[t][0][0] = s[t][0][1] = s[t][1][0] = s[t][1][1] = 0.f;
      const int left = there - t * ATT_TILE - warp * 16;
      if (there > t * ATT_TILE) {
        landed();
        if (left > 0) {
          const uint32_t row = k_row();
#pragma unroll
          for (int k = 0; k < 8; ++k) keys(row, k, s[t]);
        }
        release(advance());
      }
      if (left < 16) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (i * 8 + c * 2 + e >= left) s[t][i][e] = -INFINITY;
      }
    }
  };
  if (FEW && blocks > 0) scores(len - (blocks - 1) * WD_BLOCK);
  for (int j = blocks - 1; j >= 0; --j) {
    const int there = min(WD_BLOCK, len - j * WD_BLOCK);  // tokens of the block that exist
    if (!FEW) scores(there);
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, s[i >> 2][(i >> 1) & 1][i & 1]);
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    if (c == 0) s_m[warp][g] = mx;
    consumers_meet();
    mx = fmaxf(fmaxf(fmaxf(s_m[0][g], s_m[1][g]), fmaxf(s_m[2][g], s_m[3][g])), m);
    const float f = mx == m ? 1.f : b2::ex2((m - mx) * a.scale_log2);
    const float ref = mx == -INFINITY ? 0.f : mx * a.scale_log2;
    m = mx;
    l *= f;
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<float2*>(&s_p[g][t * ATT_TILE + warp * 16 + i * 8 + c * 2]) =
            make_float2(b2::ex2(fmaf(s[t][i][0], a.scale_log2, -ref)), b2::ex2(fmaf(s[t][i][1], a.scale_log2, -ref)));
    consumers_meet();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[i][0] *= f;
      o[i][1] *= f;
    }
    if (FEW && j > 0 && there == WD_BLOCK) {
      // this block's product and the next one's scores side by side: four and four chains, of which a warp alone fills the gaps of neither
      uint32_t vr[2], kr[2];
      int from[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < 2) vr[i] = v_row();
        else kr[i - 2] = k_row();
        landed();
        from[i] = advance();
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) s[t][0][0] = s[t][0][1] = s[t][1][0] = s[t][1][1] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        keys(kr[0], k, s[0]);
        keys(kr[1], k, s[1]);
        values(vr[k >> 2], k >> 2, k & 3, 0xffffffffu, 0xffffffffu);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) release(from[i]);
      continue;
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (there <= t * ATT_TILE) break;
      const uint32_t row = v_row();
      landed();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int left = there - t * ATT_TILE - k * 16;
        if (left <= 0) break;
        uint32_t keep[2] = {0xffffffffu, 0xffffffffu};
        if (left < 16) {
#pragma unroll
          for (int i = 0; i < 2; ++i) keep[i] = (i * 8 + c * 2 < left ? 0xffffu : 0u) | (i * 8 + c * 2 + 1 < left ? 0xffff0000u : 0u);
        }
        values(row, t, k, keep[0], keep[1]);
      }
      release(advance());
    }
    if (FEW && j > 0) scores(WD_BLOCK);
  }
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  if (g < a.group) {
    const float inv = l > 0.f ? __fdividef(1.f, l) : 0.f;  // (no context: zeros)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<uint32_t*>(out + g * ATT_HD + warp * 32 + i * 8 + c * 2) = b2::pack_bf16(o[i][0] * inv, o[i][1] * inv);
  }
  const int aborted = *abort_flag;
  if (aborted) {
    for (int i = 0; i < 100; ++i) __nanosleep(2000);  // copies in flight land before the CTA leaves
    if (threadIdx.x == 0) b2::report_timeout(a.status, aborted);
  }
}

// ---------------------------------------------------------------------------
// prefill_attention_kernel
//
// Causal attention of many query tokens per sequence over keys and values in rows of a matrix (the qkv output) or in the paged
// cache.  Bound: the tensor pipe and what feeds it.  A block of 64 keys takes both heads' scores 768 clocks (Q is read again for
// every 64 columns: 48 KB of shared memory per head), their products 512 and their exponentials 1024 of the units that run beside
// those; the walk does a block in about 1900, and in 1800 with the softmax left out.  One sequence of 8192 tokens, 16 heads, 458 -> 246 us
// (1120 TFLOP/s); eight of 2048 244 -> 168; four of 1024, 32 / 8 heads, 131 us in flash-attn, 57 here.
//
// A CTA takes 128 query tokens of one sequence for two heads that share a KV head, and walks the keys from the tile's diagonal
// down in blocks of 64:
//   warp 0        TMA: Q of both heads once, then K and V blocks, four of each in flight
//   warps 1, 2    tcgen05.mma of a head each: S = Q K^T (128 x 64, fp32, tensor memory), O += P V with P read from tensor memory
//   warps 4..11   one thread per query row and head: running maximum and sum, P = exp2(...) rounded to bf16 over S
//   warps 12..15  O is rescaled where a row's maximum has grown, while the softmax warps are at their exponentials
// Tensor memory: two S of 64 columns per head, then O of the two heads, 128 columns each.  With two S the scores of the next
// block are there before this one's are done with: a head's warp issues P V (block j), then Q K^T (block j + 2) into the columns
// that P is read from.  The order of issue is promised only to products of one shape and accumulator, which these are not: the warp waits for P V
// in between, while the other head's products run (without the wait the times were the same: 246 us at 8192 tokens, 16 heads).  (With one S of 128 keys per head
// and one warp for both, the heads ran in step: 7700 clocks per 128 keys.  One warp for both, here: 275 us instead of 246; values that are
// the same in all lanes but not in a form that shows it, b2::uniform: 346.)
//
// Every probability is rounded to bf16 against the maximum of its block and those walked before, as in flash-attn, whose results
// these are, bit for bit on random data.  Over a block table that library takes blocks of 128 tokens; PAIRS does the same: two blocks share the
// maximum of both, the lower one goes first.  Narrow groups do without: 28 layers of a 1024-wide model move by 0.5 %.
//
// O is rescaled whenever a row's maximum grows, so that the largest probability so far is exactly 1 (rescaling only past a growth of
// 2^8 rounds it: 2.13e-3 from float64 where scores have standard deviation 3, against 1.76e-3).
// ---------------------------------------------------------------------------
constexpr int PF_ROWS = 128, PF_KEYS = 64, PF_THREADS = 512, PF_STAGES = 4;
constexpr uint32_t PF_Q = 128 * 128 * 2;        // 128 rows of 128 bf16, as two 64-wide swizzled halves
constexpr uint32_t PF_KV = PF_KEYS * 128 * 2;   // a block of keys or of values, the same way
constexpr uint32_t PF_SMEM = 1024 + 2 * PF_Q + 2 * PF_STAGES * PF_KV;
constexpr uint64_t PF_LIMIT_NS = 1000000000ull;

struct PrefillArgs {
  const int32_t *cu_q, *cu_k, *tables;  // tables: null = keys and values are rows cu_k[b] .. of the matrices
  int64_t bt_stride;
  int bt_width, block_size, kv_rows, nq, group;
  uint16_t* out;
  uint32_t negate;   // the instruction descriptor's bit that negates Q, where the scale is negative
  float scale_log2;  // size of softmax scale * log2(e)
  B2Status* status;
};

__device__ __forceinline__ void umma_bf16_ts(uint32_t d, uint32_t a_tmem, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a_tmem), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
      "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// tcgen05.wait::ld, before which nothing reads the 64 columns
__device__ __forceinline__ void tc_wait_ld(uint32_t (&r)[2][32]) {
  b2::tc_wait_ld();
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 32; i += 8)
      asm volatile("" : "+r"(r[h][i]), "+r"(r[h][i + 1]), "+r"(r[h][i + 2]), "+r"(r[h][i + 3]), "+r"(r[h][i + 4]), "+r"(r[h][i + 5]), "+r"(r[h][i + 6]), "+r"(r[h][i + 7]));
}
// two products and sums in one instruction, each rounded as fmaf rounds it
__device__ __forceinline__ uint64_t pair_of(float x, float y) {
  uint64_t p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(x), "f"(y));
  return p;
}
__device__ __forceinline__ void fma_pair(float& x, float& y, uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(d));
}
// V as the second operand, [tokens][dimensions] with the dimensions contiguous: MN-major, 128-byte swizzle.  8 tokens are 1024
// bytes apart (stride offset), the two halves of 64 dimensions PF_KV / 2 (leading offset).
__device__ __forceinline__ uint64_t umma_smem_desc_mn(uint32_t addr) {
  return static_cast<uint64_t>((addr & 0x3FFFF) >> 4) | (static_cast<uint64_t>((PF_KV / 2) >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}

template <bool PAIRS>
__global__ void __launch_bounds__(PF_THREADS, 1)
prefill_attention_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const PrefillArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t s_q = b2::smem_u32(smem), s_k = s_q + 2 * PF_Q, s_v = s_k + PF_STAGES * PF_KV;
  __shared__ __align__(8) uint64_t s_bars[1 + 4 * PF_STAGES + 4 + 4 + 16 + 2 + 2];
  __shared__ float s_factor[2][2][PF_ROWS];  // [head][block & 1][row]: what O is multiplied by before the block's product
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  volatile int* abort_flag = &s_abort;
  const uint32_t bars = b2::smem_u32(s_bars);
  const uint32_t q_full = bars, k_full = bars + 8, k_empty = k_full + PF_STAGES * 8, v_full = k_empty + PF_STAGES * 8, v_empty = v_full + PF_STAGES * 8;
  // [head][block & 1], and for the factors one per warp beside those; o_done: the product of a block, o_final: of the last one
  const uint32_t s_full = v_empty + PF_STAGES * 8, p_full = s_full + 4 * 8, f_full = p_full + 4 * 8, o_done = f_full + 16 * 8, o_final = o_done + 2 * 8;
  const int warp = b2::uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    b2::tma_prefetch_desc(&tmQ);
    b2::tma_prefetch_desc(&tmK);
    b2::tma_prefetch_desc(&tmV);
    b2::mbar_init(q_full, 1);
    for (int i = 0; i < 4 * PF_STAGES; ++i) b2::mbar_init(k_full + i * 8, (i / PF_STAGES) & 1 ? 2 : 1);  // (a block is free when both heads are done with it)
    for (int i = 0; i < 4; ++i) b2::mbar_init(s_full + i * 8, 1);
    for (int i = 0; i < 4; ++i) b2::mbar_init(p_full + i * 8, 8);
    for (int i = 0; i < 16 + 4; ++i) b2::mbar_init(f_full + i * 8, 1);
    s_abort = 0;
    b2::mbar_fence_init();
  }
  if (warp == 1) {
    b2::tmem_alloc(b2::smem_u32(&s_tmem), 512);
    b2::tmem_relinquish();
  }
  b2::tc_fence_before();
  __syncthreads();
  b2::tc_fence_after();
  const uint32_t tmem = b2::uniform(s_tmem);
  b2::pdl_launch_dependents();
  b2::pdl_wait();

  // sequence, pair of heads, tile of 128 query tokens (the long rows of the causal triangle first)
  const int b = blockIdx.y, head = blockIdx.x * 2, kv_head = head / a.group;
  const int q0 = b2::uniform(__ldg(a.cu_q + b)), q_len = b2::uniform(__ldg(a.cu_q + b + 1)) - q0;
  const int k0 = b2::uniform(__ldg(a.cu_k + b)), kv_len = b2::uniform(__ldg(a.cu_k + b + 1)) - k0;
  const int t0 = (gridDim.z - 1 - blockIdx.z) * PF_ROWS;
  const int shift = kv_len - q_len;  // position of the first query token
  const int n = kv_len > 0 ? max(1, (min(kv_len, shift + min(q_len, t0 + PF_ROWS)) + PF_KEYS - 1) / PF_KEYS) : 0;  // key blocks
  if (t0 >= q_len || n == 0) {
    // queries of a sequence without keys: nothing to attend to
    for (int i = threadIdx.x; i < min(PF_ROWS, q_len - t0) * 32; i += PF_THREADS)
      *reinterpret_cast<uint4*>(a.out + (static_cast<int64_t>(q0 + t0 + (i >> 5)) * a.nq + head) * 128 + (i & 31) * 8) = make_uint4(0, 0, 0, 0);
    if (warp == 1) b2::tmem_dealloc(tmem, 512);
    return;
  }
  auto all_wait = [&](uint32_t bar, uint32_t phase, int code) {
    return __all_sync(0xffffffffu, b2::mbar_wait(bar, phase, abort_flag, PF_LIMIT_NS, code)) != 0;
  };
  // block j of the walk in the order of the keys (its scores are in buffer j & 1 of its head)
  const int odd = PAIRS ? n & 1 : 0;
  auto block_of = [&](int j) { return !PAIRS || j < odd ? n - 1 - j : n - odd - 2 - ((j - odd) & ~1) + ((j - odd) & 1); };

  if (warp == 0) {
    // (the whole warp walks and one thread issues, here and in the next warp: operands then stay in uniform registers)
    if (b2::elect_one()) {
      b2::mbar_arrive_expect_tx(q_full, 2 * PF_Q);
      for (int h = 0; h < 2; ++h)
        for (int i = 0; i < 2; ++i) b2::tma_load_2d(s_q + h * PF_Q + i * (PF_Q / 2), &tmQ, q_full, (head + h) * 128 + i * 64, q0 + t0, b2::kEvictFirst);
    }
    __syncwarp();
    const int x = kv_head * 128;
    auto load = [&](int j, const CUtensorMap* map, uint32_t full, uint32_t empty, uint32_t dst) {
      const int st = j & (PF_STAGES - 1), tok = block_of(j) * PF_KEYS;
      int y = k0 + tok;
      if (a.tables != nullptr) {
        const int blk = tok / a.block_size;
        y = max(0, __ldg(a.tables + static_cast<int64_t>(b) * a.bt_stride + min(blk, a.bt_width - 1))) * a.block_size + tok - blk * a.block_size;
        y = min(y, a.kv_rows - 1);  // (a bad table entry must not lead outside the cache)
      }
      if (!all_wait(empty + st * 8, ((j / PF_STAGES) & 1) ^ 1, B2_WAIT_SMEM_EMPTY)) return false;
      if (b2::elect_one()) {
        b2::mbar_arrive_expect_tx(full + st * 8, PF_KV);
        for (int i = 0; i < 2; ++i) b2::tma_load_2d(dst + st * PF_KV + i * (PF_KV / 2), map, full + st * 8, x + i * 64, y, b2::kEvictLast);
      }
      __syncwarp();
      return true;
    };
    // in the order of use: K of two blocks, then V of a block and K of the one after the next
    bool ok = load(0, &tmK, k_full, k_empty, s_k);
    if (n > 1) ok = ok && load(1, &tmK, k_full, k_empty, s_k);
    for (int j = 0; ok && j < n; ++j) {
      ok = load(j, &tmV, v_full, v_empty, s_v);
      if (j + 2 < n) ok = ok && load(j + 2, &tmK, k_full, k_empty, s_k);
    }
  } else if (warp <= 2) {
    const int h = warp - 1;
    const uint32_t idesc_s = b2::umma_idesc_bf16(PF_KEYS) | a.negate;
    constexpr uint32_t idesc_o = b2::umma_idesc_bf16(128) | (1u << 16);  // second operand MN-major
    const uint64_t desc_q = b2::umma_smem_desc(s_q + h * PF_Q), desc_k = b2::umma_smem_desc(s_k), desc_v = umma_smem_desc_mn(s_v);  // (addresses in 16 bytes)
    auto wait = [&](uint32_t bar, uint32_t phase, int code) {
      const bool ok = all_wait(bar, phase, code);
      b2::tc_fence_after();
      return ok;
    };
    auto scores = [&](int j) {
      const int st = j & (PF_STAGES - 1), buf = h * 2 + (j & 1);
      const bool ok = wait(k_full + st * 8, (j / PF_STAGES) & 1, B2_WAIT_SMEM_FULL);
      if (ok && b2::elect_one()) {
        const uint64_t dk = desc_k + st * (PF_KV >> 4);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          b2::umma_bf16(tmem + buf * PF_KEYS, desc_q + (k >> 2) * (PF_Q >> 5) + 2 * (k & 3), dk + (k >> 2) * (PF_KV >> 5) + 2 * (k & 3), idesc_s, k > 0 ? 1u : 0u);
        b2::umma_commit(s_full + buf * 8);
        b2::umma_commit(k_empty + st * 8);
      }
      __syncwarp();
      return ok;
    };
    bool ok = wait(q_full, 0, B2_WAIT_SMEM_FULL) && scores(0);
    if (n > 1) ok = ok && scores(1);
    for (int j = 0; ok && j < n; ++j) {
      const int st = j & (PF_STAGES - 1), buf = h * 2 + (j & 1);
      ok = wait(v_full + st * 8, (j / PF_STAGES) & 1, B2_WAIT_SMEM_FULL) && wait(p_full + buf * 8, (j >> 1) & 1, B2_WAIT_TMEM_EMPTY);
      if (!ok) break;
      if (b2::elect_one()) {
        const uint64_t dv = desc_v + st * (PF_KV >> 4);
#pragma unroll
        for (int k = 0; k < PF_KEYS / 16; ++k)  // 16 tokens: 8 columns of P, 2048 bytes of V
          umma_bf16_ts(tmem + 256 + h * 128, tmem + buf * PF_KEYS + k * 8, dv + k * (2048 >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
        b2::umma_commit(o_done + h * 8);
        b2::umma_commit(v_empty + st * 8);
        if (j == n - 1) b2::umma_commit(o_final + h * 8);
      }
      __syncwarp();
      // into the columns that P of this block is read from, once it has been
      if (j + 2 < n) ok = wait(o_done + h * 8, j & 1, B2_WAIT_TMEM_FULL) && scores(j + 2);
    }
  } else if (warp >= 4 && warp < 12) {
    const int h = (warp >> 2) - 1, q = warp & 3, row = q * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(q * 32) << 16;
    const int pos = shift + t0 + row;  // the last key this row sees
    float m = -INFINITY;               // the row's maximum, in units of scores
    float l[4] = {};                   // its sum, of columns 2 i and 2 i + 1 of every eight
    const uint64_t scale2 = pair_of(a.scale_log2, a.scale_log2);
    bool ok = true;
    for (int j = 0; ok && j < n; ++j) {
      const int buf = h * 2 + (j & 1);
      const uint32_t t_s = tmem + buf * PF_KEYS + lanes;
      // this block's scores, and without those that the row does not see
      uint32_t r[2][32];
      auto fetch = [&](int i) {
        const uint32_t at = tmem + (h * 2 + (i & 1)) * PF_KEYS + lanes;
        ok = all_wait(s_full + (h * 2 + (i & 1)) * 8, (i >> 1) & 1, B2_WAIT_TMEM_FULL);
        b2::tc_fence_after();
        b2::tmem_ld_32x32(at, r[0]);
        b2::tmem_ld_32x32(at + 32, r[1]);
        tc_wait_ld(r);
        const int last = min(pos, kv_len - 1) - block_of(i) * PF_KEYS;  // keys 0 .. last of the block count
        if (__any_sync(0xffffffffu, last < PF_KEYS - 1)) {
#pragma unroll
          for (int e = 0; e < 64; ++e)
            if (e > last) r[e >> 5][e & 31] = 0xff800000u;  // -inf
        }
      };
      float mx[4] = {m, m, m, m};
      auto maxima = [&]() {
#pragma unroll
        for (int e = 0; e < 64; e += 4)
#pragma unroll
          for (int i = 0; i < 4; ++i) mx[i] = fmaxf(mx[i], __uint_as_float(r[e >> 5][(e & 31) + i]));
      };
      if (PAIRS && j >= odd && ((j - odd) & 1) == 0) {  // the second of a pair is seen first for its maximum
        fetch(j + 1);
        maxima();
      }
      fetch(j);
      if (!PAIRS || j < odd || ((j - odd) & 1) == 0) maxima();
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const float f = top > m ? b2::ex2((m - top) * a.scale_log2) : 1.f;
      m = top;
      s_factor[h][j & 1][row] = f;
      __syncwarp();
      if (lane == 0) b2::mbar_arrive(f_full + (buf * 4 + q) * 8);
      const float ref = m == -INFINITY ? 0.f : m * a.scale_log2;
      const uint64_t ref2 = pair_of(-ref, -ref);
#pragma unroll
      for (int i = 0; i < 4; ++i) l[i] *= f;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t p[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float x, y;
          fma_pair(x, y, pair_of(__uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1])), scale2, ref2);
          x = b2::ex2(x);
          y = b2::ex2(y);
          l[(e >> 1) & 3] = l[(e >> 1) & 3] + x + y;
          p[e >> 1] = b2::pack_bf16(x, y);
        }
        tmem_st_32x16(t_s + c * 16, p);  // (this row has read its columns)
      }
      tc_wait_st();
      b2::tc_fence_before();
      __syncwarp();
      if (lane == 0) b2::mbar_arrive(p_full + buf * 8);
    }
    ok = all_wait(o_final + h * 8, 0, B2_WAIT_TMEM_FULL) && ok;
    b2::tc_fence_after();
    if (ok && !*abort_flag) {
      // rows leave through this head's part of the Q buffer (its last product is complete): whole 256-byte rows
      const float sum = (l[0] + l[2]) + (l[1] + l[3]), inv = sum > 0.f ? __fdividef(1.f, sum) : 0.f;
      const uint32_t t_o = tmem + 256 + h * 128 + lanes;
      unsigned char* mine = smem + h * PF_Q + q * 32 * 256;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[2][32];
        b2::tmem_ld_32x32(t_o + c * 64, r[0]);
        b2::tmem_ld_32x32(t_o + c * 64 + 32, r[1]);
        tc_wait_ld(r);
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            w[e] = b2::pack_bf16(__uint_as_float(r[g >> 2][(g & 3) * 8 + 2 * e]) * inv, __uint_as_float(r[g >> 2][(g & 3) * 8 + 2 * e + 1]) * inv);
          const int piece = c * 8 + g;
          *reinterpret_cast<uint4*>(mine + lane * 256 + ((piece ^ (lane & 15)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      __syncwarp();
#pragma unroll 4
      for (int i = 0; i < 16; ++i) {
        const int r = i * 2 + (lane >> 4), piece = lane & 15, t = t0 + q * 32 + r;
        if (t < q_len)
          *reinterpret_cast<uint4*>(a.out + (static_cast<int64_t>(q0 + t) * a.nq + head + h) * 128 + piece * 8) =
              *reinterpret_cast<const uint4*>(mine + r * 256 + ((piece ^ (r & 15)) << 4));
      }
    }
  } else if (warp >= 12) {
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(q * 32) << 16;
    bool ok = true;
    const int at = PAIRS && n > 1 ? 1 - odd : 0;  // where in the walk the last block of the keys is
    if (n * PF_KEYS > kv_len) {
      // Rows past the sequence's last key count as zero: in the cache they may hold anything, in a matrix they are the next
      // sequence's, and a probability of zero times Inf or NaN is NaN.
      ok = all_wait(v_full + at * 8, 0, B2_WAIT_SMEM_FULL);
      const int key = row & 63;
      if ((n - 1) * PF_KEYS + key >= kv_len) {
        unsigned char* v = smem + (s_v - s_q) + at * PF_KV + (row >> 6) * (PF_KV / 2) + key * 128;
#pragma unroll
        for (int i = 0; i < 8; ++i)  // (another piece of every row of eight, so that they do not meet in a bank)
          *reinterpret_cast<uint4*>(v + ((i ^ key) & 7) * 16) = make_uint4(0, 0, 0, 0);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    for (int j = 0; ok && j < n; ++j)
      for (int h = 0; ok && h < 2; ++h) {
        const int buf = h * 2 + (j & 1);
        ok = all_wait(f_full + (buf * 4 + q) * 8, (j >> 1) & 1, B2_WAIT_TMEM_FULL);
        const float f = s_factor[h][j & 1][row];
        if (ok && j > 0) ok = all_wait(o_done + h * 8, (j - 1) & 1, B2_WAIT_TMEM_FULL);  // (every phase is seen: none is taken for the one before)
        if (ok && j > 0 && __any_sync(0xffffffffu, f != 1.f)) {
          b2::tc_fence_after();
          const uint32_t t_o = tmem + 256 + h * 128 + lanes;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t r[2][32];
            b2::tmem_ld_32x32(t_o + c * 64, r[0]);
            b2::tmem_ld_32x32(t_o + c * 64 + 32, r[1]);
            tc_wait_ld(r);
#pragma unroll
            for (int e = 0; e < 64; ++e) r[e >> 5][e & 31] = __float_as_uint(__uint_as_float(r[e >> 5][e & 31]) * f);
#pragma unroll
            for (int i = 0; i < 4; ++i) tmem_st_32x16(t_o + c * 64 + i * 16, &r[i >> 1][(i & 1) * 16]);
          }
          tc_wait_st();
          b2::tc_fence_before();
        }
        __syncwarp();
        if (lane == 0) b2::mbar_arrive(p_full + buf * 8);
      }
  }

  __syncwarp();
  b2::tc_fence_before();
  __syncthreads();
  b2::tc_fence_after();
  const int aborted = *abort_flag;
  if (aborted) {
    for (int i = 0; i < 100; ++i) __nanosleep(2000);  // copies in flight land before the CTA leaves
    if (threadIdx.x == 0) b2::report_timeout(a.status, aborted);
  }
  if (warp == 1) b2::tmem_dealloc(tmem, 512);
}

// Softmax scale * log2(e) for kernels that mask and compare scores before they scale them: its size - masked scores are -inf, and -inf times
// zero is none -, with the query negated in a negative one's place, which changes no product but for its sign.
float scale_size(float scale) { return std::max(fabsf(scale * 1.4426950408889634f), FLT_MIN); }

constexpr size_t ATT_SMEM_LIMIT = 113 * 1024;  // two CTAs per SM (228 KB, 1 KB of it reserved per CTA)
constexpr size_t attention_smem(int n_seqs, int group) {
  return 1024 + ATT_STAGES * ATT_STAGE_BYTES + static_cast<size_t>(ATT_WARPS) * group * ATT_HD * sizeof(float) + (2 * static_cast<size_t>(n_seqs) + 1) * sizeof(int);
}
static_assert(attention_smem(ATT_MAX_SEQS, ATT_MAX_GROUP) + 512 <= ATT_SMEM_LIMIT, "the ring, the warps' parts and the batch fit (512: static)");

// the opt-in to more than 48 KB of dynamic shared memory belongs to a device, not to the process
int configure_once() {
  static std::atomic<bool> done[64];
  int dev = 0;
  B2_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return b2::set_error(B2_ERR_UNSUPPORTED, "device ordinal %d not supported", dev);
  if (!done[dev].load(std::memory_order_acquire)) {
    B2_CUDA(cudaFuncSetAttribute(paged_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM_LIMIT));
    B2_CUDA(cudaFuncSetAttribute(paged_decode_wide_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, wide_smem(4)));
    B2_CUDA(cudaFuncSetAttribute(paged_decode_wide_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, wide_smem(WD_MAX_STAGES)));
    B2_CUDA(cudaFuncSetAttribute(prefill_attention_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM));
    B2_CUDA(cudaFuncSetAttribute(prefill_attention_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM));
    done[dev].store(true, std::memory_order_release);
  }
  return B2_OK;
}

}  // namespace

extern "C" {

int b2_paged_attention_supported(int n_seqs, int nq, int nkv, int head_dim, int block_size) {
  return n_seqs > 0 && n_seqs <= ATT_MAX_SEQS && nkv > 0 && nq % nkv == 0 && nq / nkv <= WD_MAX_GROUP && head_dim == ATT_HD && block_size % ATT_TILE == 0 &&
         n_seqs <= B2_ATTN_MAX_ITEMS / nkv && (nq / nkv <= ATT_MAX_GROUP || n_seqs * nkv >= WD_MIN_ITEMS);
}

int b2_paged_attention_decode(b2_ctx* ctx, const void* q, int64_t q_stride, const void* k_cache, const void* v_cache, int num_blocks, int block_size,
                              const int32_t* block_tables, int64_t bt_stride, int bt_width, const int32_t* context_lens, int n_seqs, int nq, int nkv,
                              int head_dim, float scale, void* out, void* stream) {
  if (ctx == nullptr || n_seqs < 0 || nq <= 0 || nkv <= 0 || bt_width <= 0 || block_size <= 0 || num_blocks <= 0) return B2_ERR_ARG;
  if (n_seqs == 0) return B2_OK;
  if (!b2_paged_attention_supported(n_seqs, nq, nkv, head_dim, block_size)) return B2_ERR_UNSUPPORTED;
  if (!q || !k_cache || !v_cache || !block_tables || !context_lens || !out) return B2_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) | reinterpret_cast<uintptr_t>(out)) & 15)
    return B2_ERR_ARG;
  if (q_stride % 8 != 0 || q_stride < static_cast<int64_t>(nq) * head_dim || bt_stride < bt_width) return B2_ERR_ARG;
  AttnArgs a{};
  a.q = static_cast<const uint16_t*>(q);
  a.q_stride = q_stride;
  a.tables = block_tables;
  a.bt_stride = bt_stride;
  a.bt_width = bt_width;
  a.block_size = block_size;
  a.num_blocks = num_blocks;
  a.status = ctx->status_dev;
  a.lens = context_lens;
  a.n_seqs = n_seqs;
  a.nkv = nkv;
  a.group = nq / nkv;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.out = static_cast<uint16_t*>(out);
  a.ws = ctx->attn_ws;
  a.counters = ctx->attn_counters;
  CUtensorMap maps[4];
  const uint64_t width = static_cast<uint64_t>(nkv) * head_dim, tokens = static_cast<uint64_t>(num_blocks) * block_size;
  for (int i = 0; i < 4; ++i) {
    const int rc = b2::encode_tmap_2d(&maps[i], i & 1 ? v_cache : k_cache, width, tokens, static_cast<int64_t>(width), 64, i < 2 ? ATT_TILE : 16);
    if (rc != B2_OK) return rc;
  }
  const int64_t most = static_cast<int64_t>(n_seqs) * nkv * ((static_cast<int64_t>(bt_width) * block_size + ATT_TILE - 1) / ATT_TILE);
  const int grid = static_cast<int>(std::min<int64_t>(most, static_cast<int64_t>(ctx->num_sms) * ATT_CTAS_PER_SM));
  const int crc = configure_once();
  if (crc != B2_OK) return crc;
  const int items = n_seqs * nkv;
  if (a.group > ATT_MAX_GROUP) {
    const bool few = items <= 2 * ctx->num_sms;
    a.flip = scale < 0.f ? 0x80008000u : 0u;
    a.scale_log2 = scale_size(scale);
    a.stages = items <= ctx->num_sms ? WD_MAX_STAGES : few ? 6 : items <= 3 * ctx->num_sms ? 4 : 3;
    const auto kernel = few ? paged_decode_wide_kernel<true> : paged_decode_wide_kernel<false>;
    B2_CUDA(b2_launch(kernel, dim3(items), dim3(ATT_THREADS), wide_smem(a.stages), static_cast<cudaStream_t>(stream), maps[0], maps[1], maps[2], maps[3], a));
    return B2_OK;
  }
  const size_t smem = attention_smem(n_seqs, a.group);
  B2_CUDA(b2_launch(paged_decode_kernel, dim3(grid), dim3(ATT_THREADS), smem, static_cast<cudaStream_t>(stream), maps[0], maps[1], maps[2], maps[3], a));
  return B2_OK;
}

// An even number of query heads per KV head: a CTA's two tiles of scores are those of two heads with the same keys.
int b2_prefill_attention_supported(int nq, int nkv, int head_dim, int block_size) {
  return nkv > 0 && nq > 0 && nq % (2 * nkv) == 0 && nq <= 65534 && head_dim == 128 && (block_size <= 0 || block_size % 128 == 0);
}

int b2_prefill_attention(b2_ctx* ctx, const void* q, int64_t q_stride, const void* k, const void* v, int64_t kv_stride, int64_t kv_rows,
                         const int32_t* block_tables, int64_t bt_stride, int bt_width, int block_size, const int32_t* cu_q, const int32_t* cu_k,
                         int n_seqs, int max_q, int tokens, int nq, int nkv, int head_dim, float scale, void* out, void* stream) {
  if (ctx == nullptr || n_seqs < 0 || tokens < 0 || nq <= 0 || nkv <= 0 || max_q < 0) return B2_ERR_ARG;
  if (n_seqs == 0 || tokens == 0 || max_q == 0) return B2_OK;
  if (!b2_prefill_attention_supported(nq, nkv, head_dim, block_tables != nullptr ? block_size : 0) || n_seqs > 65535 || kv_rows > (1 << 30)) return B2_ERR_UNSUPPORTED;
  if (!q || !k || !v || !cu_q || !cu_k || !out || kv_rows <= 0) return B2_ERR_ARG;
  if (block_tables != nullptr && (bt_width <= 0 || bt_stride < bt_width || block_size <= 0)) return B2_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15) return B2_ERR_ARG;
  if (q_stride % 8 != 0 || kv_stride % 8 != 0 || q_stride < static_cast<int64_t>(nq) * head_dim || kv_stride < static_cast<int64_t>(nkv) * head_dim) return B2_ERR_ARG;
  const int crc = configure_once();
  if (crc != B2_OK) return crc;
  CUtensorMap tmQ, tmK, tmV;
  int rc = b2::encode_tmap_2d(&tmQ, q, static_cast<uint64_t>(nq) * head_dim, tokens, q_stride, 64, PF_ROWS);
  if (rc == B2_OK) rc = b2::encode_tmap_2d(&tmK, k, static_cast<uint64_t>(nkv) * head_dim, kv_rows, kv_stride, 64, PF_KEYS);
  if (rc == B2_OK) rc = b2::encode_tmap_2d(&tmV, v, static_cast<uint64_t>(nkv) * head_dim, kv_rows, kv_stride, 64, PF_KEYS);
  if (rc != B2_OK) return rc;
  PrefillArgs a{};
  a.cu_q = cu_q;
  a.cu_k = cu_k;
  a.tables = block_tables;
  a.bt_stride = bt_stride;
  a.bt_width = bt_width;
  a.block_size = block_size;
  a.kv_rows = static_cast<int>(kv_rows);
  a.nq = nq;
  a.out = static_cast<uint16_t*>(out);
  a.negate = scale < 0.f ? b2::kUmmaNegateA : 0u;
  a.scale_log2 = scale_size(scale);
  a.status = ctx->status_dev;
  a.group = nq / nkv;
  const auto kernel = block_tables != nullptr && a.group > 2 ? prefill_attention_kernel<true> : prefill_attention_kernel<false>;
  B2_CUDA(b2_launch(kernel, dim3(nq / 2, n_seqs, (max_q + PF_ROWS - 1) / PF_ROWS), dim3(PF_THREADS), PF_SMEM, static_cast<cudaStream_t>(stream),
                    tmQ, tmK, tmV, a));
  return B2_OK;
}

}  // extern "C"
