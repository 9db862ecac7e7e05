// Decode attention over the paged KV cache: one new query token per sequence, grouped-query heads.
#include <algorithm>
#include <atomic>

#include "b2_common.cuh"

namespace {

// ---------------------------------------------------------------------------
// paged_decode_kernel
//
// Bound: HBM.  Every K and V row of every context is read once (512 bytes per token and KV head) and used for the
// G = nq / nkv query heads of its group; nothing else of size moves.
//
// One warp brings the tiles (64 tokens of one (sequence, KV head): 16 KB of K, 16 KB of V) into a 3-stage ring by TMA (2
// stages where 8 heads share a KV head) and runs ahead over the borders between heads and sequences, so that two CTAs per
// SM keep up to 190 KB in flight; four warps
// take 16 tokens each from a landed tile (ldmatrix, mma.sync.m16n8k16 with the 8 upper rows empty: the tensor pipe is idle
// most of the time anyway) and keep their own running maximum and sum.  The rows of a context's last tile come in
// groups of 16, so that little is read past its end.
//
// Work split: the tiles of the whole batch, in the order (sequence, head, position), are dealt in contiguous equal ranges
// to the CTAs - the contexts' lengths are read on the device, so a captured graph stays balanced for any batch.  A
// (sequence, head) that spans several CTAs is combined by whichever of them finishes last; a CTA holds at most two such
// parts and settles both at its end.
// ---------------------------------------------------------------------------
constexpr int ATT_WARPS = 4, ATT_THREADS = (ATT_WARPS + 1) * 32;  // the last warp is the producer
constexpr int ATT_TILE = 64;          // tokens per tile
constexpr int ATT_HD = 128;           // head dimension
constexpr int ATT_ROWS = 8;           // query heads of a group the fragments have room for
// Served: groups of one and two heads.  (The kernel is faster than flash-attn's for 4 and 8 heads too: 53 us against 71 at 64
// contexts of 1056 tokens.  But its last bits differ, and over the 36 layers of a 4096-wide model, every one of which rounds
// to bf16 some ten times, that grows to 3 % of the hidden state; such models keep the results they had.)
constexpr int ATT_MAX_GROUP = 2;
constexpr int ATT_CTAS_PER_SM = 2;
constexpr int ATT_MAX_STAGES = 3;
constexpr int ATT_HALF_BYTES = ATT_TILE * 128;          // 64 tokens x 64 dimensions: one swizzled box
constexpr int ATT_STAGE_BYTES = 4 * ATT_HALF_BYTES;     // K dimensions 0..63, 64..127, V the same
constexpr int ATT_SLOT = ATT_ROWS * ATT_HD + 2 * ATT_ROWS;  // floats of one partial result: O, then the maxima and sums
constexpr int ATT_MAX_SEQS = 1024;
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
  int bt_width, block_size, num_blocks, n_seqs, nkv, group, stages;
  float scale_log2;  // softmax scale * log2(e)
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// rows 8..15 of A are zero: only the first two accumulators carry data
__device__ __forceinline__ void mma_rows8(float& c0, float& c1, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm("{\n\t.reg .f32 d2, d3;\n\t"
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, d2, d3}, {%2, %3, %4, %3}, {%5, %6}, {%0, %1, %7, %7};\n\t}"
      : "+f"(c0), "+f"(c1)
      : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}
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
  float* s_o = reinterpret_cast<float*>(smem + a.stages * ATT_STAGE_BYTES);  // [warp][head of the group][ATT_HD]
  int* first_tile = reinterpret_cast<int*>(s_o + ATT_WARPS * a.group * ATT_HD);
  int* s_len = first_tile + a.n_seqs + 1;
  __shared__ float s_m[ATT_WARPS][ATT_ROWS], s_l[ATT_WARPS][ATT_ROWS];
  __shared__ __align__(8) uint64_t s_bars[2 * ATT_MAX_STAGES];
  __shared__ int s_abort, s_last[2];
  volatile int* abort_flag = &s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar_full = b2::smem_u32(s_bars), bar_empty = bar_full + ATT_MAX_STAGES * 8;
  if (tid == 0) {
    b2::tma_prefetch_desc(&tmK);
    b2::tma_prefetch_desc(&tmV);
    for (int i = 0; i < a.stages; ++i) {
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
    int mine = 0;
#pragma unroll 4
    for (int i = 0; i < per; ++i)
      if (s0 + i < a.n_seqs) {
        const int len = max(0, min(__ldg(a.lens + s0 + i), max_len));
        const int t = max(1, (len + ATT_TILE - 1) / ATT_TILE);  // a padded row has one tile too: its output is zero
        s_len[s0 + i] = len;
        first_tile[s0 + i + 1] = t;
        mine += t;
      }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    int at = incl - mine;
    if (lane == 0) first_tile[0] = 0;
    for (int i = 0; i < per; ++i)
      if (s0 + i < a.n_seqs) first_tile[s0 + i + 1] = at += first_tile[s0 + i + 1];
  }
  __syncthreads();
  const int total = first_tile[a.n_seqs] * a.nkv;
  const int ctas = min(static_cast<int>(gridDim.x), total);
  const int cta = blockIdx.x;
  if (cta >= ctas) return;
  const int base = total / ctas, rem = total % ctas;
  auto begin_of = [&](int i) { return i * base + min(i, rem); };
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
            const int groups = (left + 15) >> 4;  // none for a padded row
            b2::mbar_arrive_expect_tx(fb, groups * (ATT_STAGE_BYTES / 4));
            for (int i = 0; i < groups; ++i) {
              const uint32_t d = dst + i * 16 * 128;
              b2::tma_load_2d(d, &tmK16, fb, x, y + i * 16, b2::kEvictFirst);
              b2::tma_load_2d(d + ATT_HALF_BYTES, &tmK16, fb, x + 64, y + i * 16, b2::kEvictFirst);
              b2::tma_load_2d(d + 2 * ATT_HALF_BYTES, &tmV16, fb, x, y + i * 16, b2::kEvictFirst);
              b2::tma_load_2d(d + 3 * ATT_HALF_BYTES, &tmV16, fb, x + 64, y + i * 16, b2::kEvictFirst);
            }
          }
          if (++stage == a.stages) { stage = 0; phase ^= 1; }
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
          ldmatrix_x4(kf, k_row + (k >> 2) * ATT_HALF_BYTES + ((((k & 3) * 2 + k_chunk) ^ (k_tok & 7)) << 4));
          mma_rows8(s[0][0], s[0][1], qf[k][0], qf[k][1], kf[0], kf[1]);
          mma_rows8(s[1][0], s[1][1], qf[k][0], qf[k][1], kf[2], kf[3]);
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
            p[i][e] = exp2f(s[i][e] - m);
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
          ldmatrix_x4_trans(vf, v_row + (j >> 2) * ATT_HALF_BYTES + ((((j & 3) * 2 + v_chunk) ^ (v_tok & 7)) << 4));
          mma_rows8(o[2 * j][0], o[2 * j][1], p0, p1, vf[0] & keep[0], vf[1] & keep[1]);
          mma_rows8(o[2 * j + 1][0], o[2 * j + 1][1], p0, p1, vf[2] & keep[0], vf[3] & keep[1]);
        }
      }
      __syncwarp();
      if (lane == 0) b2::mbar_arrive(bar_empty + stage * 8);
      if (++stage == a.stages) { stage = 0; phase ^= 1; }
    }

    // ---- the four warps' parts meet in shared memory ----
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    consumers_meet();  // the previous segment's parts have been read
    if (c == 0) {
      s_m[warp][g] = m;
      s_l[warp][g] = l;
    }
    if (g < a.group) {
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
          slot[ATT_ROWS * ATT_HD + r] = mx;
          slot[ATT_ROWS * ATT_HD + ATT_ROWS + r] = sum;
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
              pm[k] = b2::ld_cg_f32(part(k) + ATT_ROWS * ATT_HD + r);
              ps[k] = b2::ld_cg_f32(part(k) + ATT_ROWS * ATT_HD + ATT_ROWS + r);
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
        for (int k = lane; k < n; k += 32) mx = fmaxf(mx, b2::ld_cg_f32(part(k) + ATT_ROWS * ATT_HD + r));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        for (int k = lane; k < n; k += 32) {
          const float f = mx == -INFINITY ? 0.f : exp2f(b2::ld_cg_f32(part(k) + ATT_ROWS * ATT_HD + r) - mx);
          s_o[r * (ATT_WARPS * ATT_HD) + k] = f;
          sum += f * b2::ld_cg_f32(part(k) + ATT_ROWS * ATT_HD + ATT_ROWS + r);
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
  if (*abort_flag && tid == 0) b2::report_timeout(a.status, *abort_flag);
}

// dynamic shared memory, and the deepest ring with which two CTAs fit an SM (228 KB, 1 KB of it reserved per CTA)
size_t attention_smem(int n_seqs, int group, int& stages) {
  const size_t rest = 1024 + static_cast<size_t>(ATT_WARPS) * group * ATT_HD * sizeof(float) + (2 * static_cast<size_t>(n_seqs) + 1) * sizeof(int);
  stages = rest + ATT_MAX_STAGES * ATT_STAGE_BYTES + 512 <= 113 * 1024 ? ATT_MAX_STAGES : 2;
  return rest + stages * ATT_STAGE_BYTES;
}

// the opt-in to more than 48 KB of dynamic shared memory belongs to a device, not to the process
int configure_once() {
  static std::atomic<bool> done[64];
  int dev = 0;
  B2_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return b2::set_error(B2_ERR_UNSUPPORTED, "device ordinal %d not supported", dev);
  if (!done[dev].load(std::memory_order_acquire)) {
    B2_CUDA(cudaFuncSetAttribute(paged_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 113 * 1024));
    done[dev].store(true, std::memory_order_release);
  }
  return B2_OK;
}

}  // namespace

extern "C" {

int b2_paged_attention_supported(int n_seqs, int nq, int nkv, int head_dim, int block_size) {
  return n_seqs > 0 && n_seqs <= ATT_MAX_SEQS && nkv > 0 && nq % nkv == 0 && nq / nkv <= ATT_MAX_GROUP && head_dim == ATT_HD && block_size % ATT_TILE == 0 &&
         n_seqs <= B2_ATTN_MAX_ITEMS / nkv;
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
  const size_t smem = attention_smem(n_seqs, a.group, a.stages);
  const int crc = configure_once();
  if (crc != B2_OK) return crc;
  B2_CUDA(b2_launch(paged_decode_kernel, dim3(grid), dim3(ATT_THREADS), smem, static_cast<cudaStream_t>(stream), maps[0], maps[1], maps[2], maps[3], a));
  return B2_OK;
}

}  // extern "C"
