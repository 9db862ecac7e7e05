// bf16 GEMM for more than a decode step's tokens: C[M, N] = A[M, K] W[N, K]^T with the store epilogues (bias, SiLU(gate) * up
// on interleaved pairs, the head work of the qkv projection).
//
// One CTA pair (tcgen05.mma.cta_group::2) computes a tile of 256 features x bn tokens, bn <= 256 in steps of 32 chosen per
// problem (16 for whole tiles).  Weights fill the 256-row side, so a batch of any size wastes at most 31 token columns a tile; each CTA of the pair stages
// its own 128 weight rows and half of the tokens, which both tensor cores read.  Two instances:
//   MULTI   more tiles than SM pairs, or a long ring: one CTA per SM, the pair walks its tiles with two accumulators in
//           tensor memory, so that 8 epilogue warps store a tile under the next one's MMAs (with 2 CTAs per SM and one tile
//           each, the pairs run in step and every epilogue is exposed: 642 us instead of 545 at 4096 x 24576 x 4096);
//           What is left after the whole rounds is dealt out in equal ranges of K blocks, wherever these begin inside a
//           tile; the parts of a tile are added up in fp32 in L2 and whoever arrives last stores it (nobody waits).
//   single  one tile, or a share of one, per pair; 4 epilogue warps.  Where little is staged the CTA takes at most half of the
//           SM's memories, so that its set-up and first weight loads run under the neighbouring kernels of the stream.
//
// When there are too few tiles to fill the chip the K range is split over `split` pairs of one cluster (2, 3 or 4): after
// the main loop every pair hands the accumulator columns that others own to them through distributed shared memory (the ring
// is free by then), adds what it received to its own and stores its share.
//
// The TMA and the MMA warp walk with all their lanes and elect a thread to issue.  The instructions take descriptors, coordinates and barriers
// from uniform registers; in code that one lane runs alone the compiler moves every operand there anew, and a K block took 585 clocks of
// issue whatever its width (the tensor pipe wants 128 at 64 tokens, 512 at 256).  It is 310 at 64 and 333 at 160 tokens now: 391 tokens
// x 6144 x 4096 28.8 -> 21.4 us, 777 x 24576 x 4096 150 -> 130, 256 x 4096 x 1024 10.6 -> 8.0.
//
// The accumulator has features in lanes and tokens in columns.  It leaves tensor memory in the 16x256b shape, whose
// fragments are those of stmatrix: a transposing stmatrix puts 8 features of one token next to each other, and rows of
// 32 features per warp (64 bytes), or of 128 (one attention head) per four warps, go out of shared memory.
#include <algorithm>
#include <atomic>

#include "b2_common.cuh"

namespace {

constexpr int FM = 128;               // features per CTA
constexpr int BK = 64;                // K block
template <bool MULTI>
struct Shape {
  static constexpr int EW = MULTI ? 8 : 4;            // epilogue warps
  static constexpr int THREADS = 64 + EW * 32;        // and one warp each for TMA and MMA
  static constexpr int ACC = MULTI ? 2 : 1;           // accumulators in tensor memory
  static constexpr uint32_t OUT_BYTES = EW * 4096;    // staging: two buffers of 32 tokens x 128 features per 4 warps
};
constexpr int MAX_STAGES = 12;
constexpr int MAX_SPLIT = 4;
constexpr uint32_t W_BYTES = FM * BK * 2;
constexpr uint32_t SMEM_HALF = 113 * 1024, SMEM_ALL = 227 * 1024;  // two CTAs per SM, one
constexpr uint32_t SMEM_EXTRA = 1024 + 256 + 1024;  // alignment, barriers, positions of the tile's tokens
constexpr uint64_t PIPE_LIMIT_NS = 1000000000ull;

struct TileArgs {
  uint16_t* C;
  int64_t ldc;
  const uint16_t* bias;
  B2Status* status;
  int M, N, kblocks;
  int bn, stages, split;
  int rounds, ranged;         // MULTI: whole tiles per pair; tiles after those, dealt out by K blocks
  float* ws;                  // MULTI: one fp32 slot of 128 x 256 per CTA, zero between launches
  int* counters;              // MULTI: arrivals per (tile, side, set of warps), zero between launches
  int tilesF, tilesT, group;  // 256-feature tiles, token tiles, token tiles visited together
  uint32_t out_off, bar_off;  // shared memory: staging, barriers
  unsigned long long* trace;  // optional [trace_ctas][8][2] (SM clock, global ns) phase stamps
  int trace_ctas;
  int silu_pairs;
  // head work of the qkv projection (128-wide heads)
  int qkv_fused, nq, nkv;
  const int64_t* positions;
  const float* cos_sin;
  const uint16_t* q_norm_w;
  const uint16_t* k_norm_w;
  float qk_eps;
  uint16_t* k_cache;
  uint16_t* v_cache;
  const int32_t* slots;
};

// 16 lanes x 32 fp32 columns: thread t gets, of 8-column group i, columns 2 (t % 4), +1 of lane t / 4 in r[4 i], r[4 i + 1]
// and of lane t / 4 + 8 in r[4 i + 2], r[4 i + 3]
__device__ __forceinline__ void tmem_ld_16x256_x4(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_16x256_x1(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// the four epilogue warps that share a staging buffer
__device__ __forceinline__ void quad_meets(int part) {
  if (part == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}
// token t of a staging buffer of head rows: 16 pieces of 16 bytes, piece index XORed with the token so that neither the
// transposing stores nor the row reads meet in a bank
__device__ __forceinline__ uint32_t staged(int token, int piece) { return token * (FM * 2) + ((piece ^ (token & 7)) << 4); }

__device__ __forceinline__ void stamp(const TileArgs& a, int slot) {
  if (a.trace != nullptr && static_cast<int>(blockIdx.x) < a.trace_ctas) {
    unsigned long long* t = a.trace + (static_cast<size_t>(blockIdx.x) * 8 + slot) * 2;
    t[0] = static_cast<unsigned long long>(clock64());
    t[1] = b2::globaltimer_ns();
  }
}

// The remaining tiles' K blocks (of a split tile: its own) in one range per pair, the first `rem` of them one block longer.
struct Ranges {
  int len, rem;
  __host__ __device__ __forceinline__ Ranges(int units, int pairs) : len(units / pairs), rem(units % pairs) {}
  __host__ __device__ __forceinline__ int begin(int pair) const { return pair * len + (pair < rem ? pair : rem); }
  __host__ __device__ __forceinline__ int holder(int unit) const {
    const int big = rem * (len + 1);
    return unit < big ? unit / (len + 1) : rem + (unit - big) / len;
  }
};
// What a pair works through: `rounds` whole tiles, then its range of the remaining tiles' K blocks, tile by tile.  (The
// single instance: its share of the one tile.)
struct Walk {
  int pairs, pair, rounds, whole, kblocks, t, u, u1;  // whole: tiles dealt out whole; u: position in the remaining tiles' K blocks
  int tile, k0, k1;
  __host__ __device__ __forceinline__ bool next() {
    if (pair + t * pairs < whole) {
      tile = pair + t * pairs;
      k0 = 0;
      k1 = kblocks;
      ++t;
      return true;
    }
    if (u >= u1) return false;
    tile = u / kblocks;
    k0 = u - tile * kblocks;
    tile += rounds * pairs;
    k1 = k0 + u1 - u < kblocks ? k0 + u1 - u : kblocks;
    u += k1 - k0;
    return true;
  }
};
// grid_pair: of `pairs` in the grid; cluster_pair: of the `split` that share a tile (single instance)
template <bool MULTI>
__host__ __device__ __forceinline__ Walk first_walk(const Ranges& r, int pairs, int grid_pair, int cluster_pair, int kblocks, int rounds, int ranged, int tiles) {
  Walk w;
  w.pairs = pairs;
  w.pair = grid_pair;
  w.kblocks = kblocks;
  w.t = 0;
  w.rounds = MULTI ? rounds : 0;
  w.whole = MULTI ? (ranged > 0 ? rounds * pairs : tiles) : 0;
  w.u = r.begin(MULTI ? grid_pair : cluster_pair);
  w.u1 = r.begin((MULTI ? grid_pair : cluster_pair) + 1);
  return w;
}
__device__ __forceinline__ void ld_cg_f4(uint32_t* r, const float* p) {
  asm volatile("ld.global.cg.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void red_add_f4(float* p, const uint32_t* r) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(__uint_as_float(r[0])), "f"(__uint_as_float(r[1])), "f"(__uint_as_float(r[2])),
               "f"(__uint_as_float(r[3])) : "memory");
}

template <bool MULTI>
__global__ void __launch_bounds__(Shape<MULTI>::THREADS, MULTI ? 1 : 2)
gemm_tile_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const TileArgs a) {
  using T = Shape<MULTI>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t smem_base = b2::smem_u32(smem);
  const uint32_t stage_bytes = W_BYTES + a.bn * (BK * 2 / 2);  // this CTA's weights and its half of the tokens
  const uint32_t bar_full = smem_base + a.bar_off;             // used in the pair's even CTA: bytes of both CTAs' loads
  const uint32_t bar_empty = bar_full + MAX_STAGES * 8;        // in each CTA: its stage may be refilled
  const uint32_t bar_done = bar_empty + MAX_STAGES * 8;        // in each CTA: accumulator complete
  const uint32_t bar_drained = bar_done + 2 * 8;               // used in the even CTA: both CTAs' epilogues have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + a.bar_off + (2 * MAX_STAGES + 4) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = MULTI ? 1 : a.split;
  const int cr = static_cast<int>(b2::cluster_ctarank());
  const int pair = cr >> 1, side = cr & 1;  // side 0 issues the pair's MMAs
  // a tile's first feature of this CTA, and its first token: token tiles in groups, features across, tokens of a group inside
  auto place = [&](int tile, int& f0, int& tok0) {
    const int per_group = a.group * a.tilesF;
    const int grp = tile / per_group, first_t = grp * a.group;
    const int in_grp = tile - grp * per_group, width = min(a.group, a.tilesT - first_t);
    const int ft = in_grp / width;
    f0 = ft * 2 * FM + side * FM;
    tok0 = (first_t + in_grp - ft * width) * a.bn;
  };
  const int pairs = gridDim.x / 2;
  const Ranges ranges(MULTI ? a.ranged * a.kblocks : a.kblocks, MULTI ? pairs : S);
  const Walk first = first_walk<MULTI>(ranges, pairs, blockIdx.x / 2, pair, a.kblocks, a.rounds, a.ranged, a.tilesF * a.tilesT);
  auto next = [&](Walk& w) {
    const bool any = w.next();
    if (!MULTI) w.tile = blockIdx.x / (2 * S);
    return any;
  };
  const int STAGES = a.stages;

  if (threadIdx.x == 0) {
    stamp(a, 7);
    b2::tma_prefetch_desc(&tmW);
    b2::tma_prefetch_desc(&tmX);
    for (int s = 0; s < STAGES; ++s) {
      b2::mbar_init(bar_full + s * 8, 1);
      b2::mbar_init(bar_empty + s * 8, 1);
    }
    for (int i = 0; i < T::ACC; ++i) {
      b2::mbar_init(bar_done + i * 8, 1);
      b2::mbar_init(bar_drained + i * 8, 2 * T::EW);
    }
    *abort_flag = 0;
    b2::mbar_fence_init();
  }
  const uint32_t acc_cols = a.bn <= 32 ? 32u : a.bn <= 64 ? 64u : a.bn <= 128 ? 128u : 256u;
  const uint32_t tmem_cols = T::ACC * acc_cols;
  if (warp == 1) {
    b2::tmem_alloc_pair(b2::smem_u32(tmem_slot), tmem_cols);
    b2::tmem_relinquish_pair();
  }
  b2::tc_fence_before();
  __syncthreads();
  // the other CTA's barriers must exist before anything is counted on them
  b2::cluster_arrive();
  b2::cluster_wait();
  b2::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  b2::pdl_launch_dependents();
  if (threadIdx.x == 0) stamp(a, 0);

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs): the whole warp walks, one thread issues ----------------
    const uint32_t full0 = b2::map_to_cta(bar_full, cr & ~1);  // the even CTA's "full" barriers, as a cluster address
    const int x_half = side * (a.bn >> 1);
    Walk w = first;
    int f0 = 0, tok0 = 0, pre = 0;
    if (next(w)) {
      place(w.tile, f0, tok0);
      pre = min(w.k1 - w.k0, STAGES);
    } else {
      w.k0 = w.k1 = 0;
    }
    if (b2::elect_one()) {
      for (int i = 0; i < pre; ++i) {  // weights depend on no earlier kernel
        if (side == 0) b2::mbar_arrive_expect_tx(bar_full + i * 8, 2 * stage_bytes);
        b2::tma_load_2d_pair(smem_base + i * stage_bytes, &tmW, full0 + i * 8, (w.k0 + i) * BK, f0, b2::kEvictNormal);
      }
    }
    __syncwarp();
    b2::pdl_wait();
    if (lane == 0) stamp(a, 3);
    if (b2::elect_one()) {
      for (int i = 0; i < pre; ++i) b2::tma_load_2d_pair(smem_base + i * stage_bytes + W_BYTES, &tmX, full0 + i * 8, (w.k0 + i) * BK, tok0 + x_half, b2::kEvictNormal);
    }
    __syncwarp();
    int stage = pre == STAGES ? 0 : pre;
    uint32_t phase = pre == STAGES ? 1 : 0;
    int kb = w.k0 + pre;
    for (;;) {
      if (kb == w.k1) {
        if (!next(w)) break;
        place(w.tile, f0, tok0);
        kb = w.k0;
      }
      if (!__all_sync(0xffffffffu, b2::mbar_wait(bar_empty + stage * 8, phase ^ 1, abort_flag, PIPE_LIMIT_NS, B2_WAIT_SMEM_EMPTY))) break;
      if (b2::elect_one()) {
        const uint32_t dst = smem_base + stage * stage_bytes;
        if (side == 0) b2::mbar_arrive_expect_tx(bar_full + stage * 8, 2 * stage_bytes);
        b2::tma_load_2d_pair(dst, &tmW, full0 + stage * 8, kb * BK, f0, b2::kEvictNormal);
        b2::tma_load_2d_pair(dst + W_BYTES, &tmX, full0 + stage * 8, kb * BK, tok0 + x_half, b2::kEvictNormal);
      }
      __syncwarp();
      ++kb;
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (even CTA of each pair): the whole warp walks, one thread issues ----------------
    if (side == 0) {
      const uint32_t idesc = b2::umma_idesc_bf16_pair(a.bn);
      const uint16_t both = static_cast<uint16_t>(3u << (cr & ~1));
      b2::pdl_wait();  // the pipeline's time limit must not include the wait for earlier kernels
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Walk w = first;
      for (int t = 0; ok && next(w); ++t) {
        const int acc = t % T::ACC;
        if (MULTI && t >= T::ACC) {
          if (!__all_sync(0xffffffffu, b2::mbar_wait(bar_drained + acc * 8, ((t / T::ACC) & 1) ^ 1, abort_flag, PIPE_LIMIT_NS, B2_WAIT_TMEM_EMPTY))) break;
          b2::tc_fence_after();
        }
        const uint32_t d = tmem_base + acc * acc_cols;
        // Two stages a turn where the second has landed too: a turn's wait, vote and addresses take longer (about 350 clocks) than the
        // four instructions of a stage
        const int n = w.k1 - w.k0;
        for (int i = 0; i < n;) {
          if (!__all_sync(0xffffffffu, b2::mbar_wait(bar_full + stage * 8, phase, abort_flag, PIPE_LIMIT_NS, B2_WAIT_SMEM_FULL))) { ok = false; break; }
          if (t == 0 && i == 0 && lane == 0) stamp(a, 1);
          const int next_stage = stage + 1 == STAGES ? 0 : stage + 1;
          const uint32_t next_phase = phase ^ (next_stage == 0 ? 1u : 0u);
          const bool two = i + 1 < n && __all_sync(0xffffffffu, b2::mbar_test(bar_full + next_stage * 8, next_phase));
          b2::tc_fence_after();
          if (b2::elect_one()) {
            const uint32_t at = smem_base + stage * stage_bytes;
            const uint64_t dw = b2::umma_smem_desc(at), dx = b2::umma_smem_desc(at + W_BYTES);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) b2::umma_bf16_pair(d, dw + 2 * k, dx + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
            b2::umma_commit_pair(bar_empty + stage * 8, both);
            if (two) {
              const uint32_t at2 = smem_base + next_stage * stage_bytes;
              const uint64_t dw2 = b2::umma_smem_desc(at2), dx2 = b2::umma_smem_desc(at2 + W_BYTES);
#pragma unroll
              for (int k = 0; k < BK / 16; ++k) b2::umma_bf16_pair(d, dw2 + 2 * k, dx2 + 2 * k, idesc, 1u);
              b2::umma_commit_pair(bar_empty + next_stage * 8, both);
            }
          }
          __syncwarp();
          if (two) {
            i += 2;
            stage = next_stage;
            phase = next_phase;
          } else {
            ++i;
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && b2::elect_one()) b2::umma_commit_pair(bar_done + acc * 8, both);
        __syncwarp();
      }
      if (lane == 0) stamp(a, 2);
    }
  }

  const int q = warp & 3;                    // tensor-memory lane quadrant of an epilogue warp
  const int part = (warp - 2) >> 2;          // MULTI: the two sets of four warps take alternate chunks
  const int qw = (warp - 2) & 3;             // the warp's number in its set
  constexpr int PARTS = T::EW / 4;
  int f0, tok0;
  place(MULTI ? 0 : blockIdx.x / (2 * S), f0, tok0);
  // 8-token groups of the tile that hold tokens, and where each pair's share of them begins
  const int groups = MULTI ? a.bn >> 3 : (min(a.bn, a.M - tok0) + 7) >> 3;
  int begin[MAX_SPLIT + 1];
#pragma unroll
  for (int p = 0; p <= MAX_SPLIT; ++p) begin[p] = MULTI ? 0 : min(p, S) * groups / S;
  const int g0 = MULTI ? 0 : pair * groups / S, g1 = MULTI ? groups : (pair + 1) * groups / S;
  const int most = MULTI ? 0 : (groups + S - 1) / S;  // most groups any pair owns
  volatile int* s_last = reinterpret_cast<volatile int*>(tmem_slot + 2);  // [2]
  int* s_pos = reinterpret_cast<int*>(smem + a.bar_off + 256);  // positions of the tokens this CTA finishes
  bool ok = true;
  if (warp >= 2) b2::pdl_wait();

  if (!MULTI && S > 1) {
    if (warp >= 2) {
      ok = b2::mbar_wait(bar_done, 0, abort_flag, PIPE_LIMIT_NS, B2_WAIT_TMEM_FULL);
      b2::tc_fence_after();
    }
    // every pair of the cluster has finished its MMAs: the rings may take the others' parts, at [source][group][quadrant]
    // [upper or lower 16 lanes][lane] of 16 bytes, which the same lane of the owner reads
    __syncwarp();
    b2::cluster_arrive();
    b2::cluster_wait();
    if (warp >= 2 && ok) {
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      const uint32_t mine = smem_base + q * 1024 + lane * 16;
#pragma unroll
      for (int p = 0; p < MAX_SPLIT; ++p) {
        if (p >= S || p == pair) continue;
        const int n = begin[p + 1] - begin[p];
        const uint32_t dst = b2::map_to_cta(mine, p * 2 + side) + (pair < p ? pair : pair - 1) * most * 4096;
        const uint32_t src = taddr + begin[p] * 8;
        for (int g = 0; g < n; g += 2) {
          uint32_t r[2][2][4];
          tmem_ld_16x256_x1(src + g * 8, r[0][0]);
          tmem_ld_16x256_x1(src + (16u << 16) + g * 8, r[0][1]);
          if (g + 1 < n) {
            tmem_ld_16x256_x1(src + g * 8 + 8, r[1][0]);
            tmem_ld_16x256_x1(src + (16u << 16) + g * 8 + 8, r[1][1]);
          }
          b2::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (g + i < n) {
#pragma unroll
              for (int h = 0; h < 2; ++h)
                b2::st_cluster_v4(dst + (g + i) * 4096 + h * 512, __uint_as_float(r[i][h][0]), __uint_as_float(r[i][h][1]), __uint_as_float(r[i][h][2]),
                                  __uint_as_float(r[i][h][3]));
            }
        }
      }
    }
    __syncwarp();
    b2::cluster_arrive();
    b2::cluster_wait();
  }

  // (after an expired wait the warps keep meeting at their barriers, but store nothing)
  Walk w = first;
  for (int t = 0; warp >= 2 && next(w); ++t) {
    const int buf_no = t % T::ACC;
    const uint32_t taddr = tmem_base + buf_no * acc_cols + (static_cast<uint32_t>(q * 32) << 16);
    if (MULTI) place(w.tile, f0, tok0);
    const int head = f0 / FM;
    const bool heads = a.qkv_fused && f0 < a.N;
    if (heads) {  // while the main loop runs
      if (MULTI && t > 0) asm volatile("bar.sync 3, %0;" ::"n"(T::EW * 32) : "memory");  // the previous tile's rows are finished
      for (int i = threadIdx.x - 64; i < (g1 - g0) * 8; i += T::EW * 32) s_pos[i] = static_cast<int>(__ldg(a.positions + min(tok0 + g0 * 8 + i, a.M - 1)));
      asm volatile("bar.sync 3, %0;" ::"n"(T::EW * 32) : "memory");
    }
    ok = b2::mbar_wait(bar_done + buf_no * 8, (t / T::ACC) & 1, abort_flag, PIPE_LIMIT_NS, B2_WAIT_TMEM_FULL) && ok;
    b2::tc_fence_after();
    if (threadIdx.x == 64) stamp(a, 5);
    // The accumulator leaves in chunks of 4 groups (32 tokens).  The next chunk is read from tensor memory while this one
    // goes through the staging buffer, of which there are two, so that a chunk costs one synchronisation.
    uint32_t acc[2][16];
    const int first_g = g0 + 4 * part;
    constexpr int STEP = 4 * PARTS;
    bool mine = true;        // this CTA stores the tile
    float* sums = nullptr;   // where its fp32 sum lies, if not in tensor memory
    if (MULTI && w.k1 - w.k0 < a.kblocks) {
      // Part of the tile's K range: added into the slot of the first pair that holds some of it.
      const int u = (w.tile - first.rounds * pairs) * a.kblocks;
      const int p0 = ranges.holder(u), p1 = ranges.holder(u + a.kblocks - 1);
      float* slot = a.ws + static_cast<size_t>(p0 * 2 + side) * (FM * 256) + q * (32 * 256) + lane * 4;
      for (int g = first_g; g < g1; g += STEP) {
        tmem_ld_16x256_x4(taddr + g * 8, acc[0]);
        tmem_ld_16x256_x4(taddr + (16u << 16) + g * 8, acc[1]);
        b2::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          red_add_f4(slot + (g + i) * 256, acc[0] + 4 * i);
          red_add_f4(slot + (g + i) * 256 + 128, acc[1] + 4 * i);
        }
      }
      __threadfence();
      quad_meets(part);
      if (qw == 0 && lane == 0) {
        int* counter = a.counters + (w.tile * 2 + side) * 2 + part;
        const int last = atomicAdd(counter, 1) == p1 - p0;
        if (last) *counter = 0;
        s_last[part] = last;
      }
      quad_meets(part);
      mine = s_last[part] != 0;
      __threadfence();
      sums = slot;
    }
    auto fetch = [&](int g) {
      if (MULTI && sums != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          ld_cg_f4(acc[0] + 4 * i, sums + (g + i) * 256);
          ld_cg_f4(acc[1] + 4 * i, sums + (g + i) * 256 + 128);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(sums + g * 256 + i * 128) = make_float4(0.f, 0.f, 0.f, 0.f);
      } else if (MULTI || g1 - g >= 4) {  // (a whole tile's columns are allocated in powers of two from 32)
        tmem_ld_16x256_x4(taddr + g * 8, acc[0]);
        tmem_ld_16x256_x4(taddr + (16u << 16) + g * 8, acc[1]);
      } else {  // (never past the columns that are allocated)
#pragma unroll
        for (int i = 0; i < 3; ++i)
          if (g + i < g1) {
            tmem_ld_16x256_x1(taddr + (g + i) * 8, acc[0] + 4 * i);
            tmem_ld_16x256_x1(taddr + (16u << 16) + (g + i) * 8, acc[1] + 4 * i);
          }
      }
    };
    // bias of the four features whose rows this thread holds: lane / 4 + 0, 8, 16, 24 of the quadrant
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (a.bias != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int f = f0 + q * 32 + i * 8 + (lane >> 2);
        if (f < a.N) bias[i] = __uint_as_float(static_cast<uint32_t>(__ldg(a.bias + f)) << 16);
      }
    }
    // this chunk's sums as bf16 pairs of tokens: out[i] = features lane / 4 + 0, 8, 16, 24 of group g + i
    auto finish = [&](int g, uint32_t (&out)[4][4]) {
      b2::tc_wait_ld(acc);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[e] = __uint_as_float(acc[0][4 * i + e]) + bias[e >> 1];
          v[4 + e] = __uint_as_float(acc[1][4 * i + e]) + bias[2 + (e >> 1)];
        }
        if (!MULTI && S > 1 && g + i < g1) {
          const unsigned char* p = smem + (g + i - g0) * 4096 + q * 1024 + lane * 16;
#pragma unroll
          for (int src = 0; src < MAX_SPLIT - 1; ++src) {
            if (src < S - 1) {
              const float4 x = *reinterpret_cast<const float4*>(p + src * most * 4096), y = *reinterpret_cast<const float4*>(p + src * most * 4096 + 512);
              v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
              v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) out[i][e] = b2::pack_bf16(v[2 * e], v[2 * e + 1]);
      }
    };
    if (mine && first_g < g1) fetch(first_g);
    int half = 0;
    if (!mine) {
      // another CTA stores it
    } else if (!heads) {
      // Every warp on its own: 32 tokens x 64 bytes (its 32 features).  Pieces of 16 bytes are XORed with the token so that
      // neither the transposing stores nor the row reads meet in a bank.
      unsigned char* buf = smem + a.out_off + (warp - 2) * 4096;
      const int st_off = (lane & 7) * 64 + (((lane >> 3) ^ ((lane >> 1) & 3)) << 4);
      const int ld_off = (lane >> 2) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4);
      const int f = f0 + q * 32 + (lane & 3) * 8;
      uint16_t* dst = a.C + (a.silu_pairs ? f >> 1 : f);
      for (int g = first_g; g < g1; g += STEP) {
        uint32_t out[4][4];
        finish(g, out);
        if (g + STEP < g1) fetch(g + STEP);
        unsigned char* stg = buf + half * 2048;
        half ^= 1;
        const uint32_t to = b2::smem_u32(stg) + st_off;
#pragma unroll
        for (int i = 0; i < 4; ++i) stmatrix_x4_trans(to + i * 512, out[i]);
        __syncwarp();
        const int token0 = g * 8 + (lane >> 2), live = ok ? min(g1 * 8, a.M - tok0) : 0;
        uint4 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const uint4*>(stg + ld_off + i * 512);
        if (f < a.N) {
          uint16_t* row = dst + static_cast<int64_t>(tok0 + token0) * a.ldc;
          if (a.silu_pairs) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint2 act = b2::silu_mul_pairs(w[i]);
              if (token0 + i * 8 < live) *reinterpret_cast<uint2*>(row + i * 8 * a.ldc) = act;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (token0 + i * 8 < live) *reinterpret_cast<uint4*>(row + i * 8 * a.ldc) = w[i];
          }
        }
      }
    } else {
      // qkv projection: this CTA's 128 features are one head.  q: norm and rotation; k: the same, and into the cache; v: into
      // the cache.  Four warps share a staging buffer of whole head rows; a warp finishes four tokens' rows at a time, 8 lanes a
      // row with 8 dimensions of either half each, so that every access is a 16-byte vector and a norm takes three exchanges (a
      // row per warp in 4-byte accesses was bound by its memory instructions and exchanges: 97 -> 77 us at 8000 tokens x 4096 x 1024, plain stores 54).
      // Arithmetic, order of the sums and roundings are those of qk_norm_rope_store_kernel: a lane's four partial sums are what
      // four of its lanes hold.
      const bool rotated = head < a.nq + a.nkv;
      const int row4 = lane >> 3, pc = lane & 7;
      uint4 nw1 = make_uint4(0, 0, 0, 0), nw2 = nw1;
      const uint16_t* norm = rotated ? (head < a.nq ? a.q_norm_w : a.k_norm_w) : nullptr;
      uint16_t* cache = nullptr;
      if (head >= a.nq && a.k_cache != nullptr) cache = rotated ? a.k_cache + (head - a.nq) * FM : a.v_cache + (head - a.nq - a.nkv) * FM;
      if (norm != nullptr) {
        nw1 = *reinterpret_cast<const uint4*>(norm + pc * 8);
        nw2 = *reinterpret_cast<const uint4*>(norm + 64 + pc * 8);
      }
      const int own = (g1 - g0) * 8;
      float4 factors[4];  // rotary factors (cosines, sines) and cache slot of the next row travel while this one is finished
      int slot = -1;
      auto ahead = [&](int row) {
        row = min(row, own - 1);
        if (cache != nullptr) slot = __ldg(a.slots + min(tok0 + g0 * 8 + row, a.M - 1));
        if (rotated) {
          const float4* f = reinterpret_cast<const float4*>(a.cos_sin + static_cast<int64_t>(s_pos[row]) * FM + pc * 8);
          factors[0] = __ldg(f);
          factors[1] = __ldg(f + 1);
          factors[2] = __ldg(f + 16);
          factors[3] = __ldg(f + 17);
        }
      };
      if (first_g < g1) ahead((first_g - g0) * 8 + qw * 4 + row4);
      for (int g = first_g; g < g1; g += STEP) {
        uint32_t out[4][4];
        finish(g, out);
        if (g + STEP < g1) fetch(g + STEP);
        unsigned char* stg = smem + a.out_off + part * 16384 + half * 8192;
        half ^= 1;
#pragma unroll
        for (int i = 0; i < 4; ++i) stmatrix_x4_trans(b2::smem_u32(stg) + staged(i * 8 + (lane & 7), q * 4 + (lane >> 3)), out[i]);
        quad_meets(part);
        const int live = ok ? min(own, a.M - tok0 - g0 * 8) - (g - g0) * 8 : 0;
#pragma unroll
        for (int i0 = 0; i0 < 32; i0 += 16) {
          const int lt = i0 + qw * 4 + row4;
          uint4 lo = *reinterpret_cast<const uint4*>(stg + staged(lt, pc)), hi = *reinterpret_cast<const uint4*>(stg + staged(lt, 8 + pc));
          if (rotated) {
            float x1[8], x2[8];
            b2::unpack8(lo, x1);
            b2::unpack8(hi, x2);
            if (norm != nullptr) {
              float ss[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) ss[k] = (x1[2 * k] * x1[2 * k] + x2[2 * k] * x2[2 * k]) + (x1[2 * k + 1] * x1[2 * k + 1] + x2[2 * k + 1] * x2[2 * k + 1]);
#pragma unroll
              for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], o);
              const float rstd = rsqrtf(((ss[0] + ss[2]) + (ss[1] + ss[3])) / 128.0f + a.qk_eps);
              // (a product of two bf16 values has one rounding to bf16 either way)
              lo = b2::normed(x1, rstd, nw1);
              hi = b2::normed(x2, rstd, nw2);
              b2::unpack8(lo, x1);
              b2::unpack8(hi, x2);
            }
            const float* c = reinterpret_cast<const float*>(factors);
            float y1[8], y2[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {  // separate roundings of the products, as the eager reference computes them
              y1[e] = __fsub_rn(__fmul_rn(x1[e], c[e]), __fmul_rn(x2[e], c[8 + e]));
              y2[e] = __fadd_rn(__fmul_rn(x2[e], c[e]), __fmul_rn(x1[e], c[8 + e]));
            }
            lo = b2::pack8(y1);
            hi = b2::pack8(y2);
          }
          const int to_slot = cache != nullptr ? slot : -1;
          ahead((g - g0 + (i0 == 0 ? 0 : STEP)) * 8 + (i0 ^ 16) + qw * 4 + row4);
          if (lt < live) {
            uint16_t* dst = a.C + static_cast<int64_t>(tok0 + g * 8 + lt) * a.ldc + f0 + pc * 8;
            *reinterpret_cast<uint4*>(dst) = lo;
            *reinterpret_cast<uint4*>(dst + 64) = hi;
            if (to_slot >= 0) {
              uint16_t* to = cache + static_cast<int64_t>(to_slot) * a.nkv * FM + pc * 8;
              *reinterpret_cast<uint4*>(to) = lo;
              *reinterpret_cast<uint4*>(to + 64) = hi;
            }
          }
        }
      }
    }
    if (MULTI) {
      b2::tc_fence_before();
      __syncwarp();
      if (lane == 0) b2::mbar_arrive_cluster(b2::map_to_cta(bar_drained, 0) + buf_no * 8);
    }
    if (threadIdx.x == 64) stamp(a, 4);
  }

  // ---- all roles of the cluster meet; tensor memory goes back ------------------
  b2::pdl_wait();
  __syncwarp();
  b2::tc_fence_before();
  __syncthreads();
  const int aborted = *abort_flag;
  if (aborted) {
    // let bulk copies that may still be in flight land before anyone leaves
    for (int i = 0; i < 100; ++i) __nanosleep(2000);
    if (threadIdx.x == 0) b2::report_timeout(a.status, aborted);
  }
  // neither CTA may free the pair's tensor memory or leave while the other still signals its barriers
  b2::cluster_arrive();
  b2::cluster_wait();
  b2::tc_fence_after();
  if (warp == 1) b2::tmem_dealloc_pair(tmem_base, tmem_cols);
  if (threadIdx.x == 0) stamp(a, 6);
}

using TilePlan = b2_tile_plan;

// Geometry of one problem (host arithmetic only; resident(split, bytes) = clusters of 2 * split CTAs with that much shared
// memory the device holds at once).  The candidates' times are estimated, in nanoseconds, from what the parts were measured
// to take on this part, and the fastest is taken:
//   weights from DRAM at 6.4 TB/s; operands into an SM at 82 B/ns (from L2 or DRAM), and a turn of the ring takes the loaded
//   DRAM latency of 1.6 us; 2 clocks of the tensor pipe per token column and K block of a pair; the exchange of a split tile
//   at 20 B/ns per SM (SM-to-SM network; stores and bulk copies alike) plus two cluster barriers; 0.6 us per 32 tokens stored
//   by four warps (an SM sends about 14 bytes per clock).
// (The 82 B/ns date from when the TMA and MMA warps issued from one lane; 100 to 150 have been seen since.  Widths swept again from 512
// tokens on: the choices are within 4 % of the best, 777 x 24576 x 4096 takes 128.7 us at 224 and 123.7 at 160.  Below, another choice would
// also cut K elsewhere and change results.)
template <class Resident>
int plan_tile_gemm(int M, int N, int K, int num_sms, int tile_cap, Resident&& resident, TilePlan* p) {
  if (M <= 0 || N <= 0 || K <= 0 || num_sms < 2) return B2_ERR_ARG;
  const int pairs = num_sms / 2;
  const int kblocks = (K + BK - 1) / BK, tiles_f = (N + 2 * FM - 1) / (2 * FM);
  double best = 1e30;
  const int t_min = (M + 255) / 256;
  // From 512 tokens on every output is one unbroken fp32 sum over K, the same bits whatever the tile and the grid; below, the
  // K range may be cut.  The line is drawn for the results, which prompts of 512 tokens and more have had since before K was ever
  // cut here, and not for time: allowed from 512 on, cutting would win where whole tiles leave pairs idle (with the norm, 512
  // tokens x 4096 x 12288 77.9 -> 58.0 us, 600 x 1024 x 3072 22.2 -> 16.3) and lose where the estimate is off (600 x 5120 x
  // 25600 176 -> 223, 777 x 5120 x 8192 75 -> 82).
  const bool cut = M < 512;
  for (int t = t_min; t <= std::max(2 * t_min, std::min(16, (M + 63) / 64)); ++t) {
    const int bn = ((M + t - 1) / t + 31) / 32 * 32;
    const int tiles_t = (M + bn - 1) / bn;
    const int64_t tiles = static_cast<int64_t>(tiles_f) * tiles_t;
    const int stage = W_BYTES + bn * BK, groups = bn / 8;
    for (int v = 0; v <= (cut ? MAX_SPLIT : 1); ++v) {  // 0: whole tiles, two CTAs per SM, one tile each
      const int s = std::max(v, 1);
      const int64_t work = tiles * s;  // pairs launched
      if (v == 0 && (work <= pairs || work > 2 * pairs)) continue;
      if (s > 1 && (kblocks < 2 * s || work > 2 * pairs)) break;
      const int most = (groups + s - 1) / s, kb = (kblocks + s - 1) / s;
      const uint32_t red = s > 1 ? static_cast<uint32_t>(s - 1) * most * 4096 : 0;
      const bool multi = v == 1 && (work > pairs || kb * stage > static_cast<int>(SMEM_HALF - SMEM_EXTRA));
      // all of an SM's shared memory where no second CTA comes and the ring would use it
      const bool deep = multi || (work <= pairs && kb * stage > static_cast<int>(SMEM_HALF - SMEM_EXTRA));
      const uint32_t limit = deep ? SMEM_ALL : SMEM_HALF;
      const uint32_t out = multi ? Shape<true>::OUT_BYTES : Shape<false>::OUT_BYTES;
      const int stages = std::min<int>({MAX_STAGES, static_cast<int>((limit - SMEM_EXTRA - (multi ? out : 0)) / stage), std::max(2, kb)});
      // the staging buffers lie behind the ring where it stays in use (MULTI), else where the ring was
      const uint32_t out_off = multi ? stages * stage : red;
      const uint32_t ring = std::max<uint32_t>(stages * stage, out_off + out);
      if (ring + SMEM_EXTRA > limit) continue;
      if (s > 1 && resident(s, ring + SMEM_EXTRA) < tiles) continue;  // (two waves of a split tile never pay)
      const double t_mem = 2.0 * N * K / 6400.0;
      const double t_kb = std::max({stage / 82.0, (v == 0 ? 800.0 : 1600.0) / stages, (std::max(bn, 64) * 2 + 40) / 1.9});
      const double t_out = (multi ? 300.0 : 600.0) * ((groups + 4 * s - 1) / (4 * s)) + (s > 1 ? 1500.0 + (s - 1) * most * 4096 / 20.0 : 0.0);
      int64_t rounds = multi ? work / pairs : 0, ranged = multi ? work % pairs : 0;
      double cost;
      if (multi) {
        // the rest as one more round, or in ranges of K blocks: two parts per pair into L2 at 26 B/ns, one tile back
        const double whole = std::max(kb * t_kb, t_out) * (rounds + (ranged > 0 ? 1 : 0));
        const double in_ranges = std::max(kb * t_kb, t_out) * rounds + ranged * kb * t_kb / pairs + 3000.0 + 2.5 * bn * FM * 4 / 26.0;
        if (!cut || whole <= in_ranges || ranged * kb < 4 * pairs || tiles * 4 > tile_cap) {
          if (ranged > 0) ++rounds;
          ranged = 0;
        }
        cost = std::max(t_mem, ranged > 0 ? in_ranges : whole) + t_out;
      } else {
        // (two CTAs of an SM overlap each other's latencies: measured 95 B/ns where one alone gets 80; 777 tokens x 6144 x 4096
        // as 168 whole tiles on 148 SMs 57 -> 41 us)
        cost = std::max(t_mem, static_cast<double>((2 * work + num_sms - 1) / num_sms) * kb * (v == 0 ? 0.85 : 1.0) * t_kb) + t_out + (v == 0 ? t_out : 0.0);
      }
      if (cost < best) {
        best = cost;
        const int64_t grid = multi ? (ranged > 0 ? pairs : std::min<int64_t>(tiles, pairs)) * 2 : work * 2;
        *p = TilePlan{bn, tiles_f, tiles_t, kblocks, s, std::min(tiles_t, 16), stages, multi ? 1 : 0, static_cast<int>(rounds), static_cast<int>(ranged),
                      static_cast<int>(grid), static_cast<int>(out_off), static_cast<int>(ring), static_cast<int>(ring + SMEM_EXTRA), bn};
      }
    }
  }
  if (best >= 1e30) return B2_ERR_SHAPE;
  // Whole tiles are as narrow as the tokens let them be in steps of 16 columns, the least step of a pair's tcgen05.mma: 777 tokens are 4 x 208
  // and not 4 x 224.  An output's sum over K is the same; where K is cut, widths decide where, and stay.  (The choice is made by bn: by
  // the true widths it would fall on other tiles, and below 512 tokens on other cuts.)
  if (p->split == 1 && p->ranged == 0) p->width = ((M + p->tiles_t - 1) / p->tiles_t + 15) / 16 * 16;
  return B2_OK;
}

// clusters of 2 * split CTAs resident at once, asked once per device for the two sizes of shared memory
int resident_tile_clusters(int dev, int split, uint32_t smem) {
  static std::atomic<int> known[64][MAX_SPLIT + 1][2];  // answer + 1
  const int deep = smem > SMEM_HALF ? 1 : 0;
  std::atomic<int>& slot = known[dev][split][deep];
  int n = slot.load(std::memory_order_relaxed) - 1;
  if (n >= 0) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * split * 64);
  cfg.blockDim = dim3(Shape<false>::THREADS);
  cfg.dynamicSmemBytes = deep ? SMEM_ALL : SMEM_HALF;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_tile_kernel<false>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  slot.store(n + 1, std::memory_order_relaxed);
  return n;
}

}  // namespace

namespace b2 {

int launch_tile_gemm(b2_ctx* ctx, const void* A, int64_t lda, const void* W, int64_t ldw, int M, int N, int K, const StoreEpilogue& e, cudaStream_t stream) {
  static std::atomic<bool> done[64];  // the opt-in to more than 48 KB of dynamic shared memory belongs to a device
  const int dev = ctx->cfg.device;
  if (dev < 0 || dev >= 64) return set_error(B2_ERR_UNSUPPORTED, "device ordinal %d not supported", dev);
  if (!done[dev].load(std::memory_order_acquire)) {
    B2_CUDA(cudaFuncSetAttribute(gemm_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALL));
    B2_CUDA(cudaFuncSetAttribute(gemm_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALL));
    done[dev].store(true, std::memory_order_release);
  }
  TilePlan p;
  int rc = plan_tile_gemm(M, N, K, ctx->num_sms, ctx->tile_counter_cap * 4, [dev](int split, uint32_t smem) { return resident_tile_clusters(dev, split, smem); }, &p);
  if (rc != B2_OK) return rc;
  TileArgs a{};
  a.C = e.C;
  a.ldc = e.ldc;
  a.bias = e.bias;
  a.status = ctx->status_dev;
  a.M = M;
  a.N = N;
  a.kblocks = p.kblocks;
  a.bn = p.width;
  a.stages = p.stages;
  a.split = p.split;
  a.rounds = p.rounds;
  a.ranged = p.ranged;
  a.ws = ctx->splitk_ws;
  a.counters = ctx->tile_counters;
  a.tilesF = p.tiles_f;
  a.tilesT = p.tiles_t;
  a.group = p.group;
  a.out_off = p.out_off;
  a.bar_off = p.bar_off;
  a.trace = ctx->trace_on ? ctx->trace : nullptr;
  a.trace_ctas = ctx->num_sms;
  a.silu_pairs = e.silu_pairs;
  a.qkv_fused = e.qkv_fused;
  a.nq = e.nq;
  a.nkv = e.nkv;
  a.positions = e.positions;
  a.cos_sin = e.cos_sin;
  a.q_norm_w = e.q_norm_w;
  a.k_norm_w = e.k_norm_w;
  a.qk_eps = e.qk_eps;
  a.k_cache = e.k_cache;
  a.v_cache = e.v_cache;
  a.slots = e.slots;
  CUtensorMap tmW, tmX;
  rc = encode_tmap_2d(&tmW, W, K, N, ldw, BK, FM);
  if (rc != B2_OK) return rc;
  rc = encode_tmap_2d(&tmX, A, K, M, lda, BK, a.bn / 2);
  if (rc != B2_OK) return rc;
  if (p.multi)
    B2_CUDA(b2_launch_cluster(gemm_tile_kernel<true>, dim3(p.grid), dim3(Shape<true>::THREADS), p.smem, stream, 2u, tmW, tmX, a));
  else
    B2_CUDA(b2_launch_cluster(gemm_tile_kernel<false>, dim3(p.grid), dim3(Shape<false>::THREADS), p.smem, stream, 2u * p.split, tmW, tmX, a));
  return B2_OK;
}

}  // namespace b2

// ---------------------------------------------------------------------------
// The planner as data, for tests that run without a GPU (no CUDA call here).
// ---------------------------------------------------------------------------
extern "C" int b2_plan_tile_gemm(int M, int N, int K, int num_sms, const int* resident_clusters, b2_tile_plan* plan) {
  if (plan == nullptr) return B2_ERR_ARG;
  return plan_tile_gemm(M, N, K, num_sms, 1 << 18, [&](int split, uint32_t smem) { return resident_clusters != nullptr ? resident_clusters[(smem > SMEM_HALF ? MAX_SPLIT + 1 : 0) + split] : 0; }, plan);
}

extern "C" int b2_plan_tile_segments(const b2_tile_plan* plan, int pair, int* segments, int cap) {
  if (plan == nullptr || plan->grid <= 0 || pair < 0 || pair >= plan->grid / 2 || cap < 0 || (cap > 0 && segments == nullptr)) return -B2_ERR_ARG;
  const int pairs = plan->grid / 2, tiles = plan->tiles_f * plan->tiles_t;
  const Ranges r(plan->multi ? plan->ranged * plan->kblocks : plan->kblocks, plan->multi ? pairs : plan->split);
  Walk w = plan->multi ? first_walk<true>(r, pairs, pair, 0, plan->kblocks, plan->rounds, plan->ranged, tiles)
                       : first_walk<false>(r, pairs, pair, pair % plan->split, plan->kblocks, 0, 0, tiles);
  int n = 0;
  for (; w.next(); ++n)
    if (n < cap) {
      segments[3 * n] = plan->multi ? w.tile : pair / plan->split;
      segments[3 * n + 1] = w.k0;
      segments[3 * n + 2] = w.k1;
    }
  return n;
}

extern "C" int b2_plan_tile_holders(const b2_tile_plan* plan, int tile, int* first_pair, int* last_pair) {
  if (plan == nullptr || first_pair == nullptr || last_pair == nullptr || !plan->multi || plan->ranged <= 0 || plan->grid <= 0) return B2_ERR_ARG;
  const int pairs = plan->grid / 2, u = (tile - plan->rounds * pairs) * plan->kblocks;
  if (u < 0 || tile >= plan->tiles_f * plan->tiles_t) return B2_ERR_ARG;
  const Ranges r(plan->ranged * plan->kblocks, pairs);
  *first_pair = r.holder(u);
  *last_pair = r.holder(u + plan->kblocks - 1);
  return B2_OK;
}
