// All decoder layers of one decode step in one launch, for models of 1024 hidden features whose layer fits the SMs' shared memory.
//
// A layer of a small model is 30 MB of weights: 5 us of HBM time on the whole chip.  As five launches it takes 29 us (Qwen3-0.6B, one
// sequence of 300 tokens), here 17: every launch waits for the one before it, sets up, has its first bytes travel and combines its split sums, and none of
// that overlaps.  Here one CTA per SM stays for the whole step:
//   - every projection's output rows are dealt to the CTAs, whole rows: a CTA owns the same few rows with all of K in every layer, so
//     no sum crosses an SM, and its share of a layer (28 + 7 + 44 + 7 rows of Qwen3-0.6B) is brought in by bulk copies one phase and
//     more before it is used: the weights stream through the waits between the phases;
//   - what a phase hands to the next one is its own flag: a word that is all ones has not been written yet, and a reader takes its
//     fragments again until none is.  All to all, 4 KB among 148 CTAs, that is 1420 clocks a turn, with a barrier in between (fence,
//     count, polls, then the reads) 3200.  Polls that begin at once stand in the stores' way: 3600 to 4400.  (Of a probe that does nothing else;
//     here the fragments of the weights come first where a phase can begin with them.)
//   - 8 warps split K: a warp multiplies its slice of the weights' rows (the 16 rows of an mma.sync) with its slice of 8 tokens (a lane
//     takes 8 neighbouring elements of a row; which k of the instruction they stand for does not matter as long as both operands agree),
//     and the 8 partial sums meet in shared memory.  tcgen05 would want 128 rows of weights in a tile: with 7 to 44 rows
//     per SM its tiles would be mostly padding, and what bounds a phase is the exchange, not the multiplications;
//   - norms are computed by every CTA on what it reads (fp32 sums of the residual stream), so they cost no phase of their own.
// Attention deals groups of 16 tokens evenly to the warps of all CTAs.  A warp reads K straight into fragments and V through a private
// buffer, keeps its own running maximum, and the parts of a (sequence, head) meet in shared memory, or in L2 where they span CTAs.
//
// Buffers between phases exist three times; layer l uses number l % 3.  Whoever writes a word of one also sets its counterpart of the
// layer before back to all ones; that buffer is used again two layers on.  Nobody still needs the counterpart: a CTA stores in a phase
// once it has read what every CTA stored after it had finished the layer before, and a store waits for the loads that it depends on.
// Nobody sees it as it was before it was set back: ahead of the down projection the threads of a CTA meet, and each passes a fence.
// What they store from then on is a release of all that the CTA has set back so far; the threads of other CTAs that read it pass
// their fence of the next layer, which makes an acquire of it, for their whole CTA past the barriers that follow; and the layer after that is the
// first to look at those buffers again.  (Fences of each store and load would say the same and cost a round trip to L2 in every phase; this
// one is once a layer, in the shadow of the down projection's wait.)  Within a layer nothing is ordered but a word's own 32 bits: it
// says itself whether it is there.  No result is all ones: additions, conversions and products make canonical NaNs only.
//
// Every CTA waits for all others, so the launch is cooperative: all of them are resident.  Every wait has a limit.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "b2_common.cuh"

namespace {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int H = 1024;               // hidden features: the fragments' arrays and the norms' shares are laid out for this one size
constexpr int KN = H / (WARPS * 32);  // k steps (of 32) of a warp in the projections of the norms' outputs
constexpr int MT = 3;                 // and 16-row groups of a CTA's weights, at most
constexpr int KB = 1024 / (WARPS * 32), MAX_KB = 3;  // o, down: k steps for every 1024 input features, and of those at most
constexpr int HD = 128;               // head dimension
constexpr int MAX_GROUP = 2;          // query heads per KV head
constexpr int MAX_ROWS = 16;          // see layout_of
constexpr int MAX_LAYERS = 64;
constexpr int TILE = 8;               // tokens multiplied at a time
constexpr int GROUP_TOKENS = 16;      // attention: tokens a warp takes at a time
constexpr int AHEAD = 3;              // groups that keys and values are sent to L2 ahead of their use (9: 16 rows of 4000 tokens 2668 us a step, 3: 2014)
constexpr int V_BYTES = GROUP_TOKENS * HD * 2;
constexpr int PART = MAX_GROUP * HD + 2 * MAX_GROUP;  // floats of a partial attention result: O, then the maxima and sums
constexpr int COMBINE_GROUPS = 8;     // what combining the parts of a (sequence, head) over CTAs costs, in groups of a CTA
constexpr uint32_t UNWRITTEN = 0xffffffffu;
constexpr uint64_t WAIT_LIMIT_NS = 1000000000ull;

struct Args {
  b2_stack_layer layer[MAX_LAYERS];
  const uint16_t* final_norm;
  const uint16_t* x;       // [rows][H] residual stream at the start
  uint16_t* out;           // [rows][H] after the final norm
  const int64_t* positions;
  const int32_t* lens;
  const int32_t* slots;
  const int32_t* tables;
  int64_t bt_stride;
  const float* cos_sin;
  // exchanged between the phases, [3][rows] each: layer l uses number l % 3
  float *sum_o, *sum_d;    // [H] residual stream after attention, after the MLP; fp32
  uint16_t* qkv;           // [(nq + 2 nkv) HD] projections
  uint16_t* attn;          // [nq HD]
  uint16_t* act;           // [MLP features]
  float* parts;            // [3][CTAs][PART] partial attention results
  unsigned int* gave_up;   // all ones, or the wait that some CTA has given up
  unsigned int* arrivals;  // all ones before the first (staged batches only)
  B2Status* status;
  int layers, rows, nq, nkv, group, inter, bt_width, block_shift, num_blocks;
  float eps, qk_eps, scale_log2;
  uint32_t off_a, off_vec, off_b, off_s, off_x, off_small, off_own;  // shared memory
};

// ---- instructions ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds_v2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts_v2(uint32_t addr, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory"); }
// 16 bytes to shared memory, zeros where there is nothing to read
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool any) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(any ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the last group have landed
__device__ __forceinline__ void cp_async_wait_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(b2::kEvictFirst) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// exchanged words: from and to L2, where all SMs see them
__device__ __forceinline__ uint4 ld_x4(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_x1(const void* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_x1(void* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void st_x2(void* p, uint32_t x, uint32_t y) { asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(x), "r"(y) : "memory"); }
__device__ __forceinline__ void st_x4(void* p, const float4& v) {
  asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ bool unwritten(const uint4& v) { return max(max(v.x, v.y), max(v.z, v.w)) == UNWRITTEN; }
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// rows of a matrix with `n` rows (or groups of rows) that CTA `i` of `g` owns: [share(n, i, g), share(n, i + 1, g))
__host__ __device__ __forceinline__ int share(int n, int i, int g) { return n * i / g; }
// bytes between the rows of normalised activations: 64 past a multiple of 128, so that the 16-byte reads of 8 lanes (two rows, 64
// bytes of each) cover all banks
__host__ __device__ constexpr uint32_t row_bytes(int k) { return static_cast<uint32_t>(k) * 2 + 64; }

// How the groups of 16 tokens of all (sequence, head) items, in that order, are dealt: contiguous ranges to the CTAs (whole items
// where there are few enough and the longest costs less than combining), and of these to the warps.
struct Deal {
  const int* first;  // [rows + 1] groups per KV head before each sequence
  int rows, nkv, total, ctas, base, rem, by_item;
  __host__ __device__ __forceinline__ int cta_begin(int i) const {
    if (!by_item) return i * base + (i < rem ? i : rem);
    const int b = i / nkv;
    return b >= rows ? total : first[b] * nkv + (i - b * nkv) * (first[b + 1] - first[b]);
  }
  __host__ __device__ __forceinline__ int cta_of(int u) const {
    const int big = rem * (base + 1);
    return u < big ? u / (base + 1) : rem + (u - big) / base;
  }
};
__host__ __device__ __forceinline__ Deal deal_groups(const int* first, int rows, int nkv, int most, int grid) {
  Deal d;
  d.first = first;
  d.rows = rows;
  d.nkv = nkv;
  d.total = first[rows] * nkv;
  const int per = (d.total + grid - 1) / grid, items = rows * nkv;
  const int spread = per <= 8 ? (d.total + 7) / 8 : grid;  // (no fewer than 8 groups in a part)
  d.by_item = items <= grid && most <= d.total / (spread > 0 ? spread : 1) + COMBINE_GROUPS;
  d.ctas = d.by_item ? items : (spread < grid ? spread : grid);
  d.base = d.ctas > 0 ? d.total / d.ctas : 0;
  d.rem = d.ctas > 0 ? d.total % d.ctas : 0;
  return d;
}

// What a CTA keeps in shared memory in front of its buffers.  The phases are inlined into one loop, whose fragments need all registers
// there are (255 a thread, 24 bytes of spills); they find everything else here, and nothing but the loop's counter lives on from one to the next.
struct Shared {
  Args args;
  uint64_t bar_a, bar_b;  // weight buffers filled
  int abort;
  int q0, q1, h0, h1, p0, p1;  // this CTA's rows of qkv, of o and down, of gate/up
  // contexts
  int rows, most, staged;
  int first[MAX_ROWS + 1];  // groups per KV head before each sequence
  int len[MAX_ROWS], block[MAX_ROWS];
  Deal deal;
  int u0, u1, start[WARPS];  // this CTA's groups; the sequence of each warp's first
  alignas(16) float squares[TILE * WARPS];
  alignas(16) uint16_t qk_norms[2 * HD];
};
extern __shared__ __align__(1024) unsigned char smem[];
__device__ __forceinline__ Shared& shared() { return *reinterpret_cast<Shared*>(smem); }

// first row of layer l's copy of an exchange buffer
__device__ __forceinline__ size_t exchange_row(int l) { return static_cast<size_t>(l % 3) * shared().args.rows; }

// A thread's place, derived anew by every phase (see Shared).
struct Place {
  int tid, warp, lane, g, c;  // g, c: row and column pair of a fragment
  __device__ __forceinline__ Place() {
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    warp = tid >> 5;
    lane = tid & 31;
    g = lane >> 2;
    c = lane & 3;
  }
  // A warp's poll found words that are not written yet (`bad` in some lane): look again?  False when all are there, or when
  // some CTA has given up.
  __device__ __forceinline__ bool again(bool bad, uint32_t& tries, uint64_t& t0) const {
    if (!__any_sync(0xffffffffu, bad)) return false;
    volatile int* abort_flag = &shared().abort;
    if (*abort_flag) return false;
    if ((++tries & 0xFF) != 0) return true;
    if (t0 == 0) t0 = b2::globaltimer_ns();
    int stop = 0;
    if (lane == 0) {
      const uint32_t other = ld_x1(shared().args.gave_up);
      stop = other == UNWRITTEN ? 0 : static_cast<int>(other);
      if (stop == 0 && b2::time_limit_passed(t0, WAIT_LIMIT_NS)) stop = B2_WAIT_STACK;
      if (stop) {
        st_x1(shared().args.gave_up, stop);
        *abort_flag = stop;
      }
    }
    return __shfl_sync(0xffffffffu, stop, 0) == 0;
  }
};
// All CTAs meet, `times` for the times-th time; what they wrote before is visible to all after.
__device__ __forceinline__ void meet(unsigned int times) {
  const Place t;
  const Args& a = shared().args;
  __syncthreads();
  if (t.warp == 0) {
    if (t.lane == 0) {
      __threadfence();
      atomicAdd(a.arrivals, 1u);
    }
    const unsigned int last = times * gridDim.x - 1;  // (they count from all ones)
    uint32_t tries = 0;
    uint64_t since = 0;
    auto short_of = [&] {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.arrivals) : "memory");
      return static_cast<int>(v - last) < 0;
    };
    while (t.again(short_of(), tries, since)) {}
  }
  __syncthreads();
}
// The next use of a buffer, uses counted over the layers: qkv and gate/up with their norms' weights in buffer A, o and down in B.  A CTA's
// rows lie side by side, so one copy brings them all; one thread calls it.  (Rows apart, for the banks' sake, took a copy each, 45 of
// them 0.7 us to issue, in which other warps' shared-memory accesses waited; see load_fragments for the banks.)
__device__ __forceinline__ void load_a(int use) {
  Shared& sh = shared();
  const Args& a = sh.args;
  if (use >= 2 * a.layers) return;
  const b2_stack_layer& L = a.layer[use >> 1];
  const bool mlp = use & 1;
  const int r0 = mlp ? sh.p0 : sh.q0, r1 = mlp ? sh.p1 : sh.q1;
  const uint32_t bytes = static_cast<uint32_t>(r1 - r0) * (H * 2), bar = b2::smem_u32(&sh.bar_a), base = b2::smem_u32(smem);
  b2::mbar_arrive_expect_tx(bar, bytes + H * 2);
  bulk_load(base + a.off_a, static_cast<const uint16_t*>(mlp ? L.gate_up_w : L.qkv_w) + static_cast<size_t>(r0) * H, bytes, bar);
  bulk_load(base + a.off_vec, mlp ? L.post_norm : L.in_norm, H * 2, bar);
}
__device__ __forceinline__ void load_b(int use) {
  Shared& sh = shared();
  const Args& a = sh.args;
  if (use >= 2 * a.layers) return;
  const b2_stack_layer& L = a.layer[use >> 1];
  const bool mlp = use & 1;
  const int k = mlp ? a.inter : a.nq * HD;
  const uint32_t bytes = static_cast<uint32_t>(sh.h1 - sh.h0) * k * 2, bar = b2::smem_u32(&sh.bar_b);
  b2::mbar_arrive_expect_tx(bar, bytes);
  bulk_load(b2::smem_u32(smem) + a.off_b, static_cast<const uint16_t*>(mlp ? L.down_w : L.o_w) + static_cast<size_t>(sh.h0) * k, bytes, bar);
}
// A lane's fragments of row `g` of some weight rows for N k steps from `at` (16 bytes of every 64).  Rows are a multiple of 128 bytes apart,
// so the odd ones take the steps of a pair in the other order: the 8 lanes of an access then cover all banks.
template <int N>
__device__ __forceinline__ void load_fragments(uint4 (&w)[N], uint32_t at, int g) {
  const bool odd = g & 1;
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const uint4 x = lds_v4(at + (odd ? i + 1 : i) * 64), y = lds_v4(at + (odd ? i : i + 1) * 64);
    w[i] = odd ? y : x;
    w[i + 1] = odd ? x : y;
  }
}
__device__ __forceinline__ void wait_weights(uint64_t* bar, uint32_t parity) { b2::mbar_wait(b2::smem_u32(bar), parity, &shared().abort, WAIT_LIMIT_NS, B2_WAIT_SMEM_FULL); }

// Projection of the normalised residual stream in buffer A: use 2 l is layer l's qkv, use 2 l + 1 its gate/up with SiLU(gate) * up.
// (One instance for both, and one of add_project: the phases' code is walked through once a layer, and what does not fit the
// instruction cache is waited for.)
__device__ __forceinline__ void norm_project(int use) {
  const Place t;
  Shared& sh = shared();
  const Args& a = sh.args;
  const uint32_t base = b2::smem_u32(smem);
  const bool silu = use & 1, from_x = use == 0;
  const int rows = sh.rows, r0 = silu ? sh.p0 : sh.q0, R = (silu ? sh.p1 : sh.q1) - r0, features = silu ? a.inter : (a.nq + 2 * a.nkv) * HD;
  const size_t here = exchange_row(use >> 1), before = exchange_row((use >> 1) + 2);
  const float* src = silu ? a.sum_o + here * H : a.sum_d + before * H;
  uint16_t *out = (silu ? a.act : a.qkv) + here * features, *clear = (silu ? a.act : a.qkv) + before * features;
  const uint32_t xs = base + a.off_x;  // [TILE][H] bf16, row_bytes(H) apart
  const uint32_t per_row = 65536u / R + 1;  // i / R for i < TILE * R
  // the weights' fragments stay in registers; they are usually there before the stream is
  const bool third = R > 32;  // (without it those fragments are the last row's, unused)
  uint4 w[MT][2][KN];
  wait_weights(&sh.bar_a, use & 1);
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) load_fragments(w[m][h], base + a.off_a + min(m * 16 + h * 8 + t.g, R - 1) * (H * 2) + t.warp * (KN * 64) + t.c * 16, min(m * 16 + h * 8 + t.g, R - 1));
  int turn = 0;
#pragma unroll 1
  for (int t0 = 0; t0 < rows; t0 += TILE, turn ^= 1) {
    const int n = min(TILE, rows - t0);
    // The tile's rows are normalised by as many warps each as there are.
    const int per = n == 1 ? 8 : n == 2 ? 4 : n <= 4 ? 2 : 1, row = t.warp / per, span = H / per, k0 = (t.warp - row * per) * span + t.lane * 4;
    constexpr int NV = H / 128;  // 4-element pieces of a row per lane
    uint4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = make_uint4(0, 0, 0, 0);
    if (row < n) {
      const size_t at = static_cast<size_t>(t0 + row) * H + k0;
      if (from_x) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (i * 128 < span) {
            const uint2 x = __ldcg(reinterpret_cast<const uint2*>(a.x + at + i * 128));
            v[i] = make_uint4(x.x << 16, x.x & 0xffff0000u, x.y << 16, x.y & 0xffff0000u);
          }
      } else {
        uint32_t tries = 0;
        uint64_t since = 0;
        bool bad;
        do {
#pragma unroll
          for (int i = 0; i < NV; ++i)
            if (i * 128 < span) v[i] = ld_x4(src + at + i * 128);
          bad = false;
#pragma unroll
          for (int i = 0; i < NV; ++i) bad |= unwritten(v[i]);
        } while (t.again(bad, tries, since));
      }
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const float x = __uint_as_float(v[i].x), y = __uint_as_float(v[i].y), z = __uint_as_float(v[i].z), u = __uint_as_float(v[i].w);
        ss += (x * x + y * y) + (z * z + u * u);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (t.lane == 0) sh.squares[row * 8 + t.warp - row * per] = ss;
    }
    __syncthreads();
    if (row < n) {
      const float4 p = *reinterpret_cast<const float4*>(sh.squares + row * 8), q = *reinterpret_cast<const float4*>(sh.squares + row * 8 + 4);
      const float ss = per == 1 ? p.x : per == 2 ? p.x + p.y : per == 4 ? (p.x + p.y) + (p.z + p.w) : ((p.x + p.y) + (p.z + p.w)) + ((q.x + q.y) + (q.z + q.w));
      const float rstd = rsqrtf(ss / static_cast<float>(H) + a.eps);
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (i * 128 < span) {
          const uint2 nw = lds_v2(base + a.off_vec + (k0 + i * 128) * 2);
          sts_v2(xs + row * row_bytes(H) + (k0 + i * 128) * 2,
                 b2::mul_bf16x2(b2::pack_bf16(__uint_as_float(v[i].x) * rstd, __uint_as_float(v[i].y) * rstd), nw.x),
                 b2::mul_bf16x2(b2::pack_bf16(__uint_as_float(v[i].z) * rstd, __uint_as_float(v[i].w) * rstd), nw.y));
        }
    }
    __syncthreads();
    float acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][e] = 0.f;
#pragma unroll
    for (int kc = 0; kc < KN; ++kc) {
      const uint4 x = lds_v4(xs + min(t.g, n - 1) * row_bytes(H) + (t.warp * KN + kc) * 64 + t.c * 16);  // (tokens past the tile's are not stored)
#pragma unroll
      for (int m = 0; m < MT; ++m)
        if (m < 2 || third) mma(acc[m], w[m][0][kc].x, w[m][1][kc].x, w[m][0][kc].y, w[m][1][kc].y, x.x, x.y);
#pragma unroll
      for (int m = 0; m < MT; ++m)
        if (m < 2 || third) mma(acc[m], w[m][0][kc].z, w[m][1][kc].z, w[m][0][kc].w, w[m][1][kc].w, x.z, x.w);
    }
    float* scratch = reinterpret_cast<float*>(smem + a.off_s) + turn * (WARPS * TILE * R);  // [warp][token][weight row]
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (t.c * 2 + e < n) {
        float* p = scratch + (t.warp * TILE + t.c * 2 + e) * R + t.g;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (m * 16 + h * 8 + t.g < R) p[m * 16 + h * 8] = acc[m][h * 2 + e];
      }
    __syncthreads();
#pragma unroll 1
    for (int i0 = t.warp * 32; i0 < n * R; i0 += THREADS) {
      const int i = min(i0 + t.lane, n * R - 1), token = (i * per_row) >> 16, col = i - token * R;
      float s[WARPS];
#pragma unroll
      for (int k = 0; k < WARPS; ++k) s[k] = scratch[k * TILE * R + i];
#pragma unroll
      for (int o = WARPS / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; ++k) s[k] += s[k + o];
      float y = s[0], next_y;
      if (silu) {
        y = b2::bf16_round(y);
        y = b2::silu_mul(y, __shfl_down_sync(0xffffffffu, y, 1));
      }
      next_y = __shfl_down_sync(0xffffffffu, y, silu ? 2 : 1);
      if (i0 + t.lane < n * R && (col & (silu ? 3 : 1)) == 0) {
        const size_t at = static_cast<size_t>(t0 + token) * features + (silu ? (r0 + col) >> 1 : r0 + col);
        st_x1(out + at, b2::pack_bf16(y, next_y));
        st_x1(clear + at, UNWRITTEN);
      }
    }
  }
  if (t.tid == 0) load_a(use + 1);  // everyone has its weights' fragments and is through with the norm's weights
}

// Projection added to the residual stream in buffer B: use 2 l is layer l's o, use 2 l + 1 its down.  This CTA's columns of the stream, at
// most 8, stay in shared memory; all of them go out in fp32 for the next norm.
__device__ __forceinline__ void add_project(int use) {
  const Place t;
  Shared& sh = shared();
  const Args& a = sh.args;
  const bool down = use & 1;
  const int rows = sh.rows, r0 = sh.h0, R = sh.h1 - r0, K = down ? a.inter : a.nq * HD, batches = K >> 10;
  const size_t here = exchange_row(use >> 1), before = exchange_row((use >> 1) + 2);
  const uint16_t* x = (down ? a.act : a.attn) + here * K;
  float *out = (down ? a.sum_d : a.sum_o) + here * H, *clear = (down ? a.sum_d : a.sum_o) + before * H;
  float* own = reinterpret_cast<float*>(smem + a.off_own);
  uint4 w[MAX_KB][KB], v[MAX_KB][KB];
  wait_weights(&sh.bar_b, use & 1);
#pragma unroll
  for (int i = 0; i < MAX_KB; ++i) load_fragments(w[i], b2::smem_u32(smem) + a.off_b + min(t.g, R - 1) * (K * 2) + min(i, batches - 1) * 2048 + t.warp * (KB * 64) + t.c * 16, min(t.g, R - 1));
  if (down) {  // the order of what is set back and used again (see the buffers between phases)
    __syncthreads();
    __threadfence();
  }
  int turn = 0;
#pragma unroll 1
  for (int t0 = 0; t0 < rows; t0 += TILE, turn ^= 1) {
    const int n = min(TILE, rows - t0);
    const uint16_t* p = x + static_cast<size_t>(t0 + min(t.g, n - 1)) * K + t.warp * (KB * 32) + t.c * 8;  // (tokens past the tile's are not stored)
    uint32_t tries = 0;
    uint64_t since = 0;
    bool bad;
    do {
#pragma unroll
      for (int i = 0; i < MAX_KB; ++i)
#pragma unroll
        for (int kc = 0; kc < KB; ++kc) v[i][kc] = i < batches ? ld_x4(p + i * 1024 + kc * 32) : make_uint4(0, 0, 0, 0);
      bad = false;
#pragma unroll
      for (int i = 0; i < MAX_KB; ++i)
#pragma unroll
        for (int kc = 0; kc < KB; ++kc) bad |= unwritten(v[i][kc]);
    } while (t.again(bad, tries, since));
    float acc[2][4] = {};
#pragma unroll
    for (int i = 0; i < MAX_KB; ++i) {
      if (i >= batches) break;
#pragma unroll
      for (int kc = 0; kc < KB; ++kc) {
        mma(acc[0], w[i][kc].x, 0u, w[i][kc].y, 0u, v[i][kc].x, v[i][kc].y);
        mma(acc[1], w[i][kc].z, 0u, w[i][kc].w, 0u, v[i][kc].z, v[i][kc].w);
      }
    }
    float* scratch = reinterpret_cast<float*>(smem + a.off_small) + turn * (WARPS * TILE * 8);  // [warp][token][weight row]
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (t.c * 2 + e < n) scratch[(t.warp * TILE + t.c * 2 + e) * 8 + t.g] = acc[0][e] + acc[1][e];
    __syncthreads();
    const int token = t.tid >> 3, col = t.tid & 7;
    if (token < n && col < R) {
      float s[WARPS];
#pragma unroll
      for (int k = 0; k < WARPS; ++k) s[k] = scratch[k * TILE * 8 + t.tid];
#pragma unroll
      for (int o = WARPS / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; ++k) s[k] += s[k + o];
      float* o = own + (t0 + token) * 8 + col;
      const float y = s[0] + b2::bf16_round(*o);  // the stream carried on is bf16; norms see the sum before its rounding
      *o = y;
      const size_t at = static_cast<size_t>(t0 + token) * H + r0 + col;
      st_x1(out + at, __float_as_uint(y));
      st_x1(clear + at, UNWRITTEN);
    }
  }
  if (t.tid == 0) load_b(use + 1);
}

// ---- attention ---------------------------------------------------------------------------------------------------
// Norm (weights at `norm`, or none) and rotation of a head's row, with the roundings of qk_norm_rope_store_kernel: a quad holds a row, lane
// c dimensions 32 j + 8 c .. + 7 in v[j].
__device__ __forceinline__ void finish_head(uint4 (&v)[4], const uint16_t* norm, float eps, const float* factors, int c) {
  if (norm != nullptr) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x[8];
      b2::unpack8(v[j], x);
      ss += ((x[0] * x[0] + x[1] * x[1]) + (x[2] * x[2] + x[3] * x[3])) + ((x[4] * x[4] + x[5] * x[5]) + (x[6] * x[6] + x[7] * x[7]));
    }
    const float rstd = rsqrtf(quad_sum(ss) / static_cast<float>(HD) + eps);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x[8];
      b2::unpack8(v[j], x);
      v[j] = b2::normed(x, rstd, *reinterpret_cast<const uint4*>(norm + j * 32 + c * 8));
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {  // dimension d turns with d + 64
    uint32_t lo[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, hi[4] = {v[j + 2].x, v[j + 2].y, v[j + 2].z, v[j + 2].w};
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const float4 co = __ldg(reinterpret_cast<const float4*>(factors + j * 32 + c * 8 + e * 2)), si = __ldg(reinterpret_cast<const float4*>(factors + HD / 2 + j * 32 + c * 8 + e * 2));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float c0 = k == 0 ? co.x : co.z, c1 = k == 0 ? co.y : co.w, s0 = k == 0 ? si.x : si.z, s1 = k == 0 ? si.y : si.w;
        const float a0 = b2::bf16_lo(lo[e + k]), a1 = b2::bf16_hi(lo[e + k]), b0 = b2::bf16_lo(hi[e + k]), b1 = b2::bf16_hi(hi[e + k]);
        // separate roundings of the products, as the eager reference computes them
        lo[e + k] = b2::pack_bf16(__fsub_rn(__fmul_rn(a0, c0), __fmul_rn(b0, s0)), __fsub_rn(__fmul_rn(a1, c1), __fmul_rn(b1, s1)));
        hi[e + k] = b2::pack_bf16(__fadd_rn(__fmul_rn(b0, c0), __fmul_rn(a0, s0)), __fadd_rn(__fmul_rn(b1, c1), __fmul_rn(a1, s1)));
      }
    }
    v[j] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    v[j + 2] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  }
}

// element of a cache at which a token's row begins
__device__ __forceinline__ int64_t cache_row(const Args& a, int b, int token, int head) {
  const int blk = min(max(0, __ldg(a.tables + b * a.bt_stride + (token >> a.block_shift))), a.num_blocks - 1);  // inside the cache whatever the table holds
  const int slot = (blk << a.block_shift) + (token & ((1 << a.block_shift) - 1));
  return (static_cast<int64_t>(slot) * a.nkv + head) * HD;
}

// New keys and values into the cache ahead of the attention of any row, for batches in which a row may read another row's new token.
__device__ __forceinline__ void store_new_rows(int l) {
  const Place t;
  const Args& a = shared().args;
  const b2_stack_layer& L = a.layer[l];
  const int qkv_w = (a.nq + 2 * a.nkv) * HD, rows = shared().rows;
  const uint16_t* qkv = a.qkv + exchange_row(l) * qkv_w;
#pragma unroll 1
  for (int i = blockIdx.x * WARPS + t.warp; i < rows * a.nkv; i += gridDim.x * WARPS) {
    const int b = i / a.nkv, head = i - b * a.nkv, slot = __ldg(a.slots + b);
    if (slot < 0 || slot >= a.num_blocks << a.block_shift) continue;
    const uint16_t* src = qkv + static_cast<size_t>(b) * qkv_w + (a.nq + head) * HD + t.c * 8;
    uint4 v[4];  // quad 0 the key, the others the value
    uint32_t tries = 0;
    uint64_t since = 0;
    bool bad;
    do {
      bad = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = ld_x4(src + (t.g > 0 ? a.nkv * HD : 0) + j * 32);
#pragma unroll
      for (int j = 0; j < 4; ++j) bad |= unwritten(v[j]);
    } while (t.again(bad, tries, since));
    uint4 k[4] = {v[0], v[1], v[2], v[3]};
    finish_head(k, L.k_norm != nullptr ? shared().qk_norms + HD : nullptr, a.qk_eps, a.cos_sin + __ldg(a.positions + b) * HD, t.c);
    if (t.g < 2) {
      uint16_t* to = static_cast<uint16_t*>(t.g == 0 ? L.k_cache : L.v_cache) + (static_cast<int64_t>(slot) * a.nkv + head) * HD + t.c * 8;
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(to + j * 32) = t.g == 0 ? k[j] : v[j];
    }
  }
}

__device__ __forceinline__ void put_part(float* slot, const float (&o)[16][2], float m, float l, int g, int c, int group) {
  if (g >= group) return;
#pragma unroll
  for (int j = 0; j < 16; ++j) *reinterpret_cast<float2*>(slot + g * HD + j * 8 + c * 2) = make_float2(o[j][0], o[j][1]);
  if (c == 0) {
    slot[MAX_GROUP * HD + g] = m;
    slot[MAX_GROUP * HD + MAX_GROUP + g] = l;
  }
}
// One layer's exchange buffers, and the counterparts of the layer before.
struct Exchange {
  uint16_t *qkv, *attn, *attn_clear;
  float *parts, *parts_clear;  // [CTAs][PART]
};

// The parts of an item (units [begin, end)) that this CTA's warps hold, combined by the warp with the first of them, `mine`.  Where the
// item spans CTAs, the one with its beginning takes the others' combined parts as they arrive.  16 lanes a head, 8 dimensions each.
__device__ __forceinline__ void combine(const Place& t, const Exchange& x, int item, int begin, int end, const float* mine, const float* first_parts) {
  const Shared& sh = shared();
  const Args& a = sh.args;
  const int r = t.lane >> 4, i16 = t.lane & 15, n = sh.u1 - sh.u0, stop = min(end, sh.u1);
  const bool active = r < a.group;
  // lane i knows the maximum and the sum of part i; the outputs are then summed with weights that are known
  const float* part = nullptr;
  if (i16 < WARPS - t.warp) {
    const int w = t.warp + i16, b0 = sh.u0 + share(n, w, WARPS), b1 = sh.u0 + share(n, w + 1, WARPS);
    if (i16 == 0) part = mine;
    else if (b0 < stop && b1 > b0) part = first_parts + w * PART;
  }
  const unsigned int there = __ballot_sync(0xffffffffu, part != nullptr) & 0xffffu;
  const float pm = part != nullptr && active ? part[MAX_GROUP * HD + r] : -INFINITY, pl = part != nullptr && active ? part[MAX_GROUP * HD + MAX_GROUP + r] : 0.f;
  float m = pm;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  const float f = pm == -INFINITY ? 0.f : exp2f(pm - m);
  float l = f * pl, o[8] = {};
#pragma unroll
  for (int k = 8; k > 0; k >>= 1) l += __shfl_xor_sync(0xffffffffu, l, k);
  auto add = [&](float by, const uint4& p, const uint4& q) {
    o[0] += by * __uint_as_float(p.x); o[1] += by * __uint_as_float(p.y); o[2] += by * __uint_as_float(p.z); o[3] += by * __uint_as_float(p.w);
    o[4] += by * __uint_as_float(q.x); o[5] += by * __uint_as_float(q.y); o[6] += by * __uint_as_float(q.z); o[7] += by * __uint_as_float(q.w);
  };
#pragma unroll 2
  for (int i = 0; i < WARPS; ++i) {
    const float fi = __shfl_sync(0xffffffffu, f, i, 16);
    if ((there >> i & 1) == 0) continue;
    const uint4* p = reinterpret_cast<const uint4*>((i == 0 ? mine : first_parts + (t.warp + i) * PART) + t.lane * 8);
    add(fi, p[0], p[1]);
  }
  if (begin < sh.u0) {  // its beginning is another CTA's
    const size_t at = static_cast<size_t>(blockIdx.x) * PART;
    const float none = __uint_as_float(UNWRITTEN);
    if (active) {
      st_x4(x.parts + at + t.lane * 8, make_float4(o[0], o[1], o[2], o[3]));
      st_x4(x.parts + at + t.lane * 8 + 4, make_float4(o[4], o[5], o[6], o[7]));
      if (i16 < 2) st_x1(x.parts + at + MAX_GROUP * HD + i16 * MAX_GROUP + r, __float_as_uint(i16 == 0 ? m : l));
      st_x4(x.parts_clear + at + t.lane * 8, make_float4(none, none, none, none));
      st_x4(x.parts_clear + at + t.lane * 8 + 4, make_float4(none, none, none, none));
      if (i16 < 2) st_x1(x.parts_clear + at + MAX_GROUP * HD + i16 * MAX_GROUP + r, UNWRITTEN);
    }
    return;
  }
  if (end > sh.u1) {
    const int parts = sh.deal.cta_of(end - 1) - static_cast<int>(blockIdx.x);  // of the following CTAs
    constexpr int BATCH = 4;
#pragma unroll 1
    for (int k0 = 1; k0 <= parts; k0 += BATCH) {
      uint4 p[BATCH], q[BATCH];
      uint32_t qm[BATCH], ql[BATCH], tries = 0;
      uint64_t since = 0;
      bool bad;
      do {
        bad = false;
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {
          const float* from = x.parts + static_cast<size_t>(blockIdx.x + min(k0 + k, parts)) * PART;  // (past the last: it again, unused)
          p[k] = ld_x4(from + t.lane * 8);
          q[k] = ld_x4(from + t.lane * 8 + 4);
          qm[k] = ld_x1(from + MAX_GROUP * HD + r);
          ql[k] = ld_x1(from + MAX_GROUP * HD + MAX_GROUP + r);
        }
#pragma unroll
        for (int k = 0; k < BATCH; ++k) bad |= active && (unwritten(p[k]) || unwritten(q[k]) || max(qm[k], ql[k]) == UNWRITTEN);
      } while (t.again(bad, tries, since));
      float mx = m;
#pragma unroll
      for (int k = 0; k < BATCH; ++k) mx = k0 + k <= parts ? fmaxf(mx, __uint_as_float(qm[k])) : mx;
      const float keep = exp2f(m - mx);  // (a part has at least one token: its maximum is finite, or its sum NaN)
      l *= keep;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] *= keep;
#pragma unroll
      for (int k = 0; k < BATCH; ++k)
        if (k0 + k <= parts) {  // (with whatever weight: what is NaN in a part is NaN in the result)
          const float by = exp2f(__uint_as_float(qm[k]) - mx);
          l += by * __uint_as_float(ql[k]);
          add(by, p[k], q[k]);
        }
      m = mx;
    }
  }
  if (active) {
    const size_t at = static_cast<size_t>(item) * a.group * HD + t.lane * 8;
    const float inv = l > 0.f ? 1.f / l : 0.f;
    st_x2(x.attn + at, b2::pack_bf16(o[0] * inv, o[1] * inv), b2::pack_bf16(o[2] * inv, o[3] * inv));
    st_x2(x.attn + at + 4, b2::pack_bf16(o[4] * inv, o[5] * inv), b2::pack_bf16(o[6] * inv, o[7] * inv));
    st_x2(x.attn_clear + at, UNWRITTEN, UNWRITTEN);
    st_x2(x.attn_clear + at + 4, UNWRITTEN, UNWRITTEN);
  }
}

__device__ __forceinline__ void attention(int l_no) {
  const Place t;
  const Shared& sh = shared();
  const Args& a = sh.args;
  const b2_stack_layer& L = a.layer[l_no];
  const int Q = a.nq * HD, qkv_w = Q + 2 * a.nkv * HD, rows = sh.rows;
  const size_t here = exchange_row(l_no), before = exchange_row(l_no + 2);
  const Exchange x = {a.qkv + here * qkv_w, a.attn + here * Q, a.attn + before * Q, a.parts + static_cast<size_t>(l_no % 3) * gridDim.x * PART,
                      a.parts + static_cast<size_t>((l_no + 2) % 3) * gridDim.x * PART};
  // rows without a context: their output is zero
#pragma unroll 1
  for (int b = blockIdx.x; b < rows; b += gridDim.x)
    if (sh.len[b] == 0)
#pragma unroll 1
      for (int i = t.tid * 2; i < Q; i += THREADS * 2) {
        st_x1(x.attn + static_cast<size_t>(b) * Q + i, 0);
        st_x1(x.attn_clear + static_cast<size_t>(b) * Q + i, UNWRITTEN);
      }
  const int u0 = sh.u0, n = sh.u1 - u0, w0 = u0 + share(n, t.warp, WARPS), w1 = u0 + share(n, t.warp + 1, WARPS);
  if (n == 0) return;  // (the whole CTA)
  unsigned char* v_buf = smem + a.off_s + t.warp * (2 * V_BYTES);  // this warp's rows of V, two groups
  const uint32_t v_smem = b2::smem_u32(v_buf);
  float* first_parts = reinterpret_cast<float*>(smem + a.off_s + WARPS * (2 * V_BYTES));  // [WARPS][PART]
  unsigned char* new_rows = smem + a.off_small + t.warp * ((MAX_GROUP + 2) * HD * 2);     // this warp's query rows, new key, new value
  const int v_tok = (((t.lane >> 3) & 1) << 3) + (t.lane & 7), v_chunk = t.lane >> 4;

  // segments that are parts of an item: the warp's first, and one that is still open when its range ends
  int open_item[2] = {}, open_begin[2] = {}, open_end[2] = {};
  bool later = false;

  int pos = w0, b = sh.start[t.warp];
#pragma unroll 1
  while (pos < w1) {
    while (sh.first[b + 1] * a.nkv <= pos) ++b;
    const int groups = sh.first[b + 1] - sh.first[b], in_seq = pos - sh.first[b] * a.nkv;
    const int head = in_seq / groups, g0 = in_seq - head * groups, g1 = min(groups, g0 + w1 - pos), len = sh.len[b];
    const int item_begin = pos - g0;
    pos += g1 - g0;
    // the row's own new key and value: normalised, rotated and put into the cache by the warp that reads the last group
    const bool fresh = sh.staged == 0 && g1 == groups;

    uint4 kf[2][4], qf[4];
    float o[16][2], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j][0] = o[j][1] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) qf[j] = make_uint4(0, 0, 0, 0);
    float s[2][2] = {};
    // one turn more than there are groups: each multiplies its group's keys, sends for the next group and finishes its own; the
    // first only sends, for what is older than this step, and then waits for the new rows
#pragma unroll 1
    for (int grp = g0 - 1; grp < g1; ++grp) {
      const int left = len - grp * GROUP_TOKENS;  // tokens of the group that exist
      const bool has_new = fresh && grp == groups - 1;
      if (grp >= g0) {
        if (has_new) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (h * 8 + t.g == left - 1) {
#pragma unroll
              for (int j = 0; j < 4; ++j) kf[h][j] = *reinterpret_cast<const uint4*>(new_rows + MAX_GROUP * HD * 2 + j * 64 + t.c * 16);
            }
        }
        float s2[2][2] = {};
#pragma unroll
        for (int h = 0; h < 2; ++h) s[h][0] = s[h][1] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            b2::mma_rows8(s[h][0], s[h][1], qf[j].x, qf[j].y, kf[h][j].x, kf[h][j].y);
            b2::mma_rows8(s2[h][0], s2[h][1], qf[j].z, qf[j].w, kf[h][j].z, kf[h][j].w);
          }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          s[h][0] += s2[h][0];
          s[h][1] += s2[h][1];
        }
      }
      if (grp + 1 < g1) {
        const int tok0 = (grp + 1) * GROUP_TOKENS, there = len - tok0;
        const int64_t step = static_cast<int64_t>(a.nkv) * HD;
        const int64_t at = cache_row(a, b, tok0, head);  // (a group does not cross a block)
        const uint16_t* k_row = static_cast<const uint16_t*>(L.k_cache) + at + t.g * step + t.c * 8;  // keys g and g + 8
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 4; ++j) kf[h][j] = h * 8 + t.g < there ? b2::ld_cg_v4(k_row + h * 8 * step + j * 32) : make_uint4(0, 0, 0, 0);
        if (grp + AHEAD < g1) {  // further on, to L2: what fragments and buffers hold is too little for DRAM's latency
          const int token = min((grp + AHEAD) * GROUP_TOKENS + (t.lane >> 1), len - 1);
          const int64_t far = cache_row(a, b, token, head) + (t.lane & 1) * 64;  // 128 bytes of a row of 256
          prefetch_l2(static_cast<const uint16_t*>(L.k_cache) + far);
          prefetch_l2(static_cast<const uint16_t*>(L.v_cache) + far);
        }
        const int chunk = t.lane & 15, tok = t.lane >> 4;
        const uint16_t* v_row = static_cast<const uint16_t*>(L.v_cache) + at + tok * step + chunk * 8;
        const uint32_t to = v_smem + ((grp + 1) & 1) * V_BYTES + tok * (HD * 2);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const bool any = i * 2 + tok < there;
          cp_async16(to + i * (4 * HD) + ((chunk ^ ((i * 2 + tok) & 7)) << 4), any ? v_row + i * 2 * step : v_row, any);
        }
      }
      cp_async_commit();
      if (grp < g0) {
        // Quads 0 and 1 take the query rows, 2 the new key, 3 the new value.
        uint4 r[4];
        const int what = t.g < MAX_GROUP ? min(t.g, a.group - 1) + head * a.group : t.g == 2 ? a.nq + head : a.nq + a.nkv + head;
        const uint16_t* raw = x.qkv + static_cast<size_t>(b) * qkv_w + what * HD + t.c * 8;
        const bool need = t.g < MAX_GROUP || (fresh && t.g < 4);
        const float* factors = a.cos_sin + __ldg(a.positions + b) * HD;
        uint32_t tries = 0;
        uint64_t since = 0;
        bool bad;
        do {
#pragma unroll
          for (int j = 0; j < 4; ++j) r[j] = need ? ld_x4(raw + j * 32) : make_uint4(0, 0, 0, 0);
          bad = false;
#pragma unroll
          for (int j = 0; j < 4; ++j) bad |= unwritten(r[j]);
        } while (t.again(bad, tries, since));
        uint4 f[4] = {r[0], r[1], r[2], r[3]};
        finish_head(f, L.q_norm == nullptr ? nullptr : t.g < MAX_GROUP ? sh.qk_norms : sh.qk_norms + HD, a.qk_eps, factors, t.c);
        if (t.g < a.group) {
#pragma unroll
          for (int j = 0; j < 4; ++j) qf[j] = f[j];
        }
        if (fresh && (t.g == 2 || t.g == 3)) {
          uint16_t* to = static_cast<uint16_t*>(t.g == 2 ? L.k_cache : L.v_cache) + (static_cast<int64_t>(__ldg(a.slots + b)) * a.nkv + head) * HD + t.c * 8;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 y = t.g == 2 ? f[j] : r[j];
            *reinterpret_cast<uint4*>(to + j * 32) = y;
            *reinterpret_cast<uint4*>(new_rows + t.g * (HD * 2) + j * 64 + t.c * 16) = y;
          }
        }
        __syncwarp();
        continue;
      }
      float mx = m;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          s[h][e] = h * 8 + t.c * 2 + e < left ? s[h][e] * a.scale_log2 : -INFINITY;
          mx = fmaxf(mx, s[h][e]);
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
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          p[h][e] = b2::ex2(s[h][e] - m);
          l += p[h][e];
        }
      const uint32_t p0 = b2::pack_bf16(p[0][0], p[0][1]), p1 = b2::pack_bf16(p[1][0], p[1][1]), v_group = v_smem + (grp & 1) * V_BYTES;
      cp_async_wait_but_one();
      __syncwarp();
      if (has_new) {
        if (t.lane < 16)
          *reinterpret_cast<uint4*>(v_buf + (grp & 1) * V_BYTES + (left - 1) * (HD * 2) + ((t.lane ^ ((left - 1) & 7)) << 4)) = *reinterpret_cast<const uint4*>(new_rows + 3 * HD * 2 + t.lane * 16);
        __syncwarp();
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t vf[4];
        b2::ldmatrix_x4_trans(vf, v_group + v_tok * (HD * 2) + (((j * 2 + v_chunk) ^ (v_tok & 7)) << 4));
        b2::mma_rows8(o[2 * j][0], o[2 * j][1], p0, p1, vf[0], vf[1]);
        b2::mma_rows8(o[2 * j + 1][0], o[2 * j + 1][1], p0, p1, vf[2], vf[3]);
      }
      __syncwarp();
    }
    l = quad_sum(l);
    if (g0 == 0 && g1 == groups) {  // all of the item: done
      const float inv = l > 0.f ? 1.f / l : 0.f;
      if (t.g < a.group) {
        const size_t at = (static_cast<size_t>(b) * a.nkv + head) * a.group * HD + t.g * HD + t.c * 2;
#pragma unroll
        for (int j = 0; j < 16; ++j) st_x1(x.attn + at + j * 8, b2::pack_bf16(o[j][0] * inv, o[j][1] * inv));
#pragma unroll
        for (int j = 0; j < 16; ++j) st_x1(x.attn_clear + at + j * 8, UNWRITTEN);
      }
    } else {
      // a warp's first segment has a place of its own; a later one that stays open is its last, and V's buffer is free then
      put_part(later ? reinterpret_cast<float*>(v_buf) : first_parts + t.warp * PART, o, m, l, t.g, t.c, a.group);
      const int i = later ? 1 : 0;
      open_item[i] = b * a.nkv + head;
      open_begin[i] = item_begin;
      open_end[i] = item_begin + groups;
    }
    later = true;
  }
  __syncthreads();
  // The warp that holds an item's first part in this CTA combines all of them: its own and the first segments of the following warps.
#pragma unroll 1
  for (int i = 0; i < 2; ++i)
    if (open_end[i] > 0 && (i == 1 || w0 <= max(open_begin[0], u0)))
      combine(t, x, open_item[i], open_begin[i], open_end[i], i == 0 ? first_parts + t.warp * PART : reinterpret_cast<const float*>(v_buf), first_parts);
}

// The first bytes of this warp's keys and values of the coming attention on their way to L2 (they are older than this step).
__device__ __forceinline__ void prefetch_kv(int l) {
  const Place t;
  const Shared& sh = shared();
  const Args& a = sh.args;
  const b2_stack_layer& L = a.layer[l];
  const int n = sh.u1 - sh.u0, w0 = sh.u0 + share(n, t.warp, WARPS), w1 = min(sh.u0 + share(n, t.warp + 1, WARPS), w0 + AHEAD);
  int b = sh.start[t.warp];
#pragma unroll 1
  for (int u = w0; u < w1; ++u) {
    while (sh.first[b + 1] * a.nkv <= u) ++b;
    const int groups = sh.first[b + 1] - sh.first[b], in_seq = u - sh.first[b] * a.nkv, head = in_seq / groups;
    const int token = (in_seq - head * groups) * GROUP_TOKENS + (t.lane >> 1);
    if (token >= sh.len[b]) continue;
    const int64_t at = cache_row(a, b, token, head) + (t.lane & 1) * 64;  // 128 bytes of a row of 256
    prefetch_l2(static_cast<const uint16_t*>(L.k_cache) + at);
    prefetch_l2(static_cast<const uint16_t*>(L.v_cache) + at);
  }
}

// ---- the step ------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 1) decode_stack_kernel(const __grid_constant__ Args args) {
  Shared& sh = shared();
  const Args& a = sh.args;
  {
    const Place t;
#pragma unroll 1
    for (int i = t.tid; i < static_cast<int>(sizeof(Args) / 8); i += THREADS) reinterpret_cast<uint64_t*>(&sh.args)[i] = reinterpret_cast<const uint64_t*>(&args)[i];
    const int G = gridDim.x, cta = blockIdx.x, N = (args.nq + 2 * args.nkv) * HD, I = args.inter;
    if (t.tid == 0) {
      b2::mbar_init(b2::smem_u32(&sh.bar_a), 1);
      b2::mbar_init(b2::smem_u32(&sh.bar_b), 1);
      b2::mbar_fence_init();
      sh.abort = 0;
      sh.staged = 0;
      // (whole 4-byte words of what qkv and gate/up write)
      sh.q0 = 4 * share(N / 4, cta, G);
      sh.q1 = 4 * share(N / 4, cta + 1, G);
      sh.h0 = share(H, cta, G);
      sh.h1 = share(H, cta + 1, G);
      sh.p0 = 4 * share(I / 2, cta, G);
      sh.p1 = 4 * share(I / 2, cta + 1, G);
    }
    __syncthreads();
    if (t.tid == 0) {
      load_a(0);
      load_b(0);
    }
    // contexts, in groups per sequence; rows past the last one with a context are padding
    if (t.warp == 0) {
      const int b = t.lane, len = b < a.rows ? max(0, min(__ldg(a.lens + b), a.bt_width << a.block_shift)) : 0, groups = (len + GROUP_TOKENS - 1) / GROUP_TOKENS;
      int incl = groups;
#pragma unroll
      for (int o = 1; o < MAX_ROWS; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (t.lane >= o) incl += up;
      }
      if (b < MAX_ROWS) {
        sh.len[b] = len;
        sh.first[b + 1] = incl;
      }
      const int live = __reduce_max_sync(0xffffffffu, len > 0 ? b + 1 : 0), most = __reduce_max_sync(0xffffffffu, groups);
      if (t.lane == 0) {
        sh.first[0] = 0;
        sh.rows = live;
        sh.most = most;
      }
    }
    __syncthreads();
    const int rows = sh.rows;
    // A row whose new token goes where its table says, into a block that no other row reads, is attended to by warps that take the
    // new key from the projection.  Otherwise (several new tokens of one sequence in a batch, a frozen row) all new rows are stored
    // before any is attended to.
    if (t.tid < rows) {
      const int b = t.tid, n = sh.len[b], slot = __ldg(a.slots + b);
      sh.block[b] = slot >= 0 ? slot >> a.block_shift : -1;
      const int64_t want = n > 0 ? (static_cast<int64_t>(__ldg(a.tables + b * a.bt_stride + ((n - 1) >> a.block_shift))) << a.block_shift) + ((n - 1) & ((1 << a.block_shift) - 1)) : -1;
      if (slot < 0 || want != slot || slot >= a.num_blocks << a.block_shift) sh.staged = 1;
    }
    if (t.tid == 0) {
      const Deal d = deal_groups(sh.first, rows, a.nkv, sh.most, G);
      sh.deal = d;
      sh.u0 = cta < d.ctas ? d.cta_begin(cta) : 0;
      sh.u1 = cta < d.ctas ? d.cta_begin(cta + 1) : 0;
    }
    __syncthreads();
    if (t.lane == 0) {
      const int pos = sh.u0 + share(sh.u1 - sh.u0, t.warp, WARPS);
      int b = 0;
      while (b + 1 < rows && sh.first[b + 1] * a.nkv <= pos) ++b;
      sh.start[t.warp] = b;
    }
#pragma unroll 1
    for (int b = t.warp; b < rows; b += WARPS)
#pragma unroll 1
      for (int i = t.lane; (i << a.block_shift) < sh.len[b]; i += 32) {
        const int blk = __ldg(a.tables + b * a.bt_stride + i);
#pragma unroll 1
        for (int j = 0; j < rows; ++j)
          if (j != b && sh.block[j] == blk) sh.staged = 1;
      }
    // this CTA's columns of the residual stream
    float* own = reinterpret_cast<float*>(smem + a.off_own);
#pragma unroll 1
    for (int i = t.tid; i < rows * 8; i += THREADS)
      if ((i & 7) < sh.h1 - sh.h0) own[i] = __uint_as_float(static_cast<uint32_t>(a.x[static_cast<size_t>(i >> 3) * H + sh.h0 + (i & 7)]) << 16);
    __syncthreads();
  }
  const int uses = sh.rows > 0 ? 2 * a.layers : 0;
#pragma unroll 1
  for (int use = 0; use < uses; ++use) {  // two a layer: attention, the MLP
    const int l = use >> 1;
    if ((use & 1) == 0) {
      if (a.layer[l].q_norm != nullptr && threadIdx.x < 32)  // (read after the projection's barriers)
        reinterpret_cast<uint4*>(sh.qk_norms)[threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(threadIdx.x < 16 ? a.layer[l].q_norm : a.layer[l].k_norm) + (threadIdx.x & 15));
    }
    norm_project(use);
    if ((use & 1) == 0) {
      __syncthreads();  // (attention's buffers lie where the partial sums were)
      if (sh.staged != 0) {
        store_new_rows(l);
        meet(l + 1);
      }
      attention(l);
    } else if (l + 1 < a.layers && sh.staged == 0) {
      prefetch_kv(l + 1);
    }
    add_project(use);
  }
  {
    const Place t;
    const int rows = sh.rows;
    if (rows == 0) {  // nothing to do, but the first weights are on their way
      wait_weights(&sh.bar_a, 0);
      wait_weights(&sh.bar_b, 0);
    }
    // the final norm, a row per warp; padded rows are zero
#pragma unroll 1
    for (int b = blockIdx.x + gridDim.x * t.warp; b < a.rows; b += gridDim.x * WARPS) {
      uint16_t* out = a.out + static_cast<size_t>(b) * H + t.lane * 8;
      if (b >= rows) {
        for (int i = 0; i < H; i += 256) *reinterpret_cast<uint4*>(out + i) = make_uint4(0, 0, 0, 0);
        continue;
      }
      const float* src = a.sum_d + (exchange_row(a.layers - 1) + b) * H + t.lane * 8;
      float x[4][8], ss = 0.f;
      uint32_t tries = 0;
      uint64_t since = 0;
      bool bad;
      do {
        bad = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 p = ld_x4(src + j * 256), q = ld_x4(src + j * 256 + 4);
          bad |= unwritten(p) || unwritten(q);
          const uint32_t w[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
          for (int e = 0; e < 8; ++e) x[j][e] = __uint_as_float(w[e]);
        }
      } while (t.again(bad, tries, since));
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += x[j][e] * x[j][e];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float rstd = rsqrtf(ss / static_cast<float>(H) + a.eps);
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(out + j * 256) = b2::normed(x[j], rstd, __ldg(reinterpret_cast<const uint4*>(a.final_norm + j * 256 + t.lane * 8)));
    }
    __syncthreads();
    if (sh.abort != 0) {
      for (int i = 0; i < 100; ++i) __nanosleep(2000);  // copies in flight land before the CTA leaves
      if (t.tid == 0) b2::report_timeout(a.status, sh.abort);
    }
  }
}

// ---- host ------------------------------------------------------------------------------------------------------------
constexpr uint32_t SMEM_MAX = 227 * 1024;

struct Layout {
  uint32_t off_a, off_vec, off_b, off_s, off_x, off_small, off_own, smem;
  size_t words, sum_o, sum_d, qkv, attn, act, parts, bytes;  // offsets in the workspace
};
// The rule of what is served.  Hidden size: H alone (see there); a smaller one would fit and is left to the layers, as no model here has one.
// q and MLP widths: the CTAs' shares of a layer have to fit shared memory one projection ahead, and the fragments' arrays above: with
// 148 SMs up to 3072 (Qwen3-0.6B).  Larger layers stream for longer than their launches' overheads and stay on the kernels of the single
// projections.  Rows: tiles of 8 follow one another, and every CTA normalises and takes in all of them.  The 28 layers of
// Qwen3-0.6B in a graph, us, this launch against one launch per projection (the last column with kernels of an earlier state on both sides):
//   context       1 row        8 rows       16 rows       32 rows
//   40          409 / 758     494 / 793    707 / 833    1196 / 935
//   300         472 / 804     637 / 865    843 / 921    1490 / 1055
//   1200        537 / 918     849 / 1104  1204 / 1294   2229 / 1537
//   4000        685 / 1074   1266 / 1473  2025 / 2030
bool layout_of(int rows, int hidden, int nq, int nkv, int I, int G, Layout* p) {
  const int Q = nq * HD, N = (nq + 2 * nkv) * HD;
  if (rows < 1 || rows > MAX_ROWS || nkv < 1 || nq % nkv != 0 || nq / nkv > MAX_GROUP || G < 1) return false;
  if (hidden != H || Q % 1024 != 0 || I % 1024 != 0 || Q < 1024 || I < 1024 || Q > MAX_KB * 1024 || I > MAX_KB * 1024) return false;
  const auto most = [G](int n) { return (n + G - 1) / G; };
  const int rq = 4 * most(N / 4), rp = 4 * most(I / 2), rh = most(H);
  if (rq > MT * 16 || rp > MT * 16 || rh > 8 || H < G || N / 4 < G || I / 2 < G) return false;
  const auto up = [](size_t x, size_t to) { return (x + to - 1) / to * to; };
  uint32_t at = 0;
  const auto room = [&](size_t bytes) {
    const uint32_t here = at;
    at += static_cast<uint32_t>(up(bytes, 128));
    return here;
  };
  room(sizeof(Shared));
  p->off_a = room(std::max(rq, rp) * H * 2);
  p->off_vec = room(H * 2);
  p->off_b = room(rh * std::max(Q, I) * 2);
  // the warps' partial sums and a tile of normalised rows, or attention's V buffers and first parts
  const size_t sums = up(2 * static_cast<size_t>(WARPS) * TILE * std::max(rq, rp) * 4, 128);
  p->off_s = room(std::max<size_t>(sums + TILE * row_bytes(H), WARPS * (2 * V_BYTES + PART * 4)));
  p->off_x = p->off_s + static_cast<uint32_t>(sums);
  p->off_small = room(std::max(2 * WARPS * TILE * 8 * 4, WARPS * (MAX_GROUP + 2) * HD * 2));  // partial sums of o and down; attention's new rows
  p->off_own = room(MAX_ROWS * 8 * 4);
  p->smem = at;
  if (p->smem > SMEM_MAX) return false;
  size_t to = 0;
  const auto place = [&](size_t bytes) {
    const size_t here = to;
    to = up(to + bytes, 256);
    return here;
  };
  const size_t three = 3 * static_cast<size_t>(rows);
  p->words = place(256);
  p->sum_o = place(three * H * 4);
  p->sum_d = place(three * H * 4);
  p->qkv = place(three * N * 2);
  p->attn = place(three * Q * 2);
  p->act = place(three * I * 2);
  p->parts = place(3 * static_cast<size_t>(G) * PART * 4);
  p->bytes = to;
  return true;
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

extern "C" int64_t b2_decode_stack_workspace(b2_ctx* ctx, int rows, int layers, int hidden, int nq, int nkv, int head_dim, int inter, int block_size) {
  Layout p;
  if (ctx == nullptr || ctx->cfg.world != 1 || head_dim != HD || layers < 1 || layers > MAX_LAYERS || block_size < GROUP_TOKENS || (block_size & (block_size - 1)) != 0) return 0;
  return layout_of(rows, hidden, nq, nkv, inter, ctx->num_sms, &p) ? static_cast<int64_t>(p.bytes) : 0;
}

extern "C" int b2_decode_stack(b2_ctx* ctx, const b2_stack_layer* layers, int n_layers, const void* final_norm, int hidden, int nq, int nkv, int head_dim,
                               int inter, float eps, float qk_eps, float scale, const float* cos_sin, const void* x, int rows, const int64_t* positions,
                               const int32_t* context_lens, const int32_t* slot_mapping, const int32_t* block_tables, int64_t bt_stride, int bt_width,
                               int block_size, int num_blocks, void* out, void* workspace, int64_t workspace_bytes, void* stream) {
  if (ctx == nullptr || layers == nullptr || rows < 0) return B2_ERR_ARG;
  if (rows == 0) return B2_OK;
  const int64_t need = b2_decode_stack_workspace(ctx, rows, n_layers, hidden, nq, nkv, head_dim, inter, block_size);
  if (need == 0) return b2::set_error(B2_ERR_UNSUPPORTED, "b2_decode_stack does not serve this shape");
  if (!final_norm || !cos_sin || !x || !positions || !context_lens || !slot_mapping || !block_tables || !out || !workspace || workspace_bytes < need) return B2_ERR_ARG;
  if (bt_width < 1 || bt_stride < bt_width || num_blocks < 1 || static_cast<int64_t>(num_blocks) * block_size > 0x7fffffff) return B2_ERR_ARG;
  if (!aligned16(final_norm) || !aligned16(cos_sin) || !aligned16(x) || !aligned16(out) || !aligned16(workspace)) return B2_ERR_ARG;
  Args a;
  for (int i = 0; i < n_layers; ++i) {
    const b2_stack_layer& l = layers[i];
    for (const void* p : {l.qkv_w, l.o_w, l.gate_up_w, l.down_w, l.in_norm, l.post_norm, static_cast<const void*>(l.k_cache), static_cast<const void*>(l.v_cache)})
      if (p == nullptr || !aligned16(p)) return B2_ERR_ARG;
    if ((l.q_norm == nullptr) != (l.k_norm == nullptr) || !aligned16(l.q_norm) || !aligned16(l.k_norm)) return B2_ERR_ARG;
    a.layer[i] = l;
  }
  memset(static_cast<void*>(a.layer + n_layers), 0, (MAX_LAYERS - n_layers) * sizeof(b2_stack_layer));
  Layout p;
  layout_of(rows, hidden, nq, nkv, inter, ctx->num_sms, &p);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  a.final_norm = static_cast<const uint16_t*>(final_norm);
  a.x = static_cast<const uint16_t*>(x);
  a.out = static_cast<uint16_t*>(out);
  a.positions = positions;
  a.lens = context_lens;
  a.slots = slot_mapping;
  a.tables = block_tables;
  a.bt_stride = bt_stride;
  a.cos_sin = cos_sin;
  a.gave_up = reinterpret_cast<unsigned int*>(ws + p.words);
  a.arrivals = a.gave_up + 32;
  a.sum_o = reinterpret_cast<float*>(ws + p.sum_o);
  a.sum_d = reinterpret_cast<float*>(ws + p.sum_d);
  a.qkv = reinterpret_cast<uint16_t*>(ws + p.qkv);
  a.attn = reinterpret_cast<uint16_t*>(ws + p.attn);
  a.act = reinterpret_cast<uint16_t*>(ws + p.act);
  a.parts = reinterpret_cast<float*>(ws + p.parts);
  a.status = ctx->status_dev;
  a.layers = n_layers;
  a.rows = rows;
  a.nq = nq;
  a.nkv = nkv;
  a.group = nq / nkv;
  a.bt_width = bt_width;
  a.inter = inter;
  for (a.block_shift = 0; (1 << a.block_shift) < block_size; ++a.block_shift) {}
  a.num_blocks = num_blocks;
  a.eps = eps;
  a.qk_eps = qk_eps;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.off_a = p.off_a;
  a.off_vec = p.off_vec;
  a.off_b = p.off_b;
  a.off_s = p.off_s;
  a.off_x = p.off_x;
  a.off_small = p.off_small;
  a.off_own = p.off_own;
  static std::atomic<bool> done[64];  // the opt-in to more than 48 KB of dynamic shared memory belongs to a device
  const int dev = ctx->cfg.device;
  if (dev < 0 || dev >= 64) return b2::set_error(B2_ERR_UNSUPPORTED, "device ordinal %d not supported", dev);
  if (!done[dev].load(std::memory_order_acquire)) {
    B2_CUDA(cudaFuncSetAttribute(decode_stack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    done[dev].store(true, std::memory_order_release);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  B2_CUDA(cudaMemsetAsync(ws, 0xff, p.bytes, s));  // nothing is written yet
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctx->num_sms);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_stack_kernel, a);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // this process may not use all SMs
    cudaGetLastError();
    return b2::set_error(B2_ERR_UNSUPPORTED, "b2_decode_stack: its CTAs cannot all be resident");
  }
  B2_CUDA(e);
  b2::count_launch();
  return B2_OK;
}
