// The products of a step of some tens of tokens (a decode batch of 9 to 128 requests, a short prompt portion; of wide models
// any step of up to 128), each as ONE kernel that leaves finished output.
//
// Such a step streams every weight once, and what it costs beside that is the chain: with K split over blocks
// into float32 planes (gemm_tcgen05.cu) every product is followed by a kernel that adds the planes up, and the planes
// cross the L2 twice. The few-token kernels (gemv_mma.cu) need no sum, but their warps' rings have no room for the
// operand of more tokens. Here a CLUSTER of blocks owns 128 weight rows (the rows of the MMA; the tokens are its
// columns) and shares K out: block r of C takes the r-th range of k-blocks, with its accumulator in tensor
// memory, and finishes the r-th share of the tokens. At the end every block stores each token's sums into the shared memory of the
// block that finishes it; after the cluster's barrier that block adds the C sums in the order of the blocks and runs the
// epilogue. No plane is written and nothing is left to sum:
//
//   q|k|v     a tile of 128 rows holds whole heads (head sizes that divide 128), so a rotation's pair is in one
//             place: bias, rounding, rotation, page write.
//   gate|up   rows alternate in blocks of 16 gate and 16 up: act(gate) x up.
//   o, down   + residual, rounding; and, where an RMSNorm reads the sum next, the operand of the product behind
//             it, sum x norm weight, with the sum of the squares of the tile's columns per token. The product behind it
//             adds the tiles' sums up and applies rsqrt(mean + eps) to its own sums: one factor per token. So the
//             norm needs no launch either, and a layer's products are four kernels instead of seven or eight.
//
// Weights and tokens come by TMA into one ring per block; the weights' first stages are asked for before the
// wait for the kernel before (`early`: the few-token products' rule, see launch_kernel). Mostly 112 KB a block, so that
// two fit an SM and the next product's blocks fill their rings while this one's finish.
//
// What bounds it: the chain, then memory. The four products with their norms in a row, with split K and summing kernels and so: 1,536-wide layers (93.5 MB of
// weights, 14.3 us at the copy rate) 43.3 -> 30.1 us at 40 tokens, 44.3 -> 32.0 at 64, 47.9 -> 37.5 at 100; 3,584-wide (466 MB, 71 us) 104.7 -> 89.1 at
// 64. Of these 3.5 us by issuing the MMAs from uniform registers. A block's time by %clock64, 1,536 wide, 40 tokens, o / q|k|v / down, us after its wait for the
// kernel before: first stage 0.7 / 0.6 / 1.5, MMAs 0.6 / 1.2 / 3.0, stores to the other blocks 0.7, the cluster's barrier 0.6, epilogue 0.8 / 0.7 / 0.8 (100 tokens: stores 1.4,
// barrier 0.7 to 0.9). Sums read from the other blocks' shared memory instead of stored there: a trip there and back behind the barrier, 0.6 us a kernel more;
// norm weight, bias and residual asked for behind the barrier 1.2 us a kernel more.
#include <atomic>

#include "tcgen05.cuh"

using namespace pae;
using namespace pae_tcgen05;

namespace {

constexpr int BM = 128;                // weight rows per tile
// TMA warp, MMA warp, the epilogue's: eight, or sixteen where a block finishes all tokens by itself.
template <bool CLUSTER>
constexpr int EPILOGUE_THREADS = CLUSTER ? 256 : 512;
constexpr int MAX_TOKENS = 128;
constexpr int MAX_STAGES = 12;
constexpr int MAX_CLUSTER = 8;
constexpr int A_BYTES = BM * BK * 2;
constexpr int TAIL_BYTES = 256 /* barriers */ + MAX_TOKENS * 4 /* the tokens' scales */;

enum Kind : int { QKV = 0, RESIDUAL = 1, GATE_SILU = 2, GATE_RELU = 3, GATE_GELU = 4 };
__host__ __device__ constexpr bool is_gate(int kind) { return kind >= GATE_SILU; }
__host__ __device__ constexpr int gate_of(int kind) { return kind == GATE_RELU ? kGateRelu : kind == GATE_GELU ? kGateGeluTanh : kGateSilu; }

struct Params {
  int tokens, n, k_blocks;
  int columns;                   // the MMA's columns: tokens rounded up to 16
  int rows;                      // weight rows per tile: 128, or 64 (the MMA's upper rows then mean nothing and are not read)
  int stages;
  int early;                     // weights may be read before the wait for the kernel before
  // the scale of a normed operand: sums of squares [parts, tokens] of the rows that x stands for, or null
  const float* squares_in;
  int parts_in;
  float width_in, eps;
  // RESIDUAL
  const __nv_bfloat16* residual; // [tokens, n] or null
  __nv_bfloat16* out;            // RESIDUAL: [tokens, n]; gates: [tokens, n / 2]; QKV: [tokens, n]
  const float* gamma;            // [n]: the weight of the norm that reads the sum, or null
  __nv_bfloat16* scaled;         // [tokens, n] = out * gamma
  float* squares;                // [tiles, tokens]
  // QKV
  const float* bias;             // [n] or null
  const float* rotary;           // [tokens, d]: cosines then sines, or null
  const int* slots;              // [tokens] or null
  __nv_bfloat16* keys;           // [pages, kv_heads, page_size, d]
  __nv_bfloat16* values;
  int heads, kv_heads, log_d, page_size;
  int* error;
  int skip_rank, skip_kb;        // self-test of the give-up path only: the block of each cluster, and its k-block, that is never loaded
};
constexpr uint32_t SELFTEST_WAIT_LIMIT = 1u << 12;

__device__ __forceinline__ void store_remote(uint32_t address, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(address), "f"(v) : "memory");
}
__device__ __forceinline__ void unpack4(const uint2& t, float* v) {
  const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&t.x), b = __bfloat1622float2(*(const __nv_bfloat162*)&t.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ uint2 pack4(const float* v) {
  uint2 t;
  *(__nv_bfloat162*)&t.x = __floats2bfloat162_rn(v[0], v[1]);
  *(__nv_bfloat162*)&t.y = __floats2bfloat162_rn(v[2], v[3]);
  return t;
}

// One epilogue thread's place: rows lo .. lo + 3 and hi .. hi + 3 of the tile, for one token at a time (`threads` = rows / 8
// of them share a token). What is the same for all of its tokens is read before the sums are complete: norm weight or bias.
template <int KIND>
struct Place {
  int lo, hi;                    // rows of the tile
  bool has_lo, has_hi;           // the matrix has them
  int head;                      // QKV
  float4 w_lo, w_hi;             // RESIDUAL: the norm's weight; QKV: the bias
};
// What belongs to a token: residuals, or angles and the place in the page.
struct Side {
  float4 a, b;
  int page, offset;              // page -1: no write
};

template <int KIND>
__device__ __forceinline__ Place<KIND> place_of(const Params& p, int column0, int i) {
  Place<KIND> at;
  at.head = 0;
  if (KIND == QKV) {
    const int log_half = p.log_d - 1, pair = 4 * i, head = pair >> log_half;
    at.lo = (head << p.log_d) + (pair - (head << log_half));
    at.hi = at.lo + (1 << log_half);
    at.head = (column0 >> p.log_d) + head;
  } else if (is_gate(KIND)) {
    at.lo = 32 * (i >> 2) + 4 * (i & 3);
    at.hi = at.lo + 16;
  } else {
    at.lo = 4 * i;
    at.hi = (p.rows >> 1) + 4 * i;
  }
  at.has_lo = column0 + at.lo < p.n;
  at.has_hi = column0 + at.hi < p.n;
  const float* w = KIND == QKV ? p.bias : KIND == RESIDUAL ? p.gamma : nullptr;
  at.w_lo = at.w_hi = make_float4(0.f, 0.f, 0.f, 0.f);
  if (w != nullptr && at.has_lo) at.w_lo = *(const float4*)(w + column0 + at.lo);
  if (w != nullptr && at.has_hi) at.w_hi = *(const float4*)(w + column0 + at.hi);
  return at;
}

template <int KIND>
__device__ __forceinline__ void load_side(const Params& p, int column0, const Place<KIND>& at, int token, Side& side) {
  if (KIND == QKV) {
    side.a = make_float4(1.f, 1.f, 1.f, 1.f);
    side.b = make_float4(0.f, 0.f, 0.f, 0.f);
    side.page = -1;
    const int f = at.lo & ((1 << p.log_d) - 1);
    if (p.rotary != nullptr && at.head < p.heads + p.kv_heads) {
      const float* from = p.rotary + ((size_t)token << p.log_d) + f;
      side.a = *(const float4*)from;
      side.b = *(const float4*)(from + (1 << (p.log_d - 1)));
    }
    if (p.slots != nullptr && at.head >= p.heads && at.has_lo) {
      const int slot = p.slots[token];
      if (slot >= 0 && slot_in_pool(slot, p.page_size)) {
        side.page = slot / p.page_size;
        side.offset = slot - side.page * p.page_size;
      }
    }
  } else if (KIND == RESIDUAL) {
    uint2 lo = make_uint2(0u, 0u), hi = make_uint2(0u, 0u);
    if (p.residual != nullptr) {
      const __nv_bfloat16* from = p.residual + (size_t)token * p.n + column0;
      if (at.has_lo) lo = *(const uint2*)(from + at.lo);
      if (at.has_hi) hi = *(const uint2*)(from + at.hi);
    }
    side.a = make_float4(__uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(hi.x), __uint_as_float(hi.y));
  }
}

// One thread's part of a token, from its 2 x 4 sums on.
template <int KIND>
__device__ __forceinline__ void finish(const Params& p, int tile, int column0, int token, int i, const Place<KIND>& at, float* lo, float* hi,
                                       float scale, const Side& side) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    lo[j] *= scale;
    hi[j] *= scale;
  }
  const float w_lo[4] = {at.w_lo.x, at.w_lo.y, at.w_lo.z, at.w_lo.w}, w_hi[4] = {at.w_hi.x, at.w_hi.y, at.w_hi.z, at.w_hi.w};
  if (KIND == QKV) {
    if (!at.has_lo) return;
    const float cs[4] = {side.a.x, side.a.y, side.a.z, side.a.w}, sn[4] = {side.b.x, side.b.y, side.b.z, side.b.w};
    const bool rotates = p.rotary != nullptr && at.head < p.heads + p.kv_heads;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo[j] = __bfloat162float(__float2bfloat16_rn(lo[j] + w_lo[j]));
      hi[j] = __bfloat162float(__float2bfloat16_rn(hi[j] + w_hi[j]));
      if (rotates) rotate_pair(lo[j], hi[j], cs[j], sn[j]);
    }
    const uint2 packed_lo = pack4(lo), packed_hi = pack4(hi);
    const int half = 1 << (p.log_d - 1), f = at.lo & (2 * half - 1);
    __nv_bfloat16* q = p.out + (size_t)token * p.n + column0 + at.lo;
    *(uint2*)q = packed_lo;
    *(uint2*)(q + half) = packed_hi;
    if (side.page >= 0) {
      const bool is_key = at.head < p.heads + p.kv_heads;
      const int kv_head = is_key ? at.head - p.heads : at.head - p.heads - p.kv_heads;
      __nv_bfloat16* to = (is_key ? p.keys : p.values) + ((((size_t)side.page * p.kv_heads + kv_head) * p.page_size + side.offset) << p.log_d) + f;
      *(uint2*)to = packed_lo;
      *(uint2*)(to + half) = packed_hi;
    }
  } else if (is_gate(KIND)) {
    if (!at.has_lo) return;
    float r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float g = __bfloat162float(__float2bfloat16_rn(lo[j])), u = __bfloat162float(__float2bfloat16_rn(hi[j]));
      r[j] = gated(g, u, gate_of(KIND));
    }
    *(uint2*)(p.out + (size_t)token * (p.n >> 1) + (column0 >> 1) + 4 * i) = pack4(r);
  } else {
    float a[4], b[4];
    unpack4(make_uint2(__float_as_uint(side.a.x), __float_as_uint(side.a.y)), a);
    unpack4(make_uint2(__float_as_uint(side.a.z), __float_as_uint(side.a.w)), b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] += lo[j];
      b[j] += hi[j];
    }
    const uint2 packed_lo = pack4(a), packed_hi = pack4(b);
    const size_t to = (size_t)token * p.n + column0;
    if (at.has_lo) *(uint2*)(p.out + to + at.lo) = packed_lo;
    if (at.has_hi) *(uint2*)(p.out + to + at.hi) = packed_hi;
    if (p.gamma != nullptr) {
      unpack4(packed_lo, a);               // the norm is of the rounded sum
      unpack4(packed_hi, b);
      float squares = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        squares += (at.has_lo ? a[j] * a[j] : 0.f) + (at.has_hi ? b[j] * b[j] : 0.f);
        a[j] *= w_lo[j];
        b[j] *= w_hi[j];
      }
      if (at.has_lo) *(uint2*)(p.scaled + to + at.lo) = pack4(a);
      if (at.has_hi) *(uint2*)(p.scaled + to + at.hi) = pack4(b);
      const int threads = p.rows >> 3;                                  // a token's, neighbours in a warp
      const unsigned group = ((1u << threads) - 1u) << (threadIdx.x & 31 & ~(threads - 1));
      for (int o = threads >> 1; o > 0; o >>= 1) squares += __shfl_xor_sync(group, squares, o);
      if (i == 0) p.squares[(size_t)tile * p.tokens + token] = squares;
    }
  }
}

// Blocks rank 0 .. C - 1 of a cluster (CLUSTER; else C = 1): blockIdx.x = tile * C + rank. SELFTEST: with which a test makes a wait run out, to
// see the give-up path work.
template <int KIND, bool CLUSTER, bool SELFTEST = false>
__global__ void __launch_bounds__(64 + EPILOGUE_THREADS<CLUSTER>, 2) cluster_product_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                     const __grid_constant__ CUtensorMap map_x, const Params p, int cluster) {
  constexpr int EPILOGUE = EPILOGUE_THREADS<CLUSTER>;
  constexpr uint32_t limit = SELFTEST ? SELFTEST_WAIT_LIMIT : WAIT_LIMIT;
  if (!CLUSTER) cluster = 1;
  extern __shared__ uint8_t raw_smem[];
  const uint32_t raw = smem_u32(raw_smem);
  const uint32_t base = (raw + 1023u) & ~1023u;                   // swizzled tiles start on 1024 bytes
  uint8_t* generic_base = raw_smem + (base - raw);
  // tail: full[stages], empty[stages], accumulator; tensor memory's address; abort flag; the scales of this block's tokens
  const int stages = p.stages, a_bytes = p.rows * BK * 2, stage_bytes = a_bytes + p.columns * BK * 2;
  const int ring_bytes = (stages - 1) * stage_bytes + max(stage_bytes, A_BYTES);
  // The sums that this block finishes, [blocks of the cluster][its tokens][rows]: room of its own in a cluster, whose other blocks may
  // be done before this one; else over the drained ring.
  const int per_block = CLUSTER ? (p.tokens + cluster - 1) / cluster : p.tokens;
  const int exchange_bytes = CLUSTER ? cluster * per_block * p.rows * 4 : 0;
  float* exchange = (float*)(generic_base + (CLUSTER ? ring_bytes : 0));
  const uint32_t exchange_at = base + (CLUSTER ? ring_bytes : 0);
  const uint32_t bars = base + ring_bytes + exchange_bytes;
  uint8_t* tail = generic_base + ring_bytes + exchange_bytes;
  volatile uint32_t* tmem_holder = (volatile uint32_t*)(tail + 8 * (2 * MAX_STAGES + 1));
  volatile int* abort_flag = (volatile int*)(tmem_holder + 1);
  float* scales = (float*)(tail + 256);

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
  }
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int tile = CLUSTER ? blockIdx.x / cluster : blockIdx.x, rank = CLUSTER ? blockIdx.x - tile * cluster : 0;
  const int column0 = tile * p.rows;
  const int kb_begin = CLUSTER ? rank * p.k_blocks / cluster : 0;
  const int kb_count = CLUSTER ? (rank + 1) * p.k_blocks / cluster - kb_begin : p.k_blocks;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (stages + s); };
  const uint32_t done_bar = bars + 8u * (2 * stages);
  const uint32_t tmem_columns = p.columns <= 32 ? 32u : p.columns <= 64 ? 64u : 128u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32((const void*)tmem_holder), tmem_columns);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  dependent_launch_trigger();
  tcgen05_fence_after();
  // Another block's shared memory may be written once that block has started: the arrival here, whose wait stands before the first store.
  if (CLUSTER) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;
  const int first = min(kb_count, stages);
  auto skipped = [&](int i) { return SELFTEST && rank == p.skip_rank && i == p.skip_kb; };
  auto load_weights = [&](int i, int s) { tma_load_2d(base + s * stage_bytes, &map_w, full_bar(s), (kb_begin + i) * BK, column0); };
  auto load_tokens = [&](int i, int s) { tma_load_2d(base + s * stage_bytes + a_bytes, &map_x, full_bar(s), (kb_begin + i) * BK, 0); };
  if (warp == 0 && p.early) {
    if (elect_one()) {
      for (int i = 0; i < first; ++i) {
        if (skipped(i)) continue;
        mbar_expect_tx(full_bar(i), stage_bytes);
        load_weights(i, i);
      }
    }
    __syncwarp();
  }
  dependent_launch_wait();

  // This block's share of the tokens, rows / 8 threads each.
  const int token_begin = rank * per_block, tokens = max(0, min(per_block, p.tokens - token_begin));
  const int log_threads = p.rows == 128 ? 4 : 3, items = tokens << log_threads;
  const int thread = threadIdx.x - 64, i_of = thread & ((1 << log_threads) - 1);
  Place<KIND> at;
  Side side;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    const bool leader = elect_one();
    if (leader) {
      for (int i = 0; i < first; ++i) {
        if (skipped(i)) continue;
        if (!p.early) {
          mbar_expect_tx(full_bar(i), stage_bytes);
          load_weights(i, i);
        }
        load_tokens(i, i);
      }
    }
    __syncwarp();
    int issued = first, s = 0;
    uint32_t phase = 0;
    for (int i = first; i < kb_count; ++i) {
      if (!mbar_wait_warp(empty_bar(s), phase, abort_flag, p.error, 1, limit)) break;
      if (leader) {
        mbar_expect_tx(full_bar(s), stage_bytes);
        load_weights(i, s);
        load_tokens(i, s);
      }
      __syncwarp();
      issued = i + 1;
      if (++s == stages) {
        s = 0;
        phase ^= 1u;
      }
    }
    if (leader && *abort_flag) {
      // Loads that were issued still write into this block's shared memory: wait for them.
      for (int i = max(0, issued - stages); i < issued; ++i)
        if (!skipped(i))
        for (uint32_t t = 0; t < WAIT_LIMIT && !mbar_try_wait(full_bar(i % stages), (i / stages) & 1); ++t) __nanosleep(64);
    }
    __syncwarp();
    if (CLUSTER) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    {
      const bool leader = elect_one();
      const uint32_t idesc = instruction_descriptor(BM, p.columns);
      // A stage's descriptors are the first stage's plus an offset in the address field (units of 16 bytes, below 256 KB: no carry).
      const uint64_t w_first = smem_descriptor(base), x_first = smem_descriptor(base + a_bytes);
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < kb_count; ++i) {
        ok = mbar_wait_warp(full_bar(s), phase, abort_flag, p.error, 2, limit);
        if (!ok) break;
        tcgen05_fence_after();
        const uint64_t offset = (uint64_t)(uint32_t)(s * (stage_bytes >> 4)), a = w_first + offset, b = x_first + offset;
        if (leader) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16(tmem_base, a + (uint64_t)(k * UMMA_K * 2 >> 4), b + (uint64_t)(k * UMMA_K * 2 >> 4), idesc, (i > 0 || k > 0) ? 1u : 0u);
          tcgen05_commit(empty_bar(s));
        }
        __syncwarp();
        if (++s == stages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (ok && leader) tcgen05_commit(done_bar);
    }
    __syncwarp();
    if (CLUSTER) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else {
    // ---------------------------------------------------------------- the accumulator into shared memory
    const int quadrant = warp & 3, share = (warp - 2) >> 2;          // of the quadrant's warps
    // What the epilogue reads beside the sums is asked for while they are made.
    at = place_of<KIND>(p, column0, i_of);
    if (thread < items) load_side<KIND>(p, column0, at, token_begin + (thread >> log_threads), side);
    if (thread < tokens) {
      float scale = 1.f;
      if (p.squares_in != nullptr) {
        float total = 0.f;                     // the tiles' sums in their order
#pragma unroll 8
        for (int j = 0; j < p.parts_in; ++j) total += p.squares_in[(size_t)j * p.tokens + token_begin + thread];
        scale = rsqrtf(total / p.width_in + p.eps);
      }
      scales[thread] = scale;
    }
    if (CLUSTER) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    bool ok = mbar_wait(done_bar, 0, abort_flag, p.error, 3);
    ok = __all_sync(0xffffffffu, ok);
    tcgen05_fence_after();
    if (ok && quadrant * 32 < p.rows) {
      const uint32_t lane_address = tmem_base + ((uint32_t)(quadrant * 32) << 16);
      const int row = quadrant * 32 + lane;
#pragma unroll 1
      for (int c0 = share * 16; c0 < p.columns; c0 += EPILOGUE / 8) {
        float v[16];
        tmem_load16(lane_address + c0, v);
        if (CLUSTER) {                          // to the block that finishes the token
          int owner = c0 / per_block, local = c0 - owner * per_block;
          const uint32_t mine = exchange_at + (uint32_t)((rank * per_block * p.rows + row) * 4);
          uint32_t to = in_block(mine, (uint32_t)owner) + (uint32_t)(local * p.rows * 4);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (c0 + i >= p.tokens) break;
            store_remote(to, v[i]);
            to += p.rows * 4;
            if (++local == per_block && c0 + i + 1 < p.tokens) {
              local = 0;
              to = in_block(mine, (uint32_t)++owner);
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c0 + i < p.tokens) exchange[(c0 + i) * p.rows + row] = v[i];
        }
      }
    }
  }
  tcgen05_fence_before();
  if (CLUSTER)
    cluster_sync();
  else
    __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, tmem_columns);
  }
  if (thread >= 0) {
    for (int item = thread; item < items; item += EPILOGUE) {
      const int local = item >> log_threads, token = token_begin + local;
      if (item != thread) load_side<KIND>(p, column0, at, token, side);
      float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
      const float* from = exchange + local * p.rows;
#pragma unroll 4
      for (int r = 0; r < cluster; ++r, from += per_block * p.rows) {                  // the blocks' sums in their order
        const float4 a = *(const float4*)(from + at.lo), b = *(const float4*)(from + at.hi);
        lo[0] += a.x; lo[1] += a.y; lo[2] += a.z; lo[3] += a.w;
        hi[0] += b.x; hi[1] += b.y; hi[2] += b.z; hi[3] += b.w;
      }
      finish<KIND>(p, tile, column0, token, i_of, at, lo, hi, scales[local], side);
    }
  }
}

int sm_count() {
  static int count = [] {
    int device = 0, value = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) value = 0;
    return value > 0 ? value : 148;
  }();
  return count;
}

int columns_of(int tokens) { return (tokens + 15) / 16 * 16; }
int log2_of(int v) { return v <= 1 ? 0 : 1 + log2_of(v >> 1); }

// A launch: weight rows per tile, blocks per tile, ring stages. Measured in the row of a layer's products, us:
// - blocks: as many as two an SM leave room for, 1.7 SMs' worth (clusters of eight do not pack an SM's every place): q|k|v of 3,584, 36
//   tiles, 64 tokens: 91.0 with 6 blocks a tile, 92.3 with 4, 96.6 with 8; down of 1,536, 12 tiles: 36.7 with 8, 39.7 with 5.
// - two blocks an SM (112 KB each) rather than one with a deeper ring, because the next product's blocks start beside them: q|k|v of
//   1,536 with 8 blocks a tile, 40 tokens 34.0 with 4 stages, 38.5 with 9. But where the launch leaves a third of the SMs
//   without a block and a block's K is more than two rings, the deep ring: down of 1,536, 64 tokens 36.7 with 8 stages, 39.9 with 3.
// - and where the tokens leave a block of two an SM no third stage, or no second, one an SM with a deep ring, and as many blocks a tile as let
//   every cluster run at once: a cluster lies within a part of the chip whose SMs it need not divide, so 148 SMs take 45 clusters of three,
//   33 of four, 22 of six, but 15 of seven (`clusters_at_once` asks). A sixteenth cluster of seven ran behind the others: 100 tokens of 1,536, whose
//   q|k|v has 16 tiles, 42.3 with seven blocks a tile and 37.4 with six; 128 tokens of 2,048 53.6 and 41.2, of 768 38.4 and 27.4, of 5,120 129.2 and
//   119.6.
// - gate|up whose tiles fill the SMs by themselves: tiles of 64 rows, while all run at once (280 blocks instead of 140 share the end: 64 tokens
//   36.0 against 36.6, 40 tokens 34.1 against 34.4).
struct Shape {
  int rows, cluster, stages;
};
// What a block of a cluster takes at least: no more than two of them share an SM, and none shares one with a block of the clusters that
// take all of tensor memory (see TENSOR MEMORY in common.cuh).
constexpr size_t LEAST_BYTES = 81 * 1024;
static_assert(LEAST_BYTES + WHOLE_TENSOR_MEMORY_BYTES + 2 * 1024 > 228 * 1024 && 3 * (LEAST_BYTES + 1024) > 228 * 1024, "tensor memory");
size_t smem_bytes(const Shape& s, int tokens) {
  const size_t stage = (size_t)(s.rows + columns_of(tokens)) * BK * 2;
  const size_t exchange = s.cluster > 1 ? (size_t)s.cluster * ((tokens + s.cluster - 1) / s.cluster) * s.rows * 4 : 0;
  const size_t bytes = 1024 + (s.stages - 1) * stage + (stage > (size_t)A_BYTES ? stage : (size_t)A_BYTES) + exchange + TAIL_BYTES;
  return s.cluster == 1 || bytes > LEAST_BYTES ? bytes : LEAST_BYTES;
}
constexpr int SMEM_PER_BLOCK = 112 * 1024;     // two blocks an SM

// Stands for the product's kernel in the question below: asked about a kernel that allocates tensor memory, the runtime counts one block an
// SM whatever the block takes (two of 112 KB share one all the same).
__global__ void __launch_bounds__(64 + EPILOGUE_THREADS<true>, 2) room_kernel() {}

// Clusters of `cluster` blocks that run at one time on the current device, one block to an SM or two.
int clusters_at_once(int cluster, bool one_an_sm) {
  static std::atomic<int> known[64][2][MAX_CLUSTER + 1];
  int device = 0, count = 0;
  if (cudaGetDevice(&device) != cudaSuccess) device = 0;
  const bool kept = device >= 0 && device < 64;
  if (kept && (count = known[device][one_an_sm][cluster].load(std::memory_order_relaxed)) > 0) return count;
  const size_t bytes = one_an_sm ? 227 * 1024 : SMEM_PER_BLOCK;
  static DevicesSet raised;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(cluster);
  config.blockDim = dim3(64 + EPILOGUE_THREADS<true>);
  config.dynamicSmemBytes = bytes;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = cluster;
  attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  if (raise_shared_memory(raised, room_kernel, 227 * 1024, "linear_cluster") != 0 || cudaOccupancyMaxActiveClusters(&count, room_kernel, &config) != cudaSuccess || count < 1) {
    cudaGetLastError();                                   // not known: half of what the SMs' number would allow
    return sm_count() * (one_an_sm ? 1 : 2) / (2 * cluster);
  }
  if (kept) known[device][one_an_sm][cluster].store(count, std::memory_order_relaxed);
  return count;
}

Shape shape_of(int tokens, int n, int k, bool gate) {
  const int k_blocks = (k + BK - 1) / BK, sms = sm_count();
  Shape s{BM, 1, 2};
  const int tiles = (n + BM - 1) / BM;
  // At most `blocks` in all, and all at once.
  auto blocks_a_tile = [&](int blocks, bool one_an_sm) {
    int c = blocks / tiles;
    c = c > MAX_CLUSTER ? MAX_CLUSTER : c < 1 ? 1 : c;
    c = c > k_blocks ? k_blocks : c;
    while (c > 1 && clusters_at_once(c, one_an_sm) < tiles) --c;
    return c;
  };
  auto most_stages = [&](size_t limit) {
    const int per_block = (k_blocks + s.cluster - 1) / s.cluster;
    int stages = 2;
    while (stages < MAX_STAGES && stages < per_block && smem_bytes(Shape{s.rows, s.cluster, stages + 1}, tokens) <= limit) ++stages;
    return stages;
  };
  s.cluster = blocks_a_tile(sms * 17 / 10, false);
  if (gate && s.cluster == 1 && (n + 63) / 64 <= 2 * sms) s.rows = 64;
  s.stages = most_stages(SMEM_PER_BLOCK);
  const int per_block = (k_blocks + s.cluster - 1) / s.cluster;
  if (s.cluster > 1 && tiles * s.cluster * 10 <= sms * 7 && per_block > 2 * s.stages && clusters_at_once(s.cluster, true) >= tiles) {
    s.stages = most_stages(227 * 1024);
  } else if (s.cluster > 1 && ((s.stages < 3 && per_block >= 3) || smem_bytes(s, tokens) > SMEM_PER_BLOCK)) {
    s.cluster = blocks_a_tile(sms, true);
    s.stages = most_stages(227 * 1024);
  }
  return s;
}

template <int KIND>
int launch(Params p, const void* w, const void* x, int k, int rows, int cluster, int stages, cudaStream_t stream) {
  Shape s = shape_of(p.tokens, p.n, k, is_gate(KIND));
  if (rows != 0) s = Shape{rows, cluster, stages};
  p.k_blocks = (k + BK - 1) / BK;
  p.columns = columns_of(p.tokens);
  p.rows = s.rows;
  p.stages = s.stages;
  const size_t bytes = smem_bytes(s, p.tokens);
  if ((s.rows != 64 && s.rows != 128) || s.cluster < 1 || s.cluster > MAX_CLUSTER || s.cluster > p.k_blocks || s.stages < 2 || s.stages > MAX_STAGES ||
      bytes > 227 * 1024 || (KIND == QKV && s.rows < (1 << p.log_d)) || (size_t)p.tokens * s.rows * 4 > (size_t)s.stages * (s.rows + p.columns) * BK * 2)
    return fail(2, "linear_cluster: no launch of tiles of %d rows, %d blocks a tile, %d stages", s.rows, s.cluster, s.stages);
  CUtensorMap map_w, map_x;
  if (int err = tensor_map(&map_w, w, p.n, k, s.rows)) return err;
  if (int err = tensor_map(&map_x, x, p.tokens, k, p.columns)) return err;
  const int tiles = (p.n + s.rows - 1) / s.rows;
  if (s.cluster > 1) {
    static DevicesSet raised;
    if (int err = raise_shared_memory(raised, cluster_product_kernel<KIND, true>, 227 * 1024, "linear_cluster")) return err;
    launch_kernel_cluster(cluster_product_kernel<KIND, true>, dim3(tiles * s.cluster), dim3(64 + EPILOGUE_THREADS<true>), bytes, stream, (unsigned)s.cluster, map_w, map_x, p,
                          s.cluster);
  } else {
    static DevicesSet raised;
    if (int err = raise_shared_memory(raised, cluster_product_kernel<KIND, false>, 227 * 1024, "linear_cluster")) return err;
    launch_kernel(cluster_product_kernel<KIND, false>, dim3(tiles), dim3(64 + EPILOGUE_THREADS<false>), bytes, stream, map_w, map_x, p, 1);
  }
  return check_launch("linear_cluster");
}

int check_common(const char* what, const void* out, const void* w, const void* x, const float* squares_in, int parts_in, const int* error,
                 int tokens, int n, int k) {
  if (tokens < 1 || tokens > MAX_TOKENS) return fail(2, "%s: %d tokens (1 to %d)", what, tokens, MAX_TOKENS);
  if (k < 1 || k % 8) return fail(2, "%s: K = %d is not a multiple of 8 (a TMA row pitch must be a multiple of 16 bytes)", what, k);
  if (n < 8 || n % 8) return fail(2, "%s: %d rows are not a multiple of 8", what, n);
  if (((uintptr_t)out | (uintptr_t)w | (uintptr_t)x) & 15) return fail(2, "%s: an operand does not start on a 16-byte boundary", what);
  if (squares_in != nullptr && parts_in < 1) return fail(2, "%s: %d parts of the squares", what, parts_in);
  if (error == nullptr) return fail(2, "%s: no error word", what);
  return 0;
}

}  // namespace

// Rows of `squares` that a product of n columns leaves.
PAE_EXPORT int pae_linear_cluster_parts(int tokens, int n, int k) {
  const int rows = shape_of(tokens, n, k, false).rows;
  return (n + rows - 1) / rows;
}

// Rounds of clusters that a launch takes: 0 without clusters, else 1 unless its shape is wrong.
PAE_EXPORT int pae_linear_cluster_rounds(int tokens, int n, int k, int gate) {
  const Shape s = shape_of(tokens, n, k, gate != 0);
  if (s.cluster == 1) return 0;
  const int at_once = clusters_at_once(s.cluster, smem_bytes(s, tokens) > SMEM_PER_BLOCK);
  return ((n + s.rows - 1) / s.rows + at_once - 1) / at_once;
}

// out[token, n] = x . w[n, k]^T (+ residual[token, n]), bfloat16. With `gamma` also scaled[token, n] = out * gamma and
// squares[part, token] (parts as above), the sums of the squares of 128 columns of out each: what the next product needs to
// stand for RMSNorm(out) * gamma. `squares_in` [parts_in, tokens]: x is such a `scaled`, of rows of `width_in`, and the product is
// multiplied by rsqrt(sum / width_in + eps). early: w may be read while the kernel before is still running. cluster, stages: 0, or
// the blocks per tile and the ring's stages (measurements).
PAE_EXPORT int pae_linear_cluster(void* out, const void* x, const void* w, const void* residual, const float* gamma, void* scaled, float* squares,
                                  const float* squares_in, int parts_in, int width_in, float eps, int tokens, int n, int k, int early, int rows,
                                  int cluster, int stages, int* error, void* stream) {
  if (int err = check_common("linear_cluster", out, w, x, squares_in, parts_in, error, tokens, n, k)) return err;
  if (((uintptr_t)residual | (uintptr_t)gamma | (uintptr_t)scaled) & 15) return fail(2, "linear_cluster: an operand does not start on a 16-byte boundary");
  if (gamma != nullptr && (scaled == nullptr || squares == nullptr)) return fail(2, "linear_cluster: a norm's weight without its outputs");
  Params p{};
  p.tokens = tokens;
  p.n = n;
  p.early = early;
  p.squares_in = squares_in;
  p.parts_in = parts_in;
  p.width_in = (float)width_in;
  p.eps = eps;
  p.residual = (const __nv_bfloat16*)residual;
  p.out = (__nv_bfloat16*)out;
  p.gamma = gamma;
  p.scaled = (__nv_bfloat16*)scaled;
  p.squares = squares;
  p.error = error;
  return launch<RESIDUAL>(p, w, x, k, rows, cluster, stages, (cudaStream_t)stream);
}

// out[token, n / 2] = act(g) * u with g, u the products of the gate and up rows of w [n, k] (alternating in blocks of 16), each rounded to
// bfloat16 first. The rest as above.
PAE_EXPORT int pae_linear_swiglu_cluster(void* out, const void* x, const void* w, const float* squares_in, int parts_in, int width_in, float eps,
                                         int tokens, int n, int k, int gate_kind, int early, int rows, int cluster, int stages, int* error, void* stream) {
  if (int err = check_common("linear_swiglu_cluster", out, w, x, squares_in, parts_in, error, tokens, n, k)) return err;
  if (n % 32) return fail(2, "linear_swiglu_cluster: %d rows are not blocks of 16 gate and 16 up rows", n);
  Params p{};
  p.tokens = tokens;
  p.n = n;
  p.early = early;
  p.squares_in = squares_in;
  p.parts_in = parts_in;
  p.width_in = (float)width_in;
  p.eps = eps;
  p.out = (__nv_bfloat16*)out;
  p.error = error;
  cudaStream_t s = (cudaStream_t)stream;
  if (gate_kind == kGateRelu) return launch<GATE_RELU>(p, w, x, k, rows, cluster, stages, s);
  if (gate_kind == kGateGeluTanh) return launch<GATE_GELU>(p, w, x, k, rows, cluster, stages, s);
  return launch<GATE_SILU>(p, w, x, k, rows, cluster, stages, s);
}

// Self-test of the give-up path: a product of `cluster` blocks a tile in which block `skip_rank` of every cluster never loads its k-block `skip_kb` (one of
// its first `stages`; nothing is in flight for it). Its wait for the stage runs out after a few thousand polls, the other blocks go on, and all leave.
PAE_EXPORT int pae_linear_cluster_selftest_giveup(void* out, const void* x, const void* w, int tokens, int n, int k, int cluster, int stages, int skip_rank,
                                                  int skip_kb, int* error, void* stream) {
  if (int err = check_common("linear_cluster_selftest_giveup", out, w, x, nullptr, 0, error, tokens, n, k)) return err;
  Params p{};
  p.tokens = tokens;
  p.n = n;
  p.k_blocks = (k + BK - 1) / BK;
  p.columns = columns_of(tokens);
  p.rows = BM;
  p.stages = stages;
  p.early = 1;
  p.out = (__nv_bfloat16*)out;
  p.error = error;
  p.skip_rank = skip_rank;
  p.skip_kb = skip_kb;
  const Shape s{BM, cluster, stages};
  const int tiles = (n + BM - 1) / BM;
  if (cluster < 2 || cluster > MAX_CLUSTER || cluster > p.k_blocks || stages < 2 || stages > MAX_STAGES || smem_bytes(s, tokens) > 227 * 1024 || skip_rank < 0 ||
      skip_rank >= cluster || skip_kb < 0 || skip_kb >= stages || skip_kb >= p.k_blocks / cluster)
    return fail(2, "linear_cluster_selftest_giveup: block %d of %d, k-block %d of %d stages", skip_rank, cluster, skip_kb, stages);
  CUtensorMap map_w, map_x;
  if (int err = tensor_map(&map_w, w, n, k, BM)) return err;
  if (int err = tensor_map(&map_x, x, tokens, k, p.columns)) return err;
  static DevicesSet raised;
  if (int err = raise_shared_memory(raised, cluster_product_kernel<RESIDUAL, true, true>, 227 * 1024, "linear_cluster_selftest_giveup")) return err;
  launch_kernel_cluster(cluster_product_kernel<RESIDUAL, true, true>, dim3(tiles * cluster), dim3(64 + EPILOGUE_THREADS<true>), smem_bytes(s, tokens), (cudaStream_t)stream,
                        (unsigned)cluster, map_w, map_x, p, cluster);
  return check_launch("linear_cluster_selftest_giveup");
}

// 1 for head sizes of which a tile of 128 rows holds whole heads.
PAE_EXPORT int pae_qkv_cluster_supports(int d) { return d >= 16 && d <= BM && (d & (d - 1)) == 0; }

// qkv[token, (heads + 2 kv_heads) d] = x . w^T + bias, q and k rotated by `rotary` [tokens, d] (cosines, then sines; or
// null), k and v also written to their pages at `slots`. The rest as above.
PAE_EXPORT int pae_qkv_cluster(void* qkv, const void* x, const void* w, const float* bias, const float* squares_in, int parts_in, int width_in,
                               float eps, const float* rotary, const int* slots, void* keys, void* values, int tokens, int heads, int kv_heads,
                               int d, int page_size, int k, int early, int rows, int cluster, int stages, int* error, void* stream) {
  const int n = (heads + 2 * kv_heads) * d;
  if (int err = check_common("qkv_cluster", qkv, w, x, squares_in, parts_in, error, tokens, n, k)) return err;
  if (!pae_qkv_cluster_supports(d)) return fail(2, "qkv_cluster: a tile of 128 rows does not hold whole heads of %d", d);
  if (slots != nullptr && (keys == nullptr || values == nullptr || page_size < 1)) return fail(2, "qkv_cluster: slots without pages");
  if (((uintptr_t)rotary | (uintptr_t)keys | (uintptr_t)values) & 15) return fail(2, "qkv_cluster: an operand does not start on a 16-byte boundary");
  Params p{};
  p.tokens = tokens;
  p.n = n;
  p.early = early;
  p.squares_in = squares_in;
  p.parts_in = parts_in;
  p.width_in = (float)width_in;
  p.eps = eps;
  p.out = (__nv_bfloat16*)qkv;
  p.bias = bias;
  p.rotary = rotary;
  p.slots = slots;
  p.keys = (__nv_bfloat16*)keys;
  p.values = (__nv_bfloat16*)values;
  p.heads = heads;
  p.kv_heads = kv_heads;
  p.log_d = log2_of(d);
  p.page_size = page_size;
  p.error = error;
  return launch<QKV>(p, w, x, k, rows, cluster, stages, (cudaStream_t)stream);
}

PAE_DEFINE_LAST_ERROR()
