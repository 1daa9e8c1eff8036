// Attention of prompt portions over the paged cache on the fifth-generation tensor cores:
// both products of attention are tcgen05.mma with accumulators in tensor memory, keys and
// values come page by page through TMA, and the softmax runs in plain threads beside them.
//
// A block owns 128 consecutive query tokens of one request and one query head, and walks
// that request's keys 128 at a time:
//
//   warp 0      TMA: the query tile once; per key tile the pages of K and of V (one box of
//               page_size rows x 64 columns per page and half of the head dimension), two
//               stages deep. Pages are found through the block table; nothing is gathered.
//   warp 1      MMA: S = Q . K^T into one of two score buffers in tensor memory (so the
//               scores of the next tile are computed while the softmax works on this one),
//               then O_tile = P . V, into one of two product buffers, once the probabilities
//               are in one of two buffers in shared memory. V is used as it lies in the
//               cache (head dimension contiguous): an MN-major operand.
//   warps 2-9   softmax: two threads share query row r (half of a tile's keys and half of
//               the output's dimensions each). A thread reads its scores from tensor memory
//               twice (maximum; then exponentials, sum and the bfloat16 probabilities
//               written to shared memory in the operand's swizzled layout). The product of
//               a tile is folded into the running output in registers one tile late,
//               out = out * 2^(old max - new max) + O_tile, so the tensor core computes it
//               while the threads take the next tile's exponentials. No shuffles.
//
// The rule of the reference (engine/attention.py:581-586) is evaluated per score on tiles
// that touch the diagonal, a window's edge or the request's end; tiles that lie wholly
// inside need no mask. Scores are scaled in float32; probabilities are rounded to bfloat16
// for the second product. Every mbarrier wait is bounded and reports through `error`.
//
// When a launch has few blocks (a short portion of a prompt over a long context), a query
// tile's keys are shared out over a thread-block cluster: every block of the cluster takes a
// run of key tiles, the blocks behind the first leave their rows' maxima, sums and outputs in
// their own shared memory, and the first merges them through distributed shared memory
// between two barriers of the cluster.
//
// Sizes: head_dim 64 or 128; page sizes 16, 32, 64 or 128; any number of heads and groups.
// Requests that bring a single token are left to the decode kernel.

#include <cfloat>
#include <mutex>
#include <unordered_map>

#include "tcgen05.cuh"

using namespace pae;
using namespace pae_tcgen05;

namespace {

constexpr int BQ = 128;             // query rows per block
constexpr int BKEYS = 128;          // keys per tile
constexpr int THREADS = 320;         // TMA warp, MMA warp, eight softmax warps (two threads per query row)
constexpr int SOFTMAX_THREADS = 256;
constexpr float LOG2E = 1.4426950408889634f;

struct Params {
  __nv_bfloat16* out;               // [tokens, heads, D]
  const int* block_table;
  const int* q_start;
  const int* q_pos0;
  const int* kv_len;
  int table_width, heads, kv_heads, page_size, window, skip_single;
  const int* work_index;  // the requests that this launch works on, one per grid z (null: request z)
  float scale_log2;
  float slack;            // paired form: a row's reference may lie below its maximum by 2^slack (0: it follows every maximum)
  int* error;
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A box of keys or values: coordinates in a pool seen as [pages][kv heads][D / 64][rows of a page][64].
__device__ __forceinline__ void tma_load_pages(uint32_t dst, const CUtensorMap* map, uint32_t bar, int row, int half, int head, int page) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(half), "r"(head), "r"(page)
      : "memory");
}
// How keys and values come into shared memory. What the TMA unit takes is time per box, not bytes: with a box a page and half of
// a row, 16 boxes of 2 KB for 64 keys of a page size of 16, it set the pace of the paired kernel (8,192 tokens, 12 heads of 128: 235 us against
// 177 with pages of 64; now 173 with either, 1,190 TFLOP/s, and a tenth more where no two pages follow one another). So the pages of a tile that follow one another in the pool, as a prompt's pages mostly do, come as ONE box per half
// of the keys and one of the values; others come a box each (and half, of the keys). The values lie [page][half][row][64] (the
// halves' distance is the descriptor's leading byte offset), the keys [half][page][row][64].
struct PageMaps {
  CUtensorMap key, value;                // a page (or the rows of it that a tile covers)
  CUtensorMap key_run, value_run;        // the pages of a tile
};
// Tile of `rows` keys, `rows_a_box` of them a box, by a converged warp: lane i brings the box at `row` of `page`, or lane 0 all of them.
template <int D>
__device__ __forceinline__ void load_pages(const PageMaps& maps, bool values, uint32_t dst, uint32_t full, int rows, int rows_a_box, int lane, int head,
                                           int page, int row) {
  constexpr int HALVES = D / 64;
  const int boxes = rows / rows_a_box;
  const int first = __shfl_sync(0xffffffffu, page, 0);
  if (boxes > 1 && __all_sync(0xffffffffu, lane >= boxes || page == first + lane)) {
    if (lane == 0) {
      if (values) {
        tma_load_pages(dst, &maps.value_run, full, 0, 0, head, page);
      } else {
#pragma unroll
        for (int half = 0; half < HALVES; ++half) tma_load_pages(dst + half * rows * 128, &maps.key_run, full, 0, half, head, page);
      }
    }
  } else if (lane < boxes) {
    if (values) {
      tma_load_pages(dst + lane * rows_a_box * 128 * HALVES, &maps.value, full, row, 0, head, page);
    } else {
#pragma unroll
      for (int half = 0; half < HALVES; ++half) tma_load_pages(dst + half * rows * 128 + lane * rows_a_box * 128, &maps.key, full, row, half, head, page);
    }
  }
}
// Where the 16 keys of step k of the second product lie among a tile's values (a box has 16, 32, 64 or 128 rows).
template <int D>
__device__ __forceinline__ uint32_t value_step(int k, int rows_a_box) {
  const int row = k * 16;
  return (uint32_t)(row + (D / 64 - 1) * (row & -rows_a_box)) * 128;
}
// 32 consecutive float32 columns of this thread's lane of tensor memory.
__device__ __forceinline__ void tmem_load32(uint32_t address, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(address)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// The cluster's barrier (every thread of every block of the cluster arrives and waits), this
// block's place in its cluster, and a float read from the shared memory of another block of it.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}
__device__ __forceinline__ float load_from_block(uint32_t address, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(address), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// MN-major operand with 128-byte swizzle: a 128-byte row holds 64 consecutive MN elements of
// one K index; 8 consecutive K indices are 8 rows (1024 bytes, the stride byte offset); the
// next 64 MN elements lie `mn_group_bytes` further (the leading byte offset).
__device__ __forceinline__ uint64_t mn_major_descriptor(uint32_t address, uint32_t mn_group_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((address & 0x3FFFFu) >> 4);
  d |= (uint64_t)((mn_group_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// The descriptor of the place `bytes` (a multiple of 16) further: shared memory ends below 256 KB, so nothing carries out of the address
// field.
__device__ __forceinline__ uint64_t further(uint64_t descriptor, uint32_t bytes) {
  return (descriptor & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)descriptor + (bytes >> 4));
}
// float32 accumulator, bfloat16 operands, A K-major; B K-major or MN-major (bit 16).
__host__ __device__ constexpr uint32_t instruction_descriptor(int m, int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

template <int D>
struct Layout {
  static constexpr int HALVES = D / 64;                    // 64-column k-blocks of the head dimension
  static constexpr int HALF_TILE_BYTES = 128 * 64 * 2;     // 128 rows x 64 bfloat16 = 16 KB
  static constexpr int Q_BYTES = HALVES * HALF_TILE_BYTES;
  static constexpr int KV_BYTES = HALVES * HALF_TILE_BYTES;   // one stage of K, or of V
  static constexpr int P_BYTES = 2 * HALF_TILE_BYTES;         // 128 rows x 128 keys, one of two buffers
  static constexpr int Q_OFFSET = 0;
  static constexpr int K_OFFSET = Q_BYTES;                    // two stages
  static constexpr int V_OFFSET = K_OFFSET + 2 * KV_BYTES;
  static constexpr int P_OFFSET = V_OFFSET + 2 * KV_BYTES;
  static constexpr int BAR_OFFSET = P_OFFSET + 2 * P_BYTES;
  static constexpr int EXCHANGE_OFFSET = BAR_OFFSET + 256;    // [2][128] floats that the two threads of a row swap
  static constexpr size_t SMEM_BYTES = (size_t)EXCHANGE_OFFSET + 1024 /* exchange */ + 1024 /* alignment */;
  static constexpr int S_COLUMNS = 128;                       // per score buffer
  static constexpr int O_COLUMN = 2 * S_COLUMNS;              // two tiles' products behind the two score buffers
  static constexpr int TMEM_COLUMNS = 512;
  static_assert(O_COLUMN + 2 * D <= TMEM_COLUMNS, "two score buffers and two products must fit tensor memory");
  static_assert(SMEM_BYTES <= 227 * 1024, "the block's shared memory");
  static_assert(SMEM_BYTES >= pae::WHOLE_TENSOR_MEMORY_BYTES, "no block of another cluster with tensor memory beside this one (common.cuh)");
};

enum Bar : int { Q_FULL = 0, K_FULL = 1, V_FULL = 3, K_EMPTY = 5, V_EMPTY = 7, S_FULL = 9, S_EMPTY = 11, P_READY = 13, O_FULL = 15, O_EMPTY = 17, X_READY = 19, NUM_BARS = 20 };

template <int D, bool SPLIT>
__global__ void __launch_bounds__(THREADS) prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                  const __grid_constant__ PageMaps maps, const Params p) {
  using L = Layout<D>;
  if (threadIdx.x == 0) {         // the descriptors do not depend on the kernel before: fetch them early
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.key_run) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.value_run) : "memory");
  }
  extern __shared__ uint8_t raw_smem[];
  const uint32_t raw = smem_u32(raw_smem);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* generic_base = raw_smem + (base - raw);
  const uint32_t bars = base + L::BAR_OFFSET;
  volatile uint32_t* tmem_holder = (volatile uint32_t*)(generic_base + L::BAR_OFFSET + 8 * NUM_BARS);
  volatile int* abort_flag = (volatile int*)(tmem_holder + 1);
  auto bar = [&](int which, int i = 0) { return bars + 8u * (which + i); };
  const int warp = uniform_warp(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(bar(Q_FULL), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(K_FULL, i), 1);
      mbar_init(bar(V_FULL, i), 1);
      mbar_init(bar(K_EMPTY, i), 1);
      mbar_init(bar(V_EMPTY, i), 1);
      mbar_init(bar(S_FULL, i), 1);
      mbar_init(bar(S_EMPTY, i), SOFTMAX_THREADS);
      mbar_init(bar(P_READY, i), SOFTMAX_THREADS);
      mbar_init(bar(O_FULL, i), 1);
      mbar_init(bar(O_EMPTY, i), SOFTMAX_THREADS);
    }
    mbar_init(bar(X_READY), SOFTMAX_THREADS);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32((const void*)tmem_holder), L::TMEM_COLUMNS);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  dependent_launch_trigger();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  // ---- what this block works on (the same in every role) -------------------------------
  // The step's integers (starts, positions, lengths, block tables) were on the device before
  // the step's first kernel began: they are read before the wait for the kernel before this
  // one, whose output (q, and this step's keys and values) is not touched until after it.
  // A cluster of `ranks` blocks shares one query tile of one head: each takes a run of its key
  // tiles, and the first block folds the others' outputs into its own at the end.
  const int ranks = SPLIT ? (int)cluster_size() : 1, rank = SPLIT ? (int)cluster_rank() : 0;
  const int h = blockIdx.x / ranks, b = p.work_index != nullptr ? p.work_index[blockIdx.z] : (int)blockIdx.z;
  const int first_token = p.q_start[b];
  const int q_count = p.q_start[b + 1] - first_token;
  const int q_tiles = (q_count + BQ - 1) / BQ;
  // Late tiles see the most keys: they go first in every head (the head is the fastest grid
  // index, so the first wave holds the longest blocks of all heads), the short early ones
  // fill in behind them.
  const int tile = q_tiles - 1 - (int)blockIdx.y;
  const bool active = tile >= 0 && !(p.skip_single && q_count == 1);
  const int rows = active ? min(BQ, q_count - tile * BQ) : 0;
  const int pos0 = p.q_pos0[b] + tile * BQ;
  const int kv_end = active ? min(p.kv_len[b], pos0 + rows) : 0;
  const int first_key = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
  const int all_tiles = active ? (kv_end - (first_key / p.page_size) * p.page_size + BKEYS - 1) / BKEYS : 0;
  const int tiles_per_rank = (all_tiles + ranks - 1) / ranks;
  const int first_tile = min(rank * tiles_per_rank, all_tiles);
  const int n_tiles = min(tiles_per_rank, all_tiles - first_tile);          // this block's
  const int kv_begin = (first_key / p.page_size) * p.page_size + first_tile * BKEYS;
  const bool working = n_tiles > 0;
  const int g = h / (p.heads / p.kv_heads);

  // What the softmax threads carry out of their loop (the other warps leave it alone).
  constexpr int HALF_D = D / 2;
  const int quadrant = warp & 3;
  const int side = warp >= 2 ? (warp - 2) >> 2 : 0;         // which half of the keys and of the dimensions
  const int r = quadrant * 32 + lane;                       // row of the tile, lane of tensor memory
  float acc[HALF_D];
  float row_max = -FLT_MAX, row_sum = 0.f;
  bool ok = true;
  // The producer's lane i brings page i of a tile: the first tile's table entries, before the wait.
  const int last_page = working ? (kv_end - 1) / p.page_size : 0;    // the last page that holds a visible key
  int first_page = 0;
  if (warp == 0 && working && lane < BKEYS / p.page_size)
    first_page = checked_page(p.block_table[(size_t)b * p.table_width + checked_table_index(min(kv_begin / p.page_size + lane, last_page), p.table_width)]);
  dependent_launch_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // Lane i brings page i of a tile (its block-table entry and its boxes), so the table
    // look-ups of a tile are one round trip, not one per page. Lane 0 posts the byte counts
    // before any lane issues a copy.
    if (working) {
      if (lane == 0) {
        mbar_expect_tx(bar(Q_FULL), L::Q_BYTES);
#pragma unroll
        for (int half = 0; half < L::HALVES; ++half)
          tma_load_2d(base + L::Q_OFFSET + half * L::HALF_TILE_BYTES, &map_q, bar(Q_FULL), h * D + half * 64,
                      first_token + tile * BQ);
      }
      const int* table = p.block_table + (size_t)b * p.table_width;
      const bool mine = lane < BKEYS / p.page_size;
      // A page past the last visible key may not exist: its rows are masked, so any page of
      // the request will do; the last visible one is taken.
      auto page_of = [&](int t) {
        return mine && t < n_tiles ? checked_page(table[checked_table_index(min((kv_begin + t * BKEYS) / p.page_size + lane, last_page), p.table_width)]) : 0;
      };
      // Two tiles of K ahead of V, whose stage is free later: the scores of tile t free the stage of K for tile t + 2 while the softmax of
      // tile t - 2 or t - 1 runs, and V of tile t follows the product of tile t - 2.
      auto load = [&](bool values, int t, int page) {
        const int st = t & 1;
        const uint32_t full = bar(values ? V_FULL : K_FULL, st);
        if (t >= 2 && !mbar_wait_warp(bar(values ? V_EMPTY : K_EMPTY, st), ((t >> 1) - 1) & 1, abort_flag, p.error, values ? 10 : 1)) return false;
        if (lane == 0) mbar_expect_tx(full, L::KV_BYTES);
        __syncwarp();
        load_pages<D>(maps, values, base + (values ? L::V_OFFSET : L::K_OFFSET) + st * L::KV_BYTES, full, BKEYS, p.page_size, lane, g, page, 0);
        return true;
      };
      int page0 = first_page;
      bool ok = true;
      int keys_issued = 0, values_issued = 0;
      if (n_tiles > 0) {
        ok = load(false, 0, page0);
        keys_issued = 1;
      }
      int page1 = page_of(1), page2 = page_of(2);               // of tiles t, t + 1, t + 2
      if (n_tiles > 1 && ok) {
        ok = load(false, 1, page1);
        keys_issued = 2;
      }
      for (int t = 0; t < n_tiles && ok; ++t) {
        const int page3 = page_of(t + 3);
        if (t == 0) {                                           // nothing has to be waited for: V before K of a later tile
          load(true, 0, page0);
          values_issued = 1;
        }
        if (t + 2 < n_tiles) {
          if (!(ok = load(false, t + 2, page2))) break;
          keys_issued = t + 3;
        }
        if (t > 0) {
          if (!(ok = load(true, t, page0))) break;
          values_issued = t + 1;
        }
        page0 = page1;
        page1 = page2;
        page2 = page3;
      }
      if (lane == 0 && *abort_flag) {
        for (int t = max(0, keys_issued - 2); t < keys_issued; ++t)
          for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(bar(K_FULL, t & 1), (t >> 1) & 1); ++w) __nanosleep(64);
        for (int t = max(0, values_issued - 2); t < values_issued; ++t)
          for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(bar(V_FULL, t & 1), (t >> 1) & 1); ++w) __nanosleep(64);
        for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(bar(Q_FULL), 0); ++w) __nanosleep(64);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (working) {
      const bool leader = elect_one();
      constexpr uint32_t idesc_s = instruction_descriptor(BQ, BKEYS, false);
      constexpr uint32_t idesc_o = instruction_descriptor(BQ, D, true);
      const uint64_t q_first = smem_descriptor(base + L::Q_OFFSET), k_first = smem_descriptor(base + L::K_OFFSET);
      const uint64_t p_first = smem_descriptor(base + L::P_OFFSET), v_first = mn_major_descriptor(base + L::V_OFFSET, p.page_size * 128);
      bool ok = mbar_wait_warp(bar(Q_FULL), 0, abort_flag, p.error, 2);
      auto issue_scores = [&](int t) {
        const int st = t & 1;
        ok = ok && mbar_wait_warp(bar(K_FULL, st), (t >> 1) & 1, abort_flag, p.error, 3);
        if (t >= 2) ok = ok && mbar_wait_warp(bar(S_EMPTY, st), ((t >> 1) - 1) & 1, abort_flag, p.error, 4);
        if (!ok) return;
        tcgen05_fence_after();
        const uint64_t keys = further(k_first, st * L::KV_BYTES);
        if (leader) {
#pragma unroll
          for (int half = 0; half < L::HALVES; ++half)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_bf16(tmem_base + st * L::S_COLUMNS, further(q_first, half * L::HALF_TILE_BYTES + k * 32),
                        further(keys, half * L::HALF_TILE_BYTES + k * 32), idesc_s, (half > 0 || k > 0) ? 1u : 0u);
          tcgen05_commit(bar(S_FULL, st));
          tcgen05_commit(bar(K_EMPTY, st));       // the K stage is free once these MMAs have read it
        }
        __syncwarp();
      };
      if (n_tiles > 0) issue_scores(0);
      for (int t = 0; t < n_tiles && ok; ++t) {
        if (t + 1 < n_tiles) issue_scores(t + 1);
        const int st = t & 1;
        ok = ok && mbar_wait_warp(bar(V_FULL, st), (t >> 1) & 1, abort_flag, p.error, 5);
        ok = ok && mbar_wait_warp(bar(P_READY, st), (t >> 1) & 1, abort_flag, p.error, 6);
        if (t >= 2) ok = ok && mbar_wait_warp(bar(O_EMPTY, st), ((t >> 1) - 1) & 1, abort_flag, p.error, 7);
        if (!ok) break;
        tcgen05_fence_after();
        const uint64_t probabilities = further(p_first, st * L::P_BYTES), values = further(v_first, st * L::KV_BYTES);
        if (leader) {
#pragma unroll
        for (int k = 0; k < BKEYS / 16; ++k)     // 16 keys a step: two groups of 8 rows of V
          umma_bf16(tmem_base + L::O_COLUMN + st * D, further(probabilities, (k >> 2) * L::HALF_TILE_BYTES + (k & 3) * 32), further(values, value_step<D>(k, p.page_size)),
                    idesc_o, k > 0 ? 1u : 0u);
        tcgen05_commit(bar(O_FULL, st));
        tcgen05_commit(bar(V_EMPTY, st));
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, two threads per row
    // The two warps that may read a quarter of tensor memory's lanes (warp id modulo 4) share
    // its 32 rows: one takes keys 0-63 of a tile and the first half of the output's
    // dimensions, the other keys 64-127 and the second half. They swap their maxima through
    // shared memory once per tile and their sums once at the end.
    //
    // P and a tile's product P.V have two buffers each, and a tile's product is added to the
    // output one tile late: after the probabilities of tile t are handed over, the threads add
    // the product of tile t-1, which the tensor core finished while they were taking
    // exponentials. So the product of one tile runs under the softmax of the next, and the
    // threads wait for neither.
    const uint32_t lane_base = tmem_base + ((uint32_t)(quadrant * 32) << 16);
    const int my_pos = pos0 + r;
    float* exchange = (float*)(generic_base + L::EXCHANGE_OFFSET);
    constexpr int HALF_KEYS = BKEYS / 2;
#pragma unroll
    for (int i = 0; i < HALF_D; ++i) acc[i] = 0.f;
    // acc = acc * scale + the product of tile u (scale: what tile u's maximum did to the reference).
    auto add_product = [&](int u, float scale) {
      const int su = u & 1;
      ok = ok && mbar_wait(bar(O_FULL, su), (u >> 1) & 1, abort_flag, p.error, 9);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tcgen05_fence_after();
#pragma unroll
      for (int c = 0; c < HALF_D; c += 32) {
        float o[32];
        tmem_load32(lane_base + L::O_COLUMN + su * D + side * HALF_D + c, o);
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c + i] = acc[c + i] * scale + o[i];
      }
      tcgen05_fence_before();
      mbar_arrive(bar(O_EMPTY, su));
    };
    float owed_scale = 0.f;       // goes with the product that is not added yet
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t & 1;
      const int key0 = kv_begin + t * BKEYS;
      ok = ok && mbar_wait(bar(S_FULL, st), (t >> 1) & 1, abort_flag, p.error, 8);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      // The whole tile is visible to every row of the block: no mask. Otherwise a row sees the
      // keys lo..hi of the request (nothing when the row is past the request's tokens).
      const bool unmasked = key0 + BKEYS - 1 <= pos0 && key0 + BKEYS <= kv_end && key0 >= first_key &&
                            (p.window <= 0 || pos0 + rows - 1 - key0 < p.window);
      const int hi = r < rows ? min(my_pos, kv_end - 1) - key0 : -1;          // relative to the tile
      const int lo = (p.window > 0 ? max(first_key, my_pos - p.window + 1) : first_key) - key0;
      float m4[4] = {-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
      for (int c = side * HALF_KEYS; c < side * HALF_KEYS + HALF_KEYS; c += 32) {
        float s[32];
        tmem_load32(lane_base + st * L::S_COLUMNS + c, s);
        if (unmasked) {
#pragma unroll
          for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], s[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int key = c + i;
            m4[i & 3] = fmaxf(m4[i & 3], (key >= lo && key <= hi) ? s[i] : -FLT_MAX);
          }
        }
      }
      float tile_max = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      exchange[side * 128 + r] = tile_max;
      mbar_arrive(bar(X_READY));                                // all softmax threads have written theirs
      ok = mbar_wait(bar(X_READY), t & 1, abort_flag, p.error, 11);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tile_max = fmaxf(tile_max, exchange[(side ^ 1) * 128 + r]);
      if (tile_max != -FLT_MAX) tile_max *= p.scale_log2;        // the scale is positive: max(s) scales with it
      const float new_max = fmaxf(row_max, tile_max);
      const float rescale = row_max == -FLT_MAX ? 0.f : fast_exp2(row_max - new_max);
      row_max = new_max;
      // exp2(s * scale - max) as one fused multiply-add and one ex2; a row that has seen no key
      // yet keeps max = -FLT_MAX and every probability 0.
      const float offset = new_max == -FLT_MAX ? 0.f : -new_max;
      const float factor = new_max == -FLT_MAX ? 0.f : p.scale_log2;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
      uint8_t* p_row = generic_base + L::P_OFFSET + st * L::P_BYTES + r * 128;
#pragma unroll
      for (int c = side * HALF_KEYS; c < side * HALF_KEYS + HALF_KEYS; c += 32) {
        float s[32];
        tmem_load32(lane_base + st * L::S_COLUMNS + c, s);
        if (unmasked) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            s[i] = fast_exp2(fmaf(s[i], factor, offset));
            sum4[i & 3] += s[i];
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int key = c + i;
            const float e = fast_exp2(fmaf(s[i], factor, offset));
            s[i] = (key >= lo && key <= hi && factor != 0.f) ? e : 0.f;
            sum4[i & 3] += s[i];
          }
        }
        // 32 keys = four 16-byte chunks of this row in the k-block c / 64, swizzled by the row.
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 packed;
          __nv_bfloat162* h2 = (__nv_bfloat162*)&packed;
#pragma unroll
          for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(s[j * 8 + 2 * e], s[j * 8 + 2 * e + 1]);
          const int chunk = ((c & 63) >> 3) + j;
          *(uint4*)(p_row + (c >> 6) * L::HALF_TILE_BYTES + ((chunk ^ (r & 7)) << 4)) = packed;
        }
      }
      row_sum = row_sum * rescale + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));   // this thread's keys only
      tcgen05_fence_before();
      mbar_arrive(bar(S_EMPTY, st));                            // this thread's part of the score buffer is read
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // P is for the tensor core's eyes
      mbar_arrive(bar(P_READY, st));
      if (t >= 1) add_product(t - 1, owed_scale);
      if (!ok) break;
      owed_scale = rescale;
    }
    if (n_tiles > 0 && ok) add_product(n_tiles - 1, owed_scale);
    // The row's sum is the two threads' sums (both are relative to the same maximum).
    ok = __all_sync(0xffffffffu, ok);
    if (working && ok) {
      exchange[side * 128 + r] = row_sum;
      mbar_arrive(bar(X_READY));
      ok = mbar_wait(bar(X_READY), n_tiles & 1, abort_flag, p.error, 12);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) row_sum += exchange[(side ^ 1) * 128 + r];
    }
  }

  if constexpr (SPLIT) {
    // The blocks behind the first leave their rows' maxima, sums and outputs in their own
    // shared memory, where the keys and values lay (every product that read those has
    // completed: the softmax threads waited for the last one); the first block reads them
    // there once the whole cluster has arrived, and nobody leaves before it has.
    float* stage = (float*)(generic_base + L::K_OFFSET);              // [D][128]: a dimension's 128 rows side by side
    float* stage_stats = (float*)(generic_base + L::V_OFFSET);        // [2][128]: maximum, sum
    if (warp >= 2 && rank != 0) {
      const bool has = working && ok;
      if (side == 0) {
        stage_stats[r] = has ? row_max : -FLT_MAX;
        stage_stats[128 + r] = has ? row_sum : 0.f;
      }
      if (has) {
#pragma unroll
        for (int i = 0; i < HALF_D; ++i) stage[(side * HALF_D + i) * 128 + r] = acc[i];
      }
    }
    cluster_arrive();
    cluster_wait();
    if (warp >= 2 && rank == 0 && working && ok) {
      for (int other = 1; other < ranks; ++other) {
        const float their_sum = load_from_block(smem_u32(stage_stats + 128 + r), other);
        if (their_sum > 0.f) {
          const float their_max = load_from_block(smem_u32(stage_stats + r), other);
          const float both = fmaxf(row_max, their_max);
          const float mine = row_max == -FLT_MAX ? 0.f : fast_exp2(row_max - both);
          const float theirs = fast_exp2(their_max - both);
#pragma unroll
          for (int i = 0; i < HALF_D; ++i)
            acc[i] = acc[i] * mine + load_from_block(smem_u32(stage + (side * HALF_D + i) * 128 + r), other) * theirs;
          row_sum = row_sum * mine + their_sum * theirs;
          row_max = both;
        }
      }
    }
    cluster_arrive();
    cluster_wait();
  }

  if (warp >= 2 && rank == 0 && ok && r < rows) {
    const float inv = row_sum > 0.f ? 1.f / row_sum : 0.f;
    __nv_bfloat16* out = p.out + ((size_t)(first_token + tile * BQ + r) * p.heads + h) * D + side * HALF_D;
#pragma unroll
    for (int c = 0; c < HALF_D; c += 8) {
      uint4 packed;
      __nv_bfloat162* h2 = (__nv_bfloat162*)&packed;
#pragma unroll
      for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(acc[c + 2 * e] * inv, acc[c + 2 * e + 1] * inv);
      *(uint4*)(out + c) = packed;
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLUMNS);
  }
}

// ---------------------------------------------------------------------------------------
// The paired form, for launches of many blocks (long prompts, many requests or heads) and for short ones
// (`takes_paired`). A block walks the keys 64 at a time with one softmax thread per query row, and
// keeps O in tensor memory over all tiles instead of reading each tile's product back:
// 97 KB of shared memory, 256 columns of tensor memory and 192 threads, so two blocks share
// an SM and the softmax of one overlaps the products and the waits of the other.
//
// The probabilities of a tile go into tensor memory, over the scores they came from, and are the second product's A
// operand there: no trip through shared memory (sixteen-byte stores into the swizzled layout, a proxy fence, and 16 KB that
// the tensor core reads back), and the softmax never waits for a product unless a reference moves. The thread that issues the MMAs
// waits for the product of the tile before last before the next scores are written over the probabilities it reads; its warp runs the
// role together and an elected lane issues, and K is asked for two tiles ahead of its scores. Scale and sum take two scores an instruction. 8,192 tokens,
// 12 heads of 128, us: 277 with the probabilities in shared memory and one score an instruction, 258 without, 235 with K asked for early, 173 with a
// tile's pages in one box and no look at the maximum (below): 1,190 TFLOP/s, bound by the exponentials and by the tensor cores' turns between two blocks.
//
// The reference of a row is its running maximum, but in launches that fill the GPU it is left behind: probabilities are taken against it
// without a look at the tile's maximum (which costs a pass over the scores), and while the tile's sum is at most REFERENCE_LIMIT, 2^8, for every row of the warp, that
// holds: no probability is above 2^8, which float32 sums and the bfloat16 operand hold as well as values below 1. A tile with a larger sum
// is taken again with all references of the warp moved to their maxima; only then is the output in tensor memory (which must be multiplied by 2^(old - new))
// touched. The sum is kept against the same reference, so the quotient is exact softmax. A largest probability that is not
// 1 is rounded, though: 1 % further from 64 bits than the wide form, 2 to 5 % where the maxima grow all along the keys by 2^8 to 2^100
// in all. The limit is what bounds that: with 2^10 the error is up to 0.6 % larger, with 2^40 up to 2 % (head size 64, 1,500 tokens after
// 3,000, growth 2^100: 0.002290, 0.002303 and 0.002337 of the outputs' norm; moved where the maximum had grown by 2^8, with a look at every tile's:
// 0.002304); taking tiles again costs growing maxima 102 -> 111 us (2^8 over 1,500 tokens after 3,000, 28 heads of 128) to 156 (2^100). Smaller launches, which would
// otherwise take the wide form, move it with every new maximum: a little closer than the wide form (0.00228) for 0.6 us at 100 tokens (7.9 -> 8.5), 1.5 at 6
// requests of 300 (14.1 -> 15.6).
// ---------------------------------------------------------------------------------------
namespace paired {

constexpr int BKEYS = 64;           // keys per tile
constexpr int THREADS = 192;        // TMA warp, MMA warp, four softmax warps (one thread per query row)
constexpr int SOFTMAX_WARPS = 4;
constexpr int KV_STAGES = 2;
constexpr float REFERENCE_SLACK = 8.f;   // of launches that fill the GPU; 0 below that (`launch`)
constexpr float REFERENCE_LIMIT = 256.f; // 2^REFERENCE_SLACK: of a tile's sum against its rows' references

// 64 consecutive float32 columns of this thread's lane of tensor memory.
__device__ __forceinline__ void tmem_load64(uint32_t address, float* v) {
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(address)
      : "memory");
#pragma unroll
  for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 columns that are there after `tmem_arrived` of the same variables.
__device__ __forceinline__ void tmem_ask32(uint32_t address, float (&v)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
               : "r"(address)
               : "memory");
}
__device__ __forceinline__ void tmem_arrived(float (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15]), "+f"(v[16]), "+f"(v[17]), "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]), "+f"(v[22]), "+f"(v[23]), "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27]), "+f"(v[28]), "+f"(v[29]), "+f"(v[30]), "+f"(v[31])
               :
               : "memory");
}
// 32 columns written (the whole warp calls it).
__device__ __forceinline__ void tmem_store32(uint32_t address, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
      "tcgen05.wait::st.sync.aligned;"
      ::"r"(address), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem]^T: a lane of A is a row, a column holds two neighbouring bfloat16 of K.
__device__ __forceinline__ void umma_bf16_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Two floats side by side: one instruction for both, each rounded as the single one rounds.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
template <int D>
struct Layout {
  static constexpr int HALVES = D / 64;                       // 64-column k-blocks of the head dimension
  static constexpr int Q_HALF_BYTES = BQ * 128;               // 128 rows x 64 bfloat16
  static constexpr int KV_HALF_BYTES = BKEYS * 128;           // 64 rows x 64 bfloat16
  static constexpr int Q_BYTES = HALVES * Q_HALF_BYTES;
  static constexpr int KV_BYTES = HALVES * KV_HALF_BYTES;     // one stage of K, or of V
  static constexpr int Q_OFFSET = 0;
  static constexpr int K_OFFSET = Q_BYTES;                    // two stages
  static constexpr int V_OFFSET = K_OFFSET + KV_STAGES * KV_BYTES;
  static constexpr int BAR_OFFSET = V_OFFSET + KV_STAGES * KV_BYTES;
  static constexpr int USED_BYTES = BAR_OFFSET + 256;
  // 768 bytes of slack for the 1024-byte alignment of the tiles: with it two blocks of head
  // size 128 still fit on one SM. The kernel checks that the slack was enough.
  static constexpr size_t SMEM_BYTES = (size_t)USED_BYTES + 768;
  static constexpr int S_COLUMNS = BKEYS;                     // per score buffer; its first half holds the tile's probabilities later
  static constexpr int O_COLUMN = 2 * S_COLUMNS;              // O behind the two score buffers
  static constexpr int TMEM_COLUMNS = 256;
};

enum Bar : int {
  Q_FULL = 0, O_FULL = 1, S_FULL = 2, P_READY = 4, O_REST = 6,
  K_FULL = 7, K_EMPTY = K_FULL + KV_STAGES, V_FULL = K_EMPTY + KV_STAGES, V_EMPTY = V_FULL + KV_STAGES, NUM_BARS = V_EMPTY + KV_STAGES
};

template <int D>
__global__ void __launch_bounds__(THREADS, 2) prefill_tcgen05_paired_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                     const __grid_constant__ PageMaps maps, const Params p) {
  using L = Layout<D>;
  if (threadIdx.x == 0) {         // the descriptors do not depend on the kernel before: fetch them early
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.key_run) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.value_run) : "memory");
  }
  extern __shared__ __align__(1024) uint8_t raw_smem[];
  const uint32_t raw = smem_u32(raw_smem);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* generic_base = raw_smem + (base - raw);
  const uint32_t bars = base + L::BAR_OFFSET;
  volatile uint32_t* tmem_holder = (volatile uint32_t*)(generic_base + L::BAR_OFFSET + 8 * NUM_BARS);
  volatile int* abort_flag = (volatile int*)(tmem_holder + 1);
  auto bar = [&](int which, int i = 0) { return bars + 8u * (which + i); };
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const bool fits = (base - raw) + (uint32_t)L::USED_BYTES <= (uint32_t)L::SMEM_BYTES;
  if (!fits) {                     // the alignment took more than the slack: nothing is touched
    if (threadIdx.x == 0) atomicCAS(p.error, 0, 20);
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(bar(Q_FULL), 1);
    for (int i = 0; i < KV_STAGES; ++i) {
      mbar_init(bar(K_FULL, i), 1);
      mbar_init(bar(K_EMPTY, i), 1);
      mbar_init(bar(V_FULL, i), 1);
      mbar_init(bar(V_EMPTY, i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(S_FULL, i), 1);
      // One arrival per warp. Two of them, like the score buffers: the softmax may finish a tile before the MMA thread has
      // looked at the tile before, but not two (the scores of tile t + 2 follow the product of tile t).
      mbar_init(bar(P_READY, i), SOFTMAX_WARPS);
    }
    mbar_init(bar(O_REST), 1);                       // by tcgen05.commit: the second product of a tile has completed
    mbar_init(bar(O_FULL), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32((const void*)tmem_holder), L::TMEM_COLUMNS);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  dependent_launch_trigger();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  // ---- what this block works on (the same in every role) -------------------------------
  // The step's integers are read before the wait for the kernel before this one (they were on
  // the device before the step's first kernel began); q and this step's keys and values after it.
  const int h = blockIdx.x, b = p.work_index != nullptr ? p.work_index[blockIdx.z] : (int)blockIdx.z;
  const int first_token = p.q_start[b];
  const int q_count = p.q_start[b + 1] - first_token;
  const int q_tiles = (q_count + BQ - 1) / BQ;
  // Late tiles see the most keys: they go first in every head (the head is the fastest grid
  // index, so the first wave holds the longest blocks of all heads), the short early ones
  // fill in behind them.
  const int tile = q_tiles - 1 - (int)blockIdx.y;
  const bool active = tile >= 0 && !(p.skip_single && q_count == 1);
  const int rows = active ? min(BQ, q_count - tile * BQ) : 0;
  const int pos0 = p.q_pos0[b] + tile * BQ;
  const int kv_end = active ? min(p.kv_len[b], pos0 + rows) : 0;
  const int first_key = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
  const int kv_begin = (first_key / BKEYS) * BKEYS;
  const int n_tiles = active ? (kv_end - kv_begin + BKEYS - 1) / BKEYS : 0;
  const int g = h / (p.heads / p.kv_heads);
  // The producer's lane i brings box i of a tile (a page, or the 64 rows of a larger page that
  // the tile covers): the first tile's table entries, before the wait.
  const int box_rows = min(p.page_size, BKEYS);
  const int last_page = active ? (kv_end - 1) / p.page_size : 0;     // the last page that holds a visible key
  // The first tile starts on a multiple of 64 keys, which may lie pages before the window's first
  // key; those pages may have been given back (their table entries are holes). Their keys are
  // masked, so the window's first page stands in for them.
  const int window_page = first_key / p.page_size;
  int first_page = 0;
  if (warp == 0 && active && lane < BKEYS / box_rows)
    first_page = checked_page(p.block_table[(size_t)b * p.table_width +
                                            checked_table_index(max(min((kv_begin + lane * box_rows) / p.page_size, last_page), window_page), p.table_width)]);
  dependent_launch_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // Lane i brings box i of a tile (its block-table entry and its copies), so the table
    // look-ups of a tile are one round trip, not one per page. A box is a page, or the 64
    // rows of a larger page that the tile covers. Lane 0 posts the byte counts before any
    // lane issues a copy.
    if (active) {
      if (lane == 0) {
        mbar_expect_tx(bar(Q_FULL), L::Q_BYTES);
#pragma unroll
        for (int half = 0; half < L::HALVES; ++half)
          tma_load_2d(base + L::Q_OFFSET + half * L::Q_HALF_BYTES, &map_q, bar(Q_FULL), h * D + half * 64,
                      first_token + tile * BQ);
      }
      const int* table = p.block_table + (size_t)b * p.table_width;
      const int boxes = BKEYS / box_rows;
      const bool mine = lane < boxes;
      // A page past the last visible key may not exist: its rows are masked, so any page of
      // the request will do; the last visible one is taken.
      const int page_shift = 31 - __clz(p.page_size);          // page sizes are powers of two
      auto page_of = [&](int t) {
        const int key = kv_begin + t * BKEYS + lane * box_rows;
        return mine && t < n_tiles ? checked_page(table[checked_table_index(max(min(key >> page_shift, last_page), window_page), p.table_width)]) : 0;
      };
      // One tile of K or of V into its stage. In this order: V of tile t may follow when the product of tile t - 2 has completed, and the
      // scores of tile t, which free the stage of K for tile t + 2, follow that product. So K is asked for two tiles ahead of its
      // scores (K and V of a tile together, K waited for V's stage, one tile: the scores then came 820 cycles late).
      auto load = [&](bool values, int t, int page) {
        const int stage = t % KV_STAGES;
        const uint32_t full = bar(values ? V_FULL : K_FULL, stage);
        if (t >= KV_STAGES && !mbar_wait_warp(bar(values ? V_EMPTY : K_EMPTY, stage), (t / KV_STAGES - 1) & 1, abort_flag, p.error, values ? 10 : 1))
          return false;
        if (lane == 0) mbar_expect_tx(full, L::KV_BYTES);
        __syncwarp();
        load_pages<D>(maps, values, base + (values ? L::V_OFFSET : L::K_OFFSET) + stage * L::KV_BYTES, full, BKEYS, box_rows, lane, g, page,
                      (kv_begin + t * BKEYS + lane * box_rows) & (p.page_size - 1));
        return true;
      };
      int page0 = first_page;
      bool ok = true;
      int keys_issued = 0, values_issued = 0;
      if (n_tiles > 0) {                                        // a request without a visible key has none: nobody would wait for a copy
        ok = load(false, 0, page0);
        keys_issued = 1;
      }
      int page1 = page_of(1), page2 = page_of(2);               // of tiles t, t + 1, t + 2
      if (n_tiles > 1) {
        ok = ok && load(false, 1, page1);
        keys_issued = 2;
      }
      for (int t = 0; t < n_tiles && ok; ++t) {
        const int page3 = page_of(t + 3);
        if (!(ok = load(true, t, page0))) break;
        values_issued = t + 1;
        if (t + 2 < n_tiles) {
          if (!(ok = load(false, t + 2, page2))) break;
          keys_issued = t + 3;
        }
        page0 = page1;
        page1 = page2;
        page2 = page3;
      }
      if (lane == 0 && *abort_flag) {      // copies that were issued still write into this block's shared memory
        for (int t = max(0, keys_issued - KV_STAGES); t < keys_issued; ++t)
          for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(bar(K_FULL, t % KV_STAGES), (t / KV_STAGES) & 1); ++w) __nanosleep(64);
        for (int t = max(0, values_issued - KV_STAGES); t < values_issued; ++t)
          for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(bar(V_FULL, t % KV_STAGES), (t / KV_STAGES) & 1); ++w) __nanosleep(64);
        for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(bar(Q_FULL), 0); ++w) __nanosleep(64);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (active) {
      const bool leader = elect_one();
      constexpr uint32_t idesc_s = instruction_descriptor(BQ, BKEYS, false);
      constexpr uint32_t idesc_o = instruction_descriptor(BQ, D, true);
      const uint64_t q_first = smem_descriptor(base + L::Q_OFFSET), k_first = smem_descriptor(base + L::K_OFFSET);
      const uint64_t v_first = mn_major_descriptor(base + L::V_OFFSET, box_rows * 128);
      bool ok = mbar_wait_warp(bar(Q_FULL), 0, abort_flag, p.error, 2);
      auto issue_scores = [&](int t) {
        const int st = t & 1, stage = t % KV_STAGES;
        ok = ok && mbar_wait_warp(bar(K_FULL, stage), (t / KV_STAGES) & 1, abort_flag, p.error, 3);
        // These scores go where the probabilities of tile t - 2 lay.
        if (t >= 2) ok = ok && mbar_wait_warp(bar(O_REST), (t - 2) & 1, abort_flag, p.error, 4);
        if (!ok) return;
        tcgen05_fence_after();
        const uint64_t keys = further(k_first, stage * L::KV_BYTES);
        if (leader) {
#pragma unroll
          for (int half = 0; half < L::HALVES; ++half)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_bf16(tmem_base + st * L::S_COLUMNS, further(q_first, half * L::Q_HALF_BYTES + k * 32),
                        further(keys, half * L::KV_HALF_BYTES + k * 32), idesc_s, (half > 0 || k > 0) ? 1u : 0u);
          tcgen05_commit(bar(S_FULL, st));
          tcgen05_commit(bar(K_EMPTY, stage));    // the K stage is free once these MMAs have read it
        }
        __syncwarp();
      };
      if (n_tiles > 0) issue_scores(0);
      for (int t = 0; t < n_tiles && ok; ++t) {
        if (t + 1 < n_tiles) issue_scores(t + 1);
        const int stage = t % KV_STAGES;
        ok = ok && mbar_wait_warp(bar(V_FULL, stage), (t / KV_STAGES) & 1, abort_flag, p.error, 5);
        ok = ok && mbar_wait_warp(bar(P_READY, t & 1), (t >> 1) & 1, abort_flag, p.error, 6);
        if (!ok) break;
        tcgen05_fence_after();
        const uint64_t values = further(v_first, stage * L::KV_BYTES);
        if (leader) {
#pragma unroll
          for (int k = 0; k < BKEYS / 16; ++k)     // 16 keys a step: eight columns of P, two groups of 8 rows of V
            umma_bf16_tmem_a(tmem_base + L::O_COLUMN, tmem_base + (t & 1) * L::S_COLUMNS + k * 8, further(values, value_step<D>(k, box_rows)), idesc_o, (t > 0 || k > 0) ? 1u : 0u);
          tcgen05_commit(bar(O_REST));             // O is at rest until the next P is ready
          tcgen05_commit(bar(V_EMPTY, stage));
          if (t + 1 == n_tiles) tcgen05_commit(bar(O_FULL));       // the output is complete
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, one thread per row
    const int quadrant = warp & 3;
    const int r = quadrant * 32 + lane;                       // row of the tile, lane of tensor memory
    const uint32_t lane_base = tmem_base + ((uint32_t)(quadrant * 32) << 16);
    const int my_pos = pos0 + r;
    float reference = -FLT_MAX, row_sum = 0.f;                // the reference in units of log2, scaled
    bool ok = true;
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t & 1;
      const int key0 = kv_begin + t * BKEYS;
      ok = ok && mbar_wait(bar(S_FULL, st), (t >> 1) & 1, abort_flag, p.error, 8);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      // The whole tile is visible to every row of the block: no mask. Otherwise a row sees the
      // keys lo..hi of the request (nothing when the row is past the request's tokens).
      const bool unmasked = key0 + BKEYS - 1 <= pos0 && key0 + BKEYS <= kv_end && key0 >= first_key &&
                            (p.window <= 0 || pos0 + rows - 1 - key0 < p.window);
      const int hi = r < rows ? min(my_pos, kv_end - 1) - key0 : -1;          // relative to the tile
      const int lo = (p.window > 0 ? max(first_key, my_pos - p.window + 1) : first_key) - key0;
      uint32_t packed[BKEYS / 2];
      uint64_t sum01, sum23;
      uint64_t factor2, offset2;
      bool has_reference;
      // exp2(s * scale - reference) as one fused multiply-add and one ex2; a row that has seen
      // no key yet has no reference and every probability 0.
      auto begin = [&] {
        has_reference = reference != -FLT_MAX;
        const float offset = has_reference ? -reference : 0.f, factor = has_reference ? p.scale_log2 : 0.f;
        factor2 = pack2(factor, factor);
        offset2 = pack2(offset, offset);
        sum01 = sum23 = 0;                                      // (0.f, 0.f)
      };
      auto take = [&](const float* s, int i, auto visible) {    // s: the scores of keys i .. i + 3
        float e[4];
        unpack2(fma2(pack2(s[0], s[1]), factor2, offset2), e[0], e[1]);
        unpack2(fma2(pack2(s[2], s[3]), factor2, offset2), e[2], e[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = visible(i + j) ? fast_exp2(e[j]) : 0.f;
        sum01 = add2(sum01, pack2(e[0], e[1]));
        sum23 = add2(sum23, pack2(e[2], e[3]));
        const __nv_bfloat162 h01 = __floats2bfloat162_rn(e[0], e[1]), h23 = __floats2bfloat162_rn(e[2], e[3]);
        packed[i / 2] = *(const uint32_t*)&h01;
        packed[i / 2 + 1] = *(const uint32_t*)&h23;
      };
      auto take32 = [&](const float* s, int first) {
        if (unmasked) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) take(s + i, first + i, [](int) { return true; });
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 4) take(s + i, first + i, [&](int key) { return key >= lo && key <= hi && has_reference; });
        }
      };
      auto tile_sum = [&] {
        float sums[4];
        unpack2(sum01, sums[0], sums[1]);
        unpack2(sum23, sums[2], sums[3]);
        return (sums[0] + sums[1]) + (sums[2] + sums[3]);
      };
      const uint32_t scores = lane_base + st * L::S_COLUMNS;
      bool taken = false;
      float slack = p.slack;
      if (p.slack > 0.f && !__any_sync(0xffffffffu, reference == -FLT_MAX)) {
        // Every row has a reference: the probabilities are taken against it without a look at the tile's maximum, the second half
        // of the scores on its way meanwhile. Should a sum come out above REFERENCE_LIMIT (or not a number), the tile is taken again below.
        float s[32], behind[32];
        tmem_ask32(scores, s);
        tmem_arrived(s);
        tmem_ask32(scores + 32, behind);
        begin();
        take32(s, 0);
        tmem_arrived(behind);
        take32(behind, 32);
        const float sum = tile_sum();
        taken = __all_sync(0xffffffffu, sum <= REFERENCE_LIMIT);
        if (taken) row_sum += sum;
        else slack = 0.f;                  // every row of the warp starts anew from its maximum: the next tiles are taken at once again
      }
      if (!taken) {
        float s[BKEYS];
        tmem_load64(scores, s);
        float m4[4] = {-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (unmasked) {
#pragma unroll
          for (int i = 0; i < BKEYS; ++i) m4[i & 3] = fmaxf(m4[i & 3], s[i]);
        } else {
#pragma unroll
          for (int i = 0; i < BKEYS; ++i) m4[i & 3] = fmaxf(m4[i & 3], (i >= lo && i <= hi) ? s[i] : -FLT_MAX);
        }
        float tile_max = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        if (tile_max != -FLT_MAX) tile_max *= p.scale_log2;        // the scale is positive: max(s) scales with it
        const bool moves = tile_max > reference + slack || (reference == -FLT_MAX && tile_max != -FLT_MAX);
        if (__any_sync(0xffffffffu, moves)) {
          // Some row of this warp moves its reference: its sum and its row of O are multiplied
          // by 2^(old - new); the other rows by 1. Reading and writing tensor memory takes the whole warp.
          const float shrink = !moves ? 1.f : (reference == -FLT_MAX ? 0.f : fast_exp2(reference - tile_max));
          if (moves) {
            reference = tile_max;
            row_sum *= shrink;
          }
          if (t >= 1) {
            ok = mbar_wait(bar(O_REST), (t - 1) & 1, abort_flag, p.error, 7);      // the product of the tile before has completed
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int c = 0; c < D; c += 32) {
              float o[32];
              uint32_t back[32];
              tmem_load32(lane_base + L::O_COLUMN + c, o);
#pragma unroll
              for (int i = 0; i < 32; ++i) back[i] = __float_as_uint(o[i] * shrink);
              tmem_store32(lane_base + L::O_COLUMN + c, back);
            }
          }
        }
        begin();
        take32(s, 0);
        take32(s + 32, 32);
        row_sum += tile_sum();
      }
      tmem_store32(scores, packed);      // over the scores, which are in registers
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(P_READY, st));
    }
    ok = __all_sync(0xffffffffu, ok);
    if (active && ok && n_tiles > 0) {
      ok = mbar_wait(bar(O_FULL), 0, abort_flag, p.error, 9);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tcgen05_fence_after();
        const float inv = row_sum > 0.f ? 1.f / row_sum : 0.f;
        __nv_bfloat16* out = p.out + ((size_t)(first_token + tile * BQ + r) * p.heads + h) * D;
#pragma unroll
        for (int c = 0; c < D; c += 32) {
          float o[32];
          tmem_load32(lane_base + L::O_COLUMN + c, o);        // every lane takes part
          if (r < rows) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 packed;
              __nv_bfloat162* h2 = (__nv_bfloat162*)&packed;
#pragma unroll
              for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(o[j * 8 + 2 * e] * inv, o[j * 8 + 2 * e + 1] * inv);
              *(uint4*)(out + c + j * 8) = packed;
            }
          }
        }
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLUMNS);
  }
}

}  // namespace paired

// ---------------------------------------------------------------------------------------
// A pool [pages, kv_heads, page_size, d] as boxes of `rows` rows of `halves` halves of `run` pages, 128-byte swizzle.
int page_map(CUtensorMap* out, const void* ptr, long long pages, int kv_heads, int page_size, int d, int rows, int halves, int run) {
  EncodeTiled encode = encode_tiled();
  if (encode == nullptr) return fail(101, "paged_attention_tcgen05: the driver does not export cuTensorMapEncodeTiled");
  const cuuint64_t dims[5] = {64, (cuuint64_t)page_size, (cuuint64_t)(d / 64), (cuuint64_t)kv_heads, (cuuint64_t)pages};
  const cuuint64_t strides[4] = {(cuuint64_t)d * 2, 128, (cuuint64_t)page_size * d * 2, (cuuint64_t)kv_heads * page_size * d * 2};
  const cuuint32_t box[5] = {64, (cuuint32_t)rows, (cuuint32_t)halves, 1, (cuuint32_t)run};
  const cuuint32_t element_strides[5] = {1, 1, 1, 1, 1};
  CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(ptr), dims, strides, box, element_strides,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(102, "paged_attention_tcgen05: cuTensorMapEncodeTiled failed with %d for pages of %d", (int)r, page_size);
  return 0;
}
// What brings tiles of `tile_keys` keys. A pool's maps say where it lies and how it is laid out, nothing of what it holds; they are kept
// (encoding four takes a microsecond and more of every launch).
struct PageMapsKey {
  const void *keys, *values;
  long long pages;
  int kv_heads, page_size, d, tile_keys;
  bool operator==(const PageMapsKey& o) const {
    return keys == o.keys && values == o.values && pages == o.pages && kv_heads == o.kv_heads && page_size == o.page_size && d == o.d && tile_keys == o.tile_keys;
  }
};
struct PageMapsKeyHash {
  size_t operator()(const PageMapsKey& key) const {
    size_t h = (size_t)key.keys;
    h = h * 1000003u ^ (size_t)key.values;
    h = h * 1000003u ^ (size_t)key.pages;
    h = h * 1000003u ^ (size_t)(key.kv_heads * 4096 + key.page_size);
    return h * 1000003u ^ (size_t)(key.d * 4096 + key.tile_keys);
  }
};
int page_maps(PageMaps* out, const void* keys, const void* values, long long pages, int kv_heads, int page_size, int d, int tile_keys) {
  static std::mutex mutex;
  static std::unordered_map<PageMapsKey, PageMaps, PageMapsKeyHash> cache;
  const PageMapsKey key{keys, values, pages, kv_heads, page_size, d, tile_keys};
  std::lock_guard<std::mutex> guard(mutex);
  auto found = cache.find(key);
  if (found != cache.end()) {
    *out = found->second;
    return 0;
  }
  const int rows = page_size < tile_keys ? page_size : tile_keys, run = tile_keys / rows, halves = d / 64;
  if (int err = page_map(&out->key, keys, pages, kv_heads, page_size, d, rows, 1, 1)) return err;
  if (int err = page_map(&out->value, values, pages, kv_heads, page_size, d, rows, halves, 1)) return err;
  if (int err = page_map(&out->key_run, keys, pages, kv_heads, page_size, d, rows, 1, run)) return err;
  if (int err = page_map(&out->value_run, values, pages, kv_heads, page_size, d, rows, halves, run)) return err;
  if (cache.size() > 1024) cache.clear();
  cache.emplace(key, *out);
  return 0;
}

int sm_count() {
  static int count = [] {
    int device = 0, n = 148;
    if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
    return n;
  }();
  return count;
}

// Whether form 0 takes the paired kernel. Two of its blocks share an SM, so up to two blocks per SM run at once; of the wide
// kernel one. Times in us from launches of 12 and 28 heads, 1 to 12 requests of 64 to 2,000 tokens over up to 4,000 keys:
// a wide block 5.5 + 1.95 per tile of 128 keys; a wide block that follows another 4 more; a round of paired blocks 6.5 + 3.0
// per tile. With more blocks than SMs and fewer than twice as many, the wide launch's second blocks follow its shortest
// first ones, so it lasts as long as its longest block or two of middling length: the two estimates are compared (6 requests
// of 300 tokens, 12 heads: wide 21.3, paired 15.8; 4 portions of 509 tokens after 512: 34.3 and 29.7; but one prompt of 2,048
// tokens: 31.9 and 43.2). From twice as many on it is the paired kernel (4,096 tokens 87.5 and 63.0). With one of its
// tiles, and up to three while at most a third of the SMs are busy, the paired kernel's shorter set-up shows (64 tokens 8.3 and 6.3, 100 tokens
// 8.9 and 8.5, 192 tokens 10.3 and 9.1; but 200 tokens of 28 heads 10.2 and 10.9, 300 of 12 11.3 and 11.7).
bool takes_paired(long long blocks, long long blocks_per_tile, int longest, int longest_keys) {
  const int sms = sm_count();
  if (blocks >= 2LL * sms) return true;
  if (blocks <= sms) return longest_keys <= 64 || (longest_keys <= 192 && blocks * 3 <= sms);
  const float middle = fmaxf(0.f, longest - (float)sms / blocks_per_tile);
  const float wide = fmaxf(5.5f + 1.95f * longest, 18.f + 3.9f * middle), paired = 6.5f + 3.f * longest;
  return paired < wide;
}

// form 0 picks by the size of the launch: the paired kernel (above), else the wide one, and when its blocks are fewer than half
// of the SMs (a short portion
// of a prompt over a long context) a query tile's keys are shared out over a cluster of 2, 4 or
// 8 blocks, as long as all blocks still run at once and each has two key tiles or more. A block
// costs about 10 us around its tiles and only one fits an SM, so a second wave of blocks would
// cost more than the shorter chains save: 128 tokens after 8,192 take 123 us in 12 blocks.
// 1: wide, no clusters; 2: paired; 4, 8, 16: wide in clusters of 2, 4, 8.
template <int D>
int launch(Params p, const void* qkv, const void* keys, const void* values, int tokens, long long pages, int seqs,
           int working_seqs, int max_q_len, int max_kv_len, int form, int* chosen, cudaStream_t stream) {
  // With a list of the requests to work on, the grid covers those only. Without one it covers
  // all, and the blocks of requests that are left to the decode kernel return at once; they do
  // not count below, but each still costs its launch (one block of 200 KB per SM at a time: 65
  // requests of which one brings a portion took 75 us where that portion needs 15).
  dim3 grid(p.heads, (max_q_len + BQ - 1) / BQ, p.work_index != nullptr ? working_seqs : seqs);
  const long long blocks = (long long)grid.x * grid.y * working_seqs;
  const int seen = p.window > 0 && p.window + BQ < max_kv_len ? p.window + BQ : max_kv_len;
  const int longest = (seen + BKEYS - 1) / BKEYS;          // key tiles of the longest block
  const bool use_paired = form == 2 || (form == 0 && takes_paired(blocks, (long long)p.heads * working_seqs, longest, seen));
  p.slack = blocks >= 2LL * sm_count() ? paired::REFERENCE_SLACK : 0.f;
  unsigned ranks = 1;
  if (form == 4 || form == 8 || form == 16) ranks = form / 2;
  if (form == 0 && !use_paired) {
    while (ranks < 8 && blocks * (ranks * 2) <= sm_count() && longest >= (int)(ranks * 2) * 2) ranks *= 2;
  }
  CUtensorMap map_q;
  if (int err = tensor_map(&map_q, qkv, tokens, (p.heads + 2 * p.kv_heads) * D, BQ)) return err;
  PageMaps maps;
  if (int err = page_maps(&maps, keys, values, pages, p.kv_heads, p.page_size, D, use_paired ? paired::BKEYS : BKEYS)) return err;
  static DevicesSet raised_one, raised_cluster, raised_paired;
  if (int err = raise_shared_memory(raised_one, prefill_tcgen05_kernel<D, false>, Layout<D>::SMEM_BYTES, "paged_attention_tcgen05")) return err;
  if (int err = raise_shared_memory(raised_cluster, prefill_tcgen05_kernel<D, true>, Layout<D>::SMEM_BYTES, "paged_attention_tcgen05")) return err;
  if (int err = raise_shared_memory(raised_paired, paired::prefill_tcgen05_paired_kernel<D>, paired::Layout<D>::SMEM_BYTES, "paged_attention_tcgen05"))
    return err;
  if (chosen != nullptr) *chosen = use_paired ? 0 : (int)ranks;
  if (use_paired) {
    launch_kernel(paired::prefill_tcgen05_paired_kernel<D>, grid, paired::THREADS, paired::Layout<D>::SMEM_BYTES, stream, map_q, maps,
                  p);
  } else {
    grid.x *= ranks;
    if (ranks > 1)
      launch_kernel_cluster(prefill_tcgen05_kernel<D, true>, grid, dim3(THREADS), Layout<D>::SMEM_BYTES, stream, ranks, map_q, maps, p);
    else
      launch_kernel(prefill_tcgen05_kernel<D, false>, grid, THREADS, Layout<D>::SMEM_BYTES, stream, map_q, maps, p);
  }
  return check_launch("paged_attention_tcgen05");
}

}  // namespace

PAE_EXPORT int pae_attention_tcgen05_supports(int heads, int kv_heads, int d, int page_size) {
  return (d == 64 || d == 128) && (page_size == 16 || page_size == 32 || page_size == 64 || page_size == 128) &&
         kv_heads >= 1 && heads % kv_heads == 0;
}

// Attention of every request that brings more than one token (or every request, unless
// skip_single; `singles` is how many bring one, -1 when the caller does not know). form 0 picks the kernel by the size of the launch, 1 and 2 name it (tests); `chosen` (a host pointer, or null) receives the blocks per query tile of this launch: 1 without clusters, 0 for the paired kernel. `work_index` (device, or null) lists the `work_count` requests that the launch is to cover, in place of all `seqs`. qkv [tokens, heads + 2 kv_heads, d]; keys, values [pages, kv_heads, page_size, d].
PAE_EXPORT int pae_paged_attention_prefill_tcgen05(void* out, const void* qkv, const void* keys, const void* values,
                                                   long long pages, const int* block_table, int table_width,
                                                   const int* q_start, const int* q_pos0, const int* kv_len, int tokens,
                                                   int seqs, int max_q_len, int max_kv_len, int heads, int kv_heads, int d,
                                                   int page_size, float scale, int window, int skip_single, int singles, int form, int* chosen,
                                                   const int* work_index, int work_count, int* error, void* stream) {
  if (seqs == 0 || max_q_len == 0 || tokens == 0) return 0;
  if (work_index != nullptr && (work_count < 1 || work_count > seqs))
    return fail(2, "paged_attention_tcgen05: a list of %d requests to work on, of %d", work_count, seqs);
  if (!pae_attention_tcgen05_supports(heads, kv_heads, d, page_size))
    return fail(2, "paged_attention_tcgen05: head_dim %d with pages of %d is not taken (64 or 128; 16, 32, 64 or 128)", d, page_size);
  if (heads > 65535 || seqs > 65535) return fail(3, "paged_attention_tcgen05: %d heads x %d requests exceed one launch", heads, seqs);
  if ((((uintptr_t)qkv | (uintptr_t)keys | (uintptr_t)values | (uintptr_t)out) & 15) != 0)
    return fail(2, "paged_attention_tcgen05: an operand does not start on a 16-byte boundary");
  Params p{};
  p.out = (__nv_bfloat16*)out;
  p.block_table = block_table;
  p.q_start = q_start;
  p.q_pos0 = q_pos0;
  p.kv_len = kv_len;
  p.table_width = table_width;
  p.heads = heads;
  p.kv_heads = kv_heads;
  p.page_size = page_size;
  p.window = window;
  p.skip_single = skip_single;
  p.scale_log2 = scale * LOG2E;
  p.error = error;
  cudaStream_t s = (cudaStream_t)stream;
  p.work_index = work_index;
  const int working_seqs = work_index != nullptr ? work_count : (skip_single && singles > 0 && singles < seqs ? seqs - singles : seqs);
  if (d == 64) return launch<64>(p, qkv, keys, values, tokens, pages, seqs, working_seqs, max_q_len, max_kv_len, form, chosen, s);
  return launch<128>(p, qkv, keys, values, tokens, pages, seqs, working_seqs, max_q_len, max_kv_len, form, chosen, s);
}

PAE_DEFINE_LAST_ERROR()
