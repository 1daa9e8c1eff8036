// Attention over the paged cache on the CUDA cores, for every size: any head size that
// is a multiple of 8 up to 256, any number of heads and kv heads, any page size, with
// or without a window, portions of prompts and single decoded tokens in one launch.
// It is the attention of the true 32-bit path, and in the bfloat16 path it takes what
// the tensor-core kernels refuse.
//
// The reference gathers each request's whole key/value history into a padded buffer,
// repeats kv heads for the query heads and calls a library with a boolean mask
// (engine/attention.py:597-624,46-74). Here a block owns 16 consecutive query tokens of
// one request and one query head, walks that request's pages in place through its block
// table, 32 keys at a time, and keeps a running softmax (max, sum) in float32. The rule
// of engine/attention.py:581-586 is evaluated per score: key j is seen by the query at
// position p when j <= p and j < kv_len, and p - j < window when the layer has one.
// Query head h reads kv head h / (heads / kv_heads).
//
// A query's result depends only on its own keys: the tile a token falls in changes the
// order in which its keys are folded in by at most the tile start, never the values.
#include "common.cuh"

#include <cfloat>

using namespace pae;

namespace {

constexpr int BQ = 16;      // query tokens per block
constexpr int BKEYS = 32;   // keys per iteration
constexpr int THREADS = 128;
constexpr int MAX_D = 256;

template <typename T>
__global__ void __launch_bounds__(THREADS) paged_attention_simt_kernel(
    T* __restrict__ out, const T* __restrict__ qkv, const T* __restrict__ keys, const T* __restrict__ values,
    const int* __restrict__ block_table, int table_width, const int* __restrict__ q_start,
    const int* __restrict__ q_pos0, const int* __restrict__ kv_len, int heads, int kv_heads, int d, int page_size,
    float scale, int window) {
  dependent_launch_prologue();
  extern __shared__ float smem[];
  const int b = blockIdx.z, h = blockIdx.y, tile = blockIdx.x;
  const int first_token = q_start[b];
  const int q_count = q_start[b + 1] - first_token;
  if (tile * BQ >= q_count) return;
  const int p0 = q_pos0[b] + tile * BQ;                // position of the tile's first query
  const int rows = min(BQ, q_count - tile * BQ);
  const int kv_end = min(kv_len[b], p0 + rows);         // keys past the last query are never seen
  const int kv_begin = window > 0 ? max(0, p0 - window + 1) : 0;
  const int g = h / (heads / kv_heads);
  const int qkv_width = (heads + 2 * kv_heads) * d;

  const int dpad = d + 1;
  float* qs = smem;                        // [BQ][d + 1]
  float* ks = qs + BQ * dpad;              // [BKEYS][d + 1]
  float* vs = ks + BKEYS * dpad;           // [BKEYS][d]
  float* ps = vs + BKEYS * d;              // [BQ][BKEYS + 1]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid >> 3;                  // query row of this thread, 0..15
  const int cg = tid & 7;                  // column group: keys cg + 8 i, dims cg + 8 i

  for (int i = tid; i < BQ * d; i += THREADS) {
    const int row = i / d, k = i - row * d;
    qs[row * dpad + k] = row < rows ? to_float(qkv[(size_t)(first_token + tile * BQ + row) * qkv_width + h * d + k]) : 0.f;
  }

  float acc[MAX_D / 8];
#pragma unroll
  for (int i = 0; i < MAX_D / 8; ++i) acc[i] = 0.f;
  float row_max = -FLT_MAX, row_sum = 0.f;
  const int my_pos = p0 + r;
  const int nd = d >> 3;
  const int* table = block_table + (size_t)b * table_width;

  for (int base = kv_begin; base < kv_end; base += BKEYS) {
    __syncthreads();   // the previous iteration's reads of ks, vs, ps are done (and qs is written)
    // Each warp brings 8 of the 32 keys; lanes run along the head dimension.
    for (int c = warp; c < BKEYS; c += THREADS / 32) {
      const int j = base + c;
      if (j < kv_end) {
        const int page = checked_page(table[checked_table_index(j / page_size, table_width)]);
        const size_t at = (((size_t)page * kv_heads + g) * page_size + (j % page_size)) * d;
        for (int k = lane; k < d; k += 32) {
          ks[c * dpad + k] = to_float(keys[at + k]);
          vs[c * d + k] = to_float(values[at + k]);
        }
      } else {
        for (int k = lane; k < d; k += 32) {
          ks[c * dpad + k] = 0.f;
          vs[c * d + k] = 0.f;
        }
      }
    }
    __syncthreads();

    float s[BKEYS / 8];
    float tile_max = -FLT_MAX;
#pragma unroll
    for (int i = 0; i < BKEYS / 8; ++i) {
      const int c = cg + 8 * i;
      const int j = base + c;
      float dot = 0.f;
      for (int k = 0; k < d; ++k) dot = fmaf(qs[r * dpad + k], ks[c * dpad + k], dot);
      const bool seen = r < rows && j < kv_end && j <= my_pos && (window <= 0 || my_pos - j < window);
      s[i] = seen ? dot * scale : -FLT_MAX;
      tile_max = fmaxf(tile_max, s[i]);
    }
    // The 8 threads of a row are 8 neighbouring lanes.
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, o));
    const float new_max = fmaxf(row_max, tile_max);
    const float rescale = (row_max == -FLT_MAX) ? 0.f : expf(row_max - new_max);
    float tile_sum = 0.f;
#pragma unroll
    for (int i = 0; i < BKEYS / 8; ++i) {
      const float p = (s[i] == -FLT_MAX) ? 0.f : expf(s[i] - new_max);
      ps[r * (BKEYS + 1) + cg + 8 * i] = p;
      tile_sum += p;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) tile_sum += __shfl_xor_sync(0xffffffffu, tile_sum, o);
    row_sum = row_sum * rescale + tile_sum;
    row_max = new_max;
    __syncwarp();   // ps of a row is written and read by the same 8 lanes of one warp
#pragma unroll
    for (int i = 0; i < MAX_D / 8; ++i) {
      if (i < nd) {
        float v = acc[i] * rescale;
        const int dim = cg + 8 * i;
        for (int c = 0; c < BKEYS; ++c) v = fmaf(ps[r * (BKEYS + 1) + c], vs[c * d + dim], v);
        acc[i] = v;
      }
    }
  }

  if (r < rows) {
    const float inv = row_sum > 0.f ? 1.f / row_sum : 0.f;
    T* to = out + ((size_t)(first_token + tile * BQ + r) * heads + h) * d;
#pragma unroll
    for (int i = 0; i < MAX_D / 8; ++i)
      if (i < nd) to[cg + 8 * i] = from_float<T>(acc[i] * inv);
  }
}

size_t smem_bytes(int d) { return sizeof(float) * (size_t)(BQ * (d + 1) + BKEYS * (d + 1) + BKEYS * d + BQ * (BKEYS + 1)); }

template <typename T>
int launch(void* out, const void* qkv, const void* keys, const void* values, const int* block_table, int table_width,
           const int* q_start, const int* q_pos0, const int* kv_len, int seqs, int max_q_len, int heads, int kv_heads,
           int d, int page_size, float scale, int window, cudaStream_t s) {
  const size_t bytes = smem_bytes(d);
  auto kernel = paged_attention_simt_kernel<T>;
  static DevicesSet raised;     // per element type: to the most any head size needs
  if (bytes > 48 * 1024)
    if (int err = raise_shared_memory(raised, kernel, smem_bytes(MAX_D), "paged_attention_simt")) return err;
  dim3 grid((max_q_len + BQ - 1) / BQ, heads, seqs);
  launch_kernel(kernel, grid, THREADS, bytes, s, (T*)out, (const T*)qkv, (const T*)keys, (const T*)values, block_table,
                                      table_width, q_start, q_pos0, kv_len, heads, kv_heads, d, page_size, scale, window);
  return check_launch("paged_attention_simt");
}

// ---------------------------------------------------------------------------------------
// The float32 form for head sizes 32, 64 and 128. A block owns ROWS query tokens of one request and one
// query head; its eight warps take the 16-key tiles of the context in turn (tile number modulo 8, whatever
// the step's shape, so a query's result depends on its own keys only). A lane holds D / 32 dimensions:
// a warp asks for the 16 keys and the 16 values of a tile at once, straight into registers, forms the lanes' parts
// of the 16 scores and adds them across the lanes in 16 exchanges (each halves what a lane holds), so a score
// ends in a lane of its own. Running maximum, sum and output are a warp's own and are merged in the warps'
// order at the end. Bound by the trips to memory of a warp's tiles, one after the other. The form above walks 32
// keys at a time with one chain of D multiply-adds per score and a block of 16 query rows for a single one:
// one token over 68 keys 56.7 us, over 250 keys 157 (12 heads of 128).
// ---------------------------------------------------------------------------------------
namespace wide {
constexpr int KEYS = 16;                     // keys of a tile

int sm_count() {
  static const int count = [] {
    int device = 0, n = 148;
    if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
    return n;
  }();
  return count;
}

template <int DL>
struct Vec {
  float v[DL];
};
template <int DL>
__device__ __forceinline__ Vec<DL> load(const float* p) {
  Vec<DL> r;
  if constexpr (DL == 4) {
    const float4 t = *(const float4*)p;
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else if constexpr (DL == 2) {
    const float2 t = *(const float2*)p;
    r.v[0] = t.x; r.v[1] = t.y;
  } else {
    r.v[0] = *p;
  }
  return r;
}

// The sum over the lanes of s[k], k = 0..15, ends in the lanes 2 k and 2 k + 1 (lane bits 4..1 are k's bits 3..0).
__device__ __forceinline__ float sum_across(float (&s)[KEYS], int lane) {
#pragma unroll
  for (int width = KEYS / 2; width >= 1; width >>= 1) {
    const bool upper = (lane & (2 * width)) != 0;
#pragma unroll
    for (int i = 0; i < width; ++i) {
      const float give = upper ? s[i] : s[i + width];
      const float keep = upper ? s[i + width] : s[i];
      s[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * width);
    }
  }
  return s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1);
}

// This lane's dimensions of the 16 rows of the cache `place` (one per pair of lanes; -1: zeros).
template <int DL>
__device__ __forceinline__ void fetch(Vec<DL> (&to)[KEYS], const float* from, int place, int lane) {
#pragma unroll
  for (int i = 0; i < KEYS; ++i) {
    const int at = __shfl_sync(0xffffffffu, place, 2 * i);
#pragma unroll
    for (int e = 0; e < DL; ++e) to[i].v[e] = 0.f;
    if (at >= 0) to[i] = load<DL>(from + (size_t)at * (32 * DL) + lane * DL);
  }
}

// PACKED: for launches of more blocks than run at once, in which what counts is how many warps an SM holds (`launch` has the rule and the
// times). A tile's values are asked for when its scores are there, into the keys' registers (128, 80 and 64 a thread at head
// sizes 128, 64 and 32 instead of 223, 128 and 101), the four rows go through a tile's steps side by side, and a block has only as many warps W as
// the longest context has tiles. A row's arithmetic is the same in both, and a warp without a tile adds nothing: the bits are the same.
template <int DL, int ROWS, int W, bool PACKED>
__global__ void __launch_bounds__(32 * W, PACKED ? (DL == 1 ? 32 : DL == 2 ? 24 : 16) / W : 0) paged_attention_f32_kernel(
    float* __restrict__ out, const float* __restrict__ qkv, const float* __restrict__ keys, const float* __restrict__ values,
    const int* __restrict__ block_table, int table_width, const int* __restrict__ q_start, const int* __restrict__ q_pos0,
    const int* __restrict__ kv_len, int heads, int kv_heads, int page_size, float scale, int window) {
  constexpr int D = 32 * DL;
  dependent_launch_prologue();
  __shared__ float merged_max[W][ROWS], merged_sum[W][ROWS];
  __shared__ __align__(16) float merged_out[W][ROWS][D];
  const int b = blockIdx.z, h = blockIdx.y;
  const int first_token = q_start[b];
  const int q_count = q_start[b + 1] - first_token;
  const int row0 = blockIdx.x * ROWS;
  if (row0 >= q_count) return;
  const int rows = min(ROWS, q_count - row0);
  const int p0 = q_pos0[b] + row0;                       // position of the first query
  const int kv_end = min(kv_len[b], p0 + rows);
  const int kv_begin = window > 0 ? max(0, p0 - window + 1) : 0;
  const int g = h / (heads / kv_heads);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int* table = block_table + (size_t)b * table_width;

  Vec<DL> q[ROWS];
  float acc[ROWS][DL], row_max[ROWS], row_sum[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    row_max[r] = -FLT_MAX;
    row_sum[r] = 0.f;
#pragma unroll
    for (int i = 0; i < DL; ++i) acc[r][i] = q[r].v[i] = 0.f;
    if (r < rows) q[r] = load<DL>(qkv + ((size_t)(first_token + row0 + r) * (heads + 2 * kv_heads) + h) * D + lane * DL);
  }
  const int first_tile = kv_begin / KEYS, end_tile = (kv_end + KEYS - 1) / KEYS;
  const int my_key = lane >> 1;                          // the key of a tile whose score ends in this lane
  for (int tile = first_tile + (warp - first_tile % W + W) % W; tile < end_tile; tile += W) {
    const int j = tile * KEYS + my_key;
    int place = -1;                                      // row of the key in the cache, -1: not seen by any query here
    if (j >= kv_begin && j < kv_end) {
      const int page = checked_page(table[checked_table_index(j / page_size, table_width)]);
      place = (page * kv_heads + g) * page_size + j % page_size;
    }
    if constexpr (PACKED) {
      float p[ROWS], tile_max[ROWS], tile_sum[ROWS], rescale[ROWS];
      bool seen[ROWS];
      {
        Vec<DL> k[KEYS];
        fetch<DL>(k, keys, place, lane);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          float s[KEYS];
#pragma unroll
          for (int i = 0; i < KEYS; ++i) {
            s[i] = q[r].v[0] * k[i].v[0];
#pragma unroll
            for (int e = 1; e < DL; ++e) s[i] = fmaf(q[r].v[e], k[i].v[e], s[i]);
          }
          p[r] = sum_across(s, lane);
        }
      }
      Vec<DL> v[KEYS];
      fetch<DL>(v, values, place, lane);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int pos = p0 + r;
        seen[r] = place >= 0 && j <= pos && (window <= 0 || pos - j < window);
        tile_max[r] = p[r] = seen[r] ? p[r] * scale : -FLT_MAX;
      }
#pragma unroll
      for (int o = 16; o > 1; o >>= 1)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) tile_max[r] = fmaxf(tile_max[r], __shfl_xor_sync(0xffffffffu, tile_max[r], o));
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float new_max = fmaxf(row_max[r], tile_max[r]);
        rescale[r] = row_max[r] == -FLT_MAX ? 0.f : expf(row_max[r] - new_max);
        tile_sum[r] = p[r] = seen[r] ? expf(p[r] - new_max) : 0.f;
        row_max[r] = new_max;
#pragma unroll
        for (int e = 0; e < DL; ++e) acc[r][e] *= rescale[r];
      }
#pragma unroll
      for (int o = 16; o > 1; o >>= 1)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) tile_sum[r] += __shfl_xor_sync(0xffffffffu, tile_sum[r], o);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) row_sum[r] = row_sum[r] * rescale[r] + tile_sum[r];
#pragma unroll
      for (int i = 0; i < KEYS; ++i)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float weight = __shfl_sync(0xffffffffu, p[r], 2 * i);
#pragma unroll
          for (int e = 0; e < DL; ++e) acc[r][e] = fmaf(weight, v[i].v[e], acc[r][e]);
        }
      continue;
    }
    Vec<DL> k[KEYS], v[KEYS];
#pragma unroll
    for (int i = 0; i < KEYS; ++i) {
      const int at = __shfl_sync(0xffffffffu, place, 2 * i);
#pragma unroll
      for (int e = 0; e < DL; ++e) k[i].v[e] = v[i].v[e] = 0.f;
      if (at >= 0) {
        k[i] = load<DL>(keys + (size_t)at * D + lane * DL);
        v[i] = load<DL>(values + (size_t)at * D + lane * DL);
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (r >= rows) break;
      float s[KEYS];
#pragma unroll
      for (int i = 0; i < KEYS; ++i) {
        s[i] = q[r].v[0] * k[i].v[0];
#pragma unroll
        for (int e = 1; e < DL; ++e) s[i] = fmaf(q[r].v[e], k[i].v[e], s[i]);
      }
      const float dot = sum_across(s, lane);
      const int pos = p0 + r;
      const bool seen = place >= 0 && j <= pos && (window <= 0 || pos - j < window);
      const float score = seen ? dot * scale : -FLT_MAX;
      float tile_max = score;
#pragma unroll
      for (int o = 16; o > 1; o >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, o));
      const float new_max = fmaxf(row_max[r], tile_max);
      const float rescale = row_max[r] == -FLT_MAX ? 0.f : expf(row_max[r] - new_max);
      const float p = seen ? expf(score - new_max) : 0.f;
      float tile_sum = p;
#pragma unroll
      for (int o = 16; o > 1; o >>= 1) tile_sum += __shfl_xor_sync(0xffffffffu, tile_sum, o);
      row_sum[r] = row_sum[r] * rescale + tile_sum;
      row_max[r] = new_max;
#pragma unroll
      for (int e = 0; e < DL; ++e) acc[r][e] *= rescale;
#pragma unroll
      for (int i = 0; i < KEYS; ++i) {
        const float weight = __shfl_sync(0xffffffffu, p, 2 * i);
#pragma unroll
        for (int e = 0; e < DL; ++e) acc[r][e] = fmaf(weight, v[i].v[e], acc[r][e]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (lane == 0) {
      merged_max[warp][r] = row_max[r];
      merged_sum[warp][r] = row_sum[r];
    }
#pragma unroll
    for (int e = 0; e < DL; ++e) merged_out[warp][r][lane * DL + e] = acc[r][e];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rows * D; i += 32 * W) {
    const int r = i / D, dim = i % D;
    float top = -FLT_MAX;
#pragma unroll
    for (int w = 0; w < W; ++w) top = fmaxf(top, merged_max[w][r]);
    float sum = 0.f, value = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float factor = merged_max[w][r] == -FLT_MAX ? 0.f : expf(merged_max[w][r] - top);
      sum += merged_sum[w][r] * factor;
      value = fmaf(merged_out[w][r][dim], factor, value);
    }
    // A row without keys is 0; a sum that is no number leaves none in its outputs either.
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    out[((size_t)(first_token + row0 + r) * heads + h) * D + dim] = value * inv;
  }
}

template <int DL>
int launch(float* out, const float* qkv, const float* keys, const float* values, const int* block_table, int table_width,
           const int* q_start, const int* q_pos0, const int* kv_len, int seqs, int max_q_len, int max_kv_len, int heads, int kv_heads,
           int page_size, float scale, int window, cudaStream_t s) {
  auto run = [&](auto kernel, int rows, int warps) {
    launch_kernel(kernel, dim3((max_q_len + rows - 1) / rows, heads, seqs), 32 * warps, 0, s, out, qkv, keys, values, block_table, table_width,
                  q_start, q_pos0, kv_len, heads, kv_heads, page_size, scale, window);
  };
  // Packed when there are more blocks than run at once (one on an SM at head size 128, two at 64 and 32) and most of what a query sees are the
  // portions' own keys. Below that its second trip to memory per tile shows (head size 128: one prompt of 16 tokens 6.4 us against 6.2), and
  // few queries after long contexts are the other form's (3 after 4,000 keys 130 against 95 us, 32 requests of 17 after 4,000 at
  // head size 64 2,541 against 1,835). Many short prompts, general form / not packed / packed: 32 prompts of 64 tokens, 28 heads of 128
  // 243 / 389 / 157 us, 16 heads of 32 57 / 98 / 38; 32 of 128 tokens 798 / 928 / 615 and 159 / 208 / 131; one of 2,048, 28 heads 5,039 / 2,776 / 2,182.
  const long long blocks = (long long)((max_q_len + 3) / 4) * heads * seqs, at_once = (DL == 4 ? 1LL : 2LL) * sm_count();
  const int seen = window > 0 && (long long)window + max_q_len < max_kv_len ? window + max_q_len : max_kv_len;
  const bool packed = blocks > at_once && seen <= 4LL * max_q_len;
  if (max_q_len == 1) run(paged_attention_f32_kernel<DL, 1, 8, false>, 1, 8);
  else if (!packed) run(paged_attention_f32_kernel<DL, 4, 8, false>, 4, 8);
  else if (max_kv_len <= KEYS) run(paged_attention_f32_kernel<DL, 4, 1, true>, 4, 1);
  else if (max_kv_len <= 2 * KEYS) run(paged_attention_f32_kernel<DL, 4, 2, true>, 4, 2);
  else if (max_kv_len <= 4 * KEYS) run(paged_attention_f32_kernel<DL, 4, 4, true>, 4, 4);
  else run(paged_attention_f32_kernel<DL, 4, 8, true>, 4, 8);
  return check_launch("paged_attention_simt");
}
}  // namespace wide

}  // namespace

// out [tokens, heads, d]; qkv [tokens, heads + 2 kv_heads, d] (queries are read from it);
// keys, values [pages, kv_heads, page_size, d]; block_table [seqs, table_width].
PAE_EXPORT int pae_paged_attention_simt(void* out, const void* qkv, const void* keys, const void* values,
                                        const int* block_table, int table_width, const int* q_start,
                                        const int* q_pos0, const int* kv_len, int seqs, int max_q_len, int max_kv_len,
                                        int heads, int kv_heads, int d, int page_size, float scale, int window, int dtype,
                                        void* stream) {
  if (seqs == 0 || max_q_len == 0) return 0;
  if (d % 8 || d > MAX_D || d < 8) return fail(2, "paged_attention_simt: head_dim %d is not a multiple of 8 in [8, %d]", d, MAX_D);
  if (kv_heads < 1 || heads % kv_heads) return fail(2, "paged_attention_simt: %d heads over %d kv heads", heads, kv_heads);
  if (heads > 65535 || seqs > 65535) return fail(3, "paged_attention_simt: %d heads x %d requests exceed one launch", heads, seqs);
  if (page_size < 1) return fail(2, "paged_attention_simt: page size %d", page_size);
  cudaStream_t s = (cudaStream_t)stream;
  // The wide form reads 16 bytes at a time: operands of other alignments, and other head sizes, take the general one.
  const bool aligned = (((uintptr_t)qkv | (uintptr_t)keys | (uintptr_t)values) & 15) == 0;
  if (dtype == kF32 && aligned && (d == 32 || d == 64 || d == 128)) {
    const auto launch_wide = d == 32 ? wide::launch<1> : (d == 64 ? wide::launch<2> : wide::launch<4>);
    return launch_wide((float*)out, (const float*)qkv, (const float*)keys, (const float*)values, block_table, table_width, q_start, q_pos0,
                       kv_len, seqs, max_q_len, max_kv_len, heads, kv_heads, page_size, scale, window, s);
  }
  if (dtype == kF32)
    return launch<float>(out, qkv, keys, values, block_table, table_width, q_start, q_pos0, kv_len, seqs, max_q_len, heads, kv_heads, d, page_size, scale, window, s);
  if (dtype == kBF16)
    return launch<__nv_bfloat16>(out, qkv, keys, values, block_table, table_width, q_start, q_pos0, kv_len, seqs, max_q_len, heads, kv_heads, d, page_size, scale, window, s);
  return fail(1, "paged_attention_simt: unknown dtype %d", dtype);
}

PAE_DEFINE_LAST_ERROR()
