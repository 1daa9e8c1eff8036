// Matrix products out[M, N] = x[M, K] . w[N, K]^T (+ bias[N]) (+ residual[M, N]) of the true 32-bit path, and of whatever the bfloat16
// path's tensor-core kernels refuse. No TF32 and no bfloat16 staging anywhere.
//
// The general kernel (CUDA cores) takes every size and every mix of element types: any M, N, K, no alignment
// needed, bfloat16 or float32 activations, weights and outputs. Float32 products have kernels of their own (second
// half of this file), from three tokens on with the tensor cores' double-precision instruction.
//
// Weights are [out, in] row-major as the checkpoint stores them, which is what
// x . w^T reads (engine/model.py:303-320 of the reference calls F.linear on the same
// layout). Every output element sums its K products in the same order whatever M is, so
// a token's result does not depend on what else is in the batch. When activations, weights
// and output are all float32 (in the general kernel if K is not a multiple of 4 or an
// operand is not 16-byte aligned) the K products are summed in double and rounded once: a
// sequential float32 sum over a long K loses several bits against what a float32 result
// can hold, and a model whose layers cancel (a recurrent state read out by a near-orthogonal
// vector) amplifies exactly that.
#include "common.cuh"

using namespace pae;

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;  // 256 threads, 4x4 outputs each

// The activations a product can apply to its own output (the sum, rounded to the output's type first):
// 1 exact GELU, 2 tanh GELU, 3 the square of max(z, 0).
__device__ __forceinline__ float activation_of(float z, int kind) {
  if (kind == 1) return 0.5f * z * (1.f + erff(z * 0.70710678118654752440f));
  if (kind == 3) { z = fmaxf(z, 0.f); return z * z; }
  return 0.5f * z * (1.f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
}

template <typename TA, typename TW, typename TO, typename TAcc>
__global__ void __launch_bounds__(256) gemm_simt_kernel(TO* __restrict__ out, const TA* __restrict__ x,
                                                        const TW* __restrict__ w, const float* __restrict__ bias,
                                                        const TO* __restrict__ residual, int M, int N, int K,
                                                        const int* __restrict__ group_tiles, int tile, int activation) {
  dependent_launch_prologue();
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (group_tiles != nullptr) {
    // Grouped: w is one [N, K] matrix per group; the rows of tile j (of `tile` rows, a multiple of BM)
    // multiply matrix group_tiles[2 j], and only the tile's first group_tiles[2 j + 1] rows count.
    const int j = m0 / tile;
    if (j >= group_tiles[2 * (M / tile)]) return;          // the table's last entry: how many tiles are in use
    const int g = group_tiles[2 * j];
    w += (size_t)g * N * K;
    M = min(M, j * tile + group_tiles[2 * j + 1]);
    if (m0 >= M) return;
  }
  const int tx = tid % 16, ty = tid / 16;      // outputs rows ty*4.., cols tx*4..
  const int load_row = tid / 4, load_k = (tid % 4) * 4;

  TAcc acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = (TAcc)0;

  for (int k0 = 0; k0 < K; k0 += BK) {
    {
      const int m = m0 + load_row;
      const TA* src = x + (size_t)m * K + k0 + load_k;
#pragma unroll
      for (int j = 0; j < 4; ++j) xs[load_k + j][load_row] = (m < M && k0 + load_k + j < K) ? to_float(src[j]) : 0.f;
      const int n = n0 + load_row;
      const TW* wsrc = w + (size_t)n * K + k0 + load_k;
#pragma unroll
      for (int j = 0; j < 4; ++j) ws[load_k + j][load_row] = (n < N && k0 + load_k + j < K) ? to_float(wsrc[j]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      TAcc a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = (TAcc)xs[k][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = (TAcc)ws[k][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n >= N) continue;
      TAcc v = acc[i][j];
      if (bias != nullptr) v += (TAcc)bias[n];
      if (activation != 0) v = (TAcc)activation_of(to_float(from_float<TO>((float)v)), activation);
      if (residual != nullptr) v += (TAcc)to_float(residual[(size_t)m * N + n]);
      out[(size_t)m * N + n] = from_float<TO>((float)v);
    }
  }
}

template <typename TA, typename TW, typename TO, typename TAcc = float>
int launch(void* out, const void* x, const void* w, const float* bias, const void* residual, int M, int N, int K,
           cudaStream_t s, const int* group_tiles = nullptr, int tile = 0, int activation = 0) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  launch_kernel(gemm_simt_kernel<TA, TW, TO, TAcc>, grid, 256, 0, s, (TO*)out, (const TA*)x, (const TW*)w, bias, (const TO*)residual, M, N, K,
                group_tiles, tile, activation);
  return check_launch("linear_simt");
}

// ---------------------------------------------------------------------------------------
// The float32 products (activations, weights and output all float32, K a multiple of 4, 16-byte
// aligned operands). K is cut into segments of SEGMENT; a segment's products are added one after the other in
// double, the segments' sums one after the other to the total, bias and residual to that, and the result is rounded
// once. All kernels below keep exactly this order, whatever M is and however K is shared out (the tensor
// cores' double-precision instruction adds its four products like four fused multiply-adds in a row; a test of
// sums that cancel compares them), so a token's result does not depend on its batch.
//
// f32_lane_kernel, one or two tokens: a lane owns a weight row in a segment, a warp two segments of 16 rows (of 32
// rows and one segment, N = 1,536 made 48 blocks), plain double multiply-adds. f32_few_kernel, 3 to 32 tokens: the same split, with mma.m8n8k4.f64 (eight weight rows x eight
// tokens; operands widened from float32, which is exact). Both are bound by the weights' bytes at few tokens and
// by the chain of a segment's sums; weights pass through a ring of cp.async stages per warp (32 k; rows 144 bytes
// apart, so that a fragment's reads meet no bank twice).
// f32_tile_kernel, more tokens: bound by the double products. 64 tokens x 64 weight rows a block, 32 x 32 a warp. While
// the tiles are fewer than half of the SMs the segments are shared out over blocks, each of which leaves its
// segments' sums in planes of double that f32_planes_kernel adds up.
//
// Measured, us, [17,920, 1,536] and [1,536, 8,960] weights: 1 token 22.9 and 15.8 (16.8 and 8.4 at the copy bandwidth;
// 24.0 and 26.0 with 32 rows a block, the eight-token kernel 36 and 40), 8 tokens 37 and 43 (63 and 78 with plain multiply-adds, whose operands meet the shared memory's
// bandwidth), 60 tokens 153 and 75 (313 and 171), 256 tokens 454 and 475 (1,232 and 1,496): 31 and 15 of 37 TFLOP/s. (The second has 96
// tiles, more than half of the SMs, so that K is not shared out.)
// ---------------------------------------------------------------------------------------
constexpr int SEGMENT = 128;
constexpr int CHUNK = 32;                   // k of a stage
constexpr int CHUNKS_PER_SEGMENT = SEGMENT / CHUNK;
constexpr int PITCH = CHUNK + 4;            // floats between the rows of a stage

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool valid) {
  const int bytes = valid ? 16 : 0;         // 0: the destination is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// c[8 x 8] += a[8 x 4] b[4 x 8]: this lane holds a[lane / 4][lane % 4], b[lane % 4][lane / 4] and
// c[lane / 4][2 (lane % 4)], c[lane / 4][2 (lane % 4) + 1].
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

namespace few {
constexpr int WARPS = 8;
constexpr int ROWS = 32;                    // weight rows of a block

template <int T>                            // groups of eight tokens
struct Layout {
  static constexpr int TOKENS = 8 * T;
  static constexpr int STAGES = T == 1 ? 4 : (T == 2 ? 3 : 2);  // what eight warps' rings leave room for
  static constexpr int STAGE_FLOATS = (ROWS + TOKENS) * PITCH;
  static constexpr int RING_BYTES = STAGES * STAGE_FLOATS * 4;
  static constexpr int PART_BYTES = TOKENS * ROWS * 8;          // a warp's segment sums, [token][row]
  static size_t bytes(int warps) { return (size_t)warps * (RING_BYTES + PART_BYTES); }
};
}  // namespace few

template <int T>
__global__ void __launch_bounds__(32 * few::WARPS) f32_few_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                                  const float* __restrict__ w, const float* __restrict__ bias,
                                                                  const float* __restrict__ residual, int M, int N, int K) {
  using L = few::Layout<T>;
  constexpr int STAGES = L::STAGES, TOKENS = L::TOKENS, ROWS = few::ROWS;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ring = (float*)(smem + (size_t)warp * L::RING_BYTES);
  double* parts = (double*)(smem + (size_t)warps * L::RING_BYTES);
  const int n0 = blockIdx.x * ROWS;
  const int segments = (K + SEGMENT - 1) / SEGMENT;
  // This warp's segments are warp, warp + warps, ...; its chunks run through all of them in order.
  const int mine = warp < segments ? (segments - warp + warps - 1) / warps : 0;
  // The last segment may be short: its chunks behind K are left out.
  const int chunks = mine * CHUNKS_PER_SEGMENT -
                     (mine > 0 && warp + (mine - 1) * warps == segments - 1 ? (segments * SEGMENT - K) / CHUNK : 0);
  auto chunk_k = [&](int c) { return (warp + (c / CHUNKS_PER_SEGMENT) * warps) * SEGMENT + (c % CHUNKS_PER_SEGMENT) * CHUNK; };
  const uint32_t ring_address = (uint32_t)__cvta_generic_to_shared(ring);
  auto fetch = [&](int c) {
    if (c < chunks) {
      const int k = chunk_k(c) + (lane & 7) * 4;                // eight lanes bring a row's 32 k
      const uint32_t dst = ring_address + ((c % STAGES) * L::STAGE_FLOATS + (lane >> 3) * PITCH + (lane & 7) * 4) * 4;
#pragma unroll
      for (int i = 0; i < ROWS / 4; ++i) {
        const int n = n0 + i * 4 + (lane >> 3);
        const bool valid = n < N && k < K;
        copy16(dst + i * 4 * PITCH * 4, valid ? w + (size_t)n * K + k : w, valid);
      }
#pragma unroll
      for (int i = 0; i < TOKENS / 4; ++i) {
        const int m = i * 4 + (lane >> 3);
        const bool valid = m < M && k < K;
        copy16(dst + (ROWS + i * 4) * PITCH * 4, valid ? x + (size_t)m * K + k : x, valid);
      }
    }
    copy_commit();                            // one group per chunk, empty ones too: the waits count groups
  };
  dependent_launch_prologue();
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) fetch(c);

  // The outputs that this thread adds up, a round's segments in their order.
  constexpr int OUTPUTS = TOKENS * ROWS / 32;                  // when one warp runs; an eighth when eight do
  double total[OUTPUTS];
#pragma unroll
  for (int i = 0; i < OUTPUTS; ++i) total[i] = 0.0;
  const int rounds = (segments + warps - 1) / warps;
  int c = 0;
  for (int round = 0; round < rounds; ++round) {
    if (round < mine) {
      double acc[ROWS / 8][T][2];
#pragma unroll
      for (int i = 0; i < ROWS / 8; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
      for (int i = 0; i < CHUNKS_PER_SEGMENT && c < chunks; ++i, ++c) {
        copy_wait<STAGES - 2>();
        __syncwarp();                         // every lane's copies of this chunk are there, and all are done with the chunk before
        fetch(c + STAGES - 1);
        const float* from = ring + (c % STAGES) * L::STAGE_FLOATS + (lane >> 2) * PITCH + (lane & 3);
#pragma unroll
        for (int k = 0; k < CHUNK; k += 4) {
          double a[ROWS / 8], b[T];
#pragma unroll
          for (int r = 0; r < ROWS / 8; ++r) a[r] = (double)from[r * 8 * PITCH + k];
#pragma unroll
          for (int j = 0; j < T; ++j) b[j] = (double)from[(ROWS + j * 8) * PITCH + k];
#pragma unroll
          for (int r = 0; r < ROWS / 8; ++r)
#pragma unroll
            for (int j = 0; j < T; ++j) mma_f64(acc[r][j], a[r], b[j]);
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS / 8; ++r)
#pragma unroll
        for (int j = 0; j < T; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            parts[(warp * TOKENS + j * 8 + 2 * (lane & 3) + e) * ROWS + r * 8 + (lane >> 2)] = acc[r][j][e];
    }
    __syncthreads();
    const int present = min(warps, segments - round * warps);
#pragma unroll
    for (int i = 0; i < OUTPUTS; ++i) {
      const int o = threadIdx.x + i * blockDim.x;
      if (o < M * ROWS)
        for (int s = 0; s < present; ++s) total[i] += parts[s * TOKENS * ROWS + o];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < OUTPUTS; ++i) {
    const int o = threadIdx.x + i * blockDim.x;
    const int m = o / ROWS, n = n0 + o % ROWS;
    if (m >= M || n >= N) continue;
    double v = total[i];
    if (bias != nullptr) v += (double)bias[n];
    if (residual != nullptr) v += (double)residual[(size_t)m * N + n];
    out[(size_t)m * N + n] = (float)v;
  }
}

template <int T>
int launch_few(float* out, const float* x, const float* w, const float* bias, const float* residual, int M, int N, int K, cudaStream_t s) {
  using L = few::Layout<T>;
  const int segments = (K + SEGMENT - 1) / SEGMENT;
  const int warps = segments < few::WARPS ? segments : few::WARPS;
  static DevicesSet raised;
  if (int err = raise_shared_memory(raised, f32_few_kernel<T>, L::bytes(few::WARPS), "linear_f32")) return err;
  launch_kernel(f32_few_kernel<T>, dim3((N + few::ROWS - 1) / few::ROWS), 32 * warps, L::bytes(warps), s, out, x, w, bias, residual, M, N, K);
  return check_launch("linear_f32");
}

namespace lane_rows {
constexpr int WARPS = 16;
constexpr int ROWS = 16;                    // weight rows of a block
constexpr int STAGES = 2;

template <int MT>
struct Layout {
  static constexpr int STAGE_FLOATS = 2 * (ROWS * PITCH + MT * CHUNK);
  static constexpr int WIDE = MT * CHUNK + 2;                   // doubles of a segment's token values (its neighbour starts on other banks)
  static constexpr int WARP_BYTES = STAGES * STAGE_FLOATS * 4 + 2 * WIDE * 8;
  static constexpr int PART_BYTES = 2 * MT * ROWS * 8;          // a warp's two segment sums, [segment][token][row]
  static size_t bytes(int warps) { return (size_t)warps * (WARP_BYTES + PART_BYTES); }
};
}  // namespace lane_rows

// A warp takes two neighbouring segments of 16 rows: lane l has row l % 16 of segment l / 16.
template <int MT>
__global__ void __launch_bounds__(32 * lane_rows::WARPS) f32_lane_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                                         const float* __restrict__ w, const float* __restrict__ bias,
                                                                         const float* __restrict__ residual, int M, int N, int K) {
  using L = lane_rows::Layout<MT>;
  constexpr int STAGES = lane_rows::STAGES, ROWS = lane_rows::ROWS;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = lane >> 4, my_row = lane & 15;
  float* ring = (float*)(smem + (size_t)warp * L::WARP_BYTES);
  double* wide = (double*)(ring + STAGES * L::STAGE_FLOATS);
  double* parts = (double*)(smem + (size_t)warps * L::WARP_BYTES);
  const int n0 = blockIdx.x * ROWS;
  const int segments = (K + SEGMENT - 1) / SEGMENT, pairs = (segments + 1) / 2;
  // This warp's pairs of segments are warp, warp + warps, ...; its chunks run through all of them in order.
  const int mine = warp < pairs ? (pairs - warp + warps - 1) / warps : 0;
  const bool owns_last = mine > 0 && warp + (mine - 1) * warps == pairs - 1;
  // A lone last segment may be short: its chunks behind K are left out.
  const int chunks = mine * CHUNKS_PER_SEGMENT - (owns_last && (segments & 1) ? (segments * SEGMENT - K) / CHUNK : 0);
  auto chunk_k = [&](int c, int h) {
    return (2 * (warp + (c / CHUNKS_PER_SEGMENT) * warps) + h) * SEGMENT + (c % CHUNKS_PER_SEGMENT) * CHUNK;
  };
  const uint32_t ring_address = (uint32_t)__cvta_generic_to_shared(ring);
  auto fetch = [&](int c) {
    if (c < chunks) {
      const int piece = (lane & 7) * 4;       // eight lanes bring a row's 32 k
      const uint32_t stage = ring_address + (c % STAGES) * L::STAGE_FLOATS * 4;
#pragma unroll
      for (int i = 0; i < 2 * ROWS / 4; ++i) {
        const int at = i * 4 + (lane >> 3), n = n0 + at % ROWS, k = chunk_k(c, at / ROWS) + piece;
        const bool valid = n < N && k < K;
        copy16(stage + (at * PITCH + piece) * 4, valid ? w + (size_t)n * K + k : w, valid);
      }
      const int at = lane >> 3, m = at % MT, k = chunk_k(c, at / MT) + piece;
      const bool valid = m < M && k < K;
      if (at < 2 * MT) copy16(stage + (2 * ROWS * PITCH + at * CHUNK + piece) * 4, valid ? x + (size_t)m * K + k : x, valid);
    }
    copy_commit();
  };
  dependent_launch_prologue();
#pragma unroll
  for (int c = 0; c < STAGES; ++c) fetch(c);
  double total = 0.0;                         // of this lane's output, in the first warp: row lane % 16 of token lane / 16
  const int rounds = (pairs + warps - 1) / warps;
  int c = 0;
  for (int round = 0; round < rounds; ++round) {
    if (round < mine) {
      double acc[MT];
#pragma unroll
      for (int m = 0; m < MT; ++m) acc[m] = 0.0;
      for (int i = 0; i < CHUNKS_PER_SEGMENT && c < chunks; ++i, ++c) {
        copy_wait<STAGES - 1>();
        __syncwarp();
        const float* stage = ring + (c % STAGES) * L::STAGE_FLOATS;
        float4 w4[CHUNK / 4];                 // the chunk leaves its stage at once, which is then filled again
#pragma unroll
        for (int q = 0; q < CHUNK / 4; ++q) w4[q] = *(const float4*)(stage + lane * PITCH + 4 * q);
#pragma unroll
        for (int m = 0; m < 2 * MT; ++m) wide[(m / MT) * L::WIDE + (m % MT) * CHUNK + lane] = (double)stage[2 * ROWS * PITCH + m * CHUNK + lane];
        __syncwarp();
        fetch(c + STAGES);
        const double* mine_wide = wide + half * L::WIDE;
#pragma unroll
        for (int q = 0; q < CHUNK / 4; ++q) {
          const double w0 = (double)w4[q].x, w1 = (double)w4[q].y, w2 = (double)w4[q].z, w3 = (double)w4[q].w;
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            const double2 x01 = *(const double2*)(mine_wide + m * CHUNK + 4 * q), x23 = *(const double2*)(mine_wide + m * CHUNK + 4 * q + 2);
            acc[m] = fma(x23.y, w3, fma(x23.x, w2, fma(x01.y, w1, fma(x01.x, w0, acc[m]))));
          }
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m) parts[((2 * warp + half) * MT + m) * ROWS + my_row] = acc[m];
    }
    __syncthreads();
    // The first warp adds a round's segments up in their order.
    if (warp == 0 && half < MT) {
      const int present = min(2 * warps, segments - 2 * round * warps);
#pragma unroll 8
      for (int s = 0; s < present; ++s) total += parts[(s * MT + half) * ROWS + my_row];
    }
    if (round + 1 < rounds) __syncthreads();
  }
  const int n = n0 + my_row, m = half;
  if (warp != 0 || n >= N || m >= M || m >= MT) return;
  if (bias != nullptr) total += (double)bias[n];
  if (residual != nullptr) total += (double)residual[(size_t)m * N + n];
  out[(size_t)m * N + n] = (float)total;
}

template <int MT>
int launch_lane(float* out, const float* x, const float* w, const float* bias, const float* residual, int M, int N, int K, cudaStream_t s) {
  using L = lane_rows::Layout<MT>;
  const int pairs = ((K + SEGMENT - 1) / SEGMENT + 1) / 2;
  const int warps = pairs < lane_rows::WARPS ? pairs : lane_rows::WARPS;
  static DevicesSet raised;
  if (int err = raise_shared_memory(raised, f32_lane_kernel<MT>, L::bytes(lane_rows::WARPS), "linear_f32")) return err;
  launch_kernel(f32_lane_kernel<MT>, dim3((N + lane_rows::ROWS - 1) / lane_rows::ROWS), 32 * warps, L::bytes(warps), s, out, x, w, bias, residual, M, N, K);
  return check_launch("linear_f32");
}

namespace tiled {
constexpr int TILE = 64;                    // tokens and weight rows of a block
constexpr int STAGES = 3;
constexpr int STAGE_FLOATS = 2 * TILE * PITCH;
constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_FLOATS * 4;
}  // namespace tiled

// planes (double [segments, M, N]): null, or where this block's segments' sums go instead of the output.
__global__ void __launch_bounds__(128, 3) f32_tile_kernel(float* __restrict__ out, double* __restrict__ planes, const float* __restrict__ x,
                                                       const float* __restrict__ w, const float* __restrict__ bias,
                                                       const float* __restrict__ residual, int M, int N, int K, int segments_per_block) {
  constexpr int TILE = tiled::TILE, STAGES = tiled::STAGES;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
  const int segments = (K + SEGMENT - 1) / SEGMENT;
  const int first_segment = blockIdx.z * segments_per_block, end_segment = min(segments, first_segment + segments_per_block);
  const int k_begin = first_segment * SEGMENT, k_end = min(K, end_segment * SEGMENT);
  const int chunks = (k_end - k_begin + CHUNK - 1) / CHUNK;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem);
  auto fetch = [&](int c) {
    if (c < chunks) {
      const int k = k_begin + c * CHUNK + (tid & 7) * 4;
      const uint32_t dst = ring + ((c % STAGES) * tiled::STAGE_FLOATS + (tid >> 3) * PITCH + (tid & 7) * 4) * 4;
#pragma unroll
      for (int i = 0; i < TILE / 16; ++i) {
        const int n = n0 + i * 16 + (tid >> 3), m = m0 + i * 16 + (tid >> 3);
        const bool w_valid = n < N && k < k_end, x_valid = m < M && k < k_end;
        copy16(dst + i * 16 * PITCH * 4, w_valid ? w + (size_t)n * K + k : w, w_valid);
        copy16(dst + (TILE + i * 16) * PITCH * 4, x_valid ? x + (size_t)m * K + k : x, x_valid);
      }
    }
    copy_commit();
  };
  dependent_launch_prologue();
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) fetch(c);
  const int row0 = (warp & 1) * 32, token0 = (warp >> 1) * 32;      // this warp's quarter of the tile
  double acc[4][4][2], total[4][4][2];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[r][j][0] = acc[r][j][1] = total[r][j][0] = total[r][j][1] = 0.0;
  for (int c = 0; c < chunks; ++c) {
    copy_wait<STAGES - 2>();
    __syncthreads();                          // this chunk is there, and all are done with the chunk before
    fetch(c + STAGES - 1);
    const float* from = (const float*)smem + (c % STAGES) * tiled::STAGE_FLOATS + (lane >> 2) * PITCH + (lane & 3);
#pragma unroll
    for (int k = 0; k < CHUNK; k += 4) {
      double a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = (double)from[(row0 + r * 8) * PITCH + k];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = (double)from[(TILE + token0 + j * 8) * PITCH + k];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_f64(acc[r][j], a[r], b[j]);
    }
    if ((c + 1) % CHUNKS_PER_SEGMENT == 0 || c + 1 == chunks) {     // a segment ends
      double* plane = planes != nullptr ? planes + (size_t)(first_segment + c / CHUNKS_PER_SEGMENT) * M * N : nullptr;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (plane != nullptr) {
              const int n = n0 + row0 + r * 8 + (lane >> 2), m = m0 + token0 + j * 8 + 2 * (lane & 3) + e;
              if (m < M && n < N) plane[(size_t)m * N + n] = acc[r][j][e];
            }
            total[r][j][e] += acc[r][j][e];
            acc[r][j][e] = 0.0;
          }
    }
  }
  if (planes != nullptr) return;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int n = n0 + row0 + r * 8 + (lane >> 2);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int m = m0 + token0 + j * 8 + 2 * (lane & 3) + e;
        if (m >= M || n >= N) continue;
        double v = total[r][j][e];
        if (bias != nullptr) v += (double)bias[n];
        if (residual != nullptr) v += (double)residual[(size_t)m * N + n];
        out[(size_t)m * N + n] = (float)v;
      }
  }
}

// out[M, N] (rows ld_out apart) = the planes' sum in their order + bias + residual (rows ld_out apart).
__global__ void __launch_bounds__(256) f32_planes_kernel(float* __restrict__ out, const double* __restrict__ planes,
                                                         const float* __restrict__ bias, const float* __restrict__ residual,
                                                         int segments, int M, int N, int ld_out) {
  dependent_launch_prologue();
  const long long count = (long long)M * N, i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= count) return;
  double v = 0.0;
#pragma unroll 8
  for (int s = 0; s < segments; ++s) v += planes[(size_t)s * count + i];
  const int m = (int)i / N, n = (int)i - m * N;            // a slice has at most half the SMs' tiles
  const size_t at = (size_t)m * ld_out + n;
  if (bias != nullptr) v += (double)bias[n];
  if (residual != nullptr) v += (double)residual[at];
  out[at] = (float)v;
}

int sm_count() {
  static const int count = [] {
    int device = 0, n = 148;
    if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
    return n;
  }();
  return count;
}

}  // namespace

constexpr int F32_FEW_TOKENS = 32;
// The planes of a launch hold a double per output and segment, which is as much as the weights are at 64 tokens: they are bounded by cutting
// the output into slices of whole tiles, one after the other through the same scratch. 96 MB hold 19 tiles of the
// longest K in use (18,944).
constexpr long long F32_SCRATCH_BYTES = 96LL << 20;

namespace {

struct Slices {
  int m, n;                  // tokens and weight rows of a slice (whole tiles); 0: K is not shared out over blocks
};

// K is shared out when the tiles would leave more than half of the SMs idle, and a single tile's segments fit the scratch.
Slices f32_slices(int M, int N, int K) {
  constexpr int TILE = tiled::TILE;
  const int segments = (K + SEGMENT - 1) / SEGMENT;
  if (M <= F32_FEW_TOKENS || segments < 2) return {0, 0};
  const int tiles_m = (M + TILE - 1) / TILE, tiles_n = (N + TILE - 1) / TILE;
  if ((long long)tiles_m * tiles_n * 2 > sm_count()) return {0, 0};
  const int most = (int)(F32_SCRATCH_BYTES / ((long long)segments * TILE * TILE * 8));      // tiles of a slice
  if (most < 1) return {0, 0};
  auto equal = [](int tiles, int at_most) { const int cuts = (tiles + at_most - 1) / at_most; return (tiles + cuts - 1) / cuts; };
  const int slice_m = tiles_m <= most ? tiles_m : equal(tiles_m, most);
  const int slice_n = equal(tiles_n, most / slice_m);
  return {slice_m * TILE < M ? slice_m * TILE : M, slice_n * TILE < N ? slice_n * TILE : N};
}

}  // namespace

// How many doubles `pae_linear_f32` needs as scratch (0: none), at most 96 MB of them.
PAE_EXPORT long long pae_linear_f32_scratch(int M, int N, int K) {
  const Slices slice = f32_slices(M, N, K);
  return (long long)((K + SEGMENT - 1) / SEGMENT) * slice.m * slice.n;
}

// How many kernels it launches.
PAE_EXPORT int pae_linear_f32_launches(int M, int N, int K) {
  const Slices slice = f32_slices(M, N, K);
  return slice.m == 0 ? 1 : 2 * ((M + slice.m - 1) / slice.m) * ((N + slice.n - 1) / slice.n);
}

// out[M, N] = x[M, K] . w[N, K]^T (+ bias[N]) (+ residual[M, N]), all float32, sums in double; K a multiple of 4,
// x and w on 16-byte boundaries. planes: pae_linear_f32_scratch(M, N, K) doubles of scratch, or null when that is 0.
PAE_EXPORT int pae_linear_f32(float* out, const float* x, const float* w, const float* bias, const float* residual, int M, int N, int K,
                              double* planes, void* stream) {
  if (M == 0 || N == 0) return 0;
  if (K % 4 || K < 4) return fail(2, "linear_f32: K = %d is not a positive multiple of 4", K);
  if (((uintptr_t)x | (uintptr_t)w) & 15) return fail(2, "linear_f32: an operand does not start on a 16-byte boundary");
  cudaStream_t s = (cudaStream_t)stream;
  if (M <= 2) return M == 1 ? launch_lane<1>(out, x, w, bias, residual, M, N, K, s) : launch_lane<2>(out, x, w, bias, residual, M, N, K, s);
  if (M <= 8) return launch_few<1>(out, x, w, bias, residual, M, N, K, s);
  if (M <= 16) return launch_few<2>(out, x, w, bias, residual, M, N, K, s);
  // A single segment is one warp's work there: 32 tokens x 96 x 96 take 11.3 us, the tiles 7.6.
  if (M <= F32_FEW_TOKENS && K > SEGMENT) return launch_few<4>(out, x, w, bias, residual, M, N, K, s);
  const int tiles_m = (M + tiled::TILE - 1) / tiled::TILE, tiles_n = (N + tiled::TILE - 1) / tiled::TILE;
  if (tiles_m > 65535) return fail(3, "linear_f32: %d rows are more than one launch takes", M);
  const int segments = (K + SEGMENT - 1) / SEGMENT;
  const Slices slice = f32_slices(M, N, K);
  if (slice.m > 0 && planes == nullptr) return fail(2, "linear_f32: [%d, %d] x [%d, %d] needs scratch planes", M, K, N, K);
  static DevicesSet raised;
  if (int err = raise_shared_memory(raised, f32_tile_kernel, tiled::SMEM_BYTES, "linear_f32")) return err;
  if (slice.m == 0) {
    launch_kernel(f32_tile_kernel, dim3(tiles_n, tiles_m, 1), 128, tiled::SMEM_BYTES, s, out, nullptr, x, w, bias, residual, M, N, K, segments);
    return check_launch("linear_f32");
  }
  for (int m0 = 0; m0 < M; m0 += slice.m)
    for (int n0 = 0; n0 < N; n0 += slice.n) {
      const int m = slice.m < M - m0 ? slice.m : M - m0, n = slice.n < N - n0 ? slice.n : N - n0;
      const int grid_m = (m + tiled::TILE - 1) / tiled::TILE, grid_n = (n + tiled::TILE - 1) / tiled::TILE;
      int blocks_k = (int)(3LL * sm_count() / ((long long)grid_m * grid_n));
      blocks_k = blocks_k > segments ? segments : blocks_k;
      const int per = (segments + blocks_k - 1) / blocks_k;
      const size_t at = (size_t)m0 * N + n0;
      launch_kernel(f32_tile_kernel, dim3(grid_n, grid_m, (segments + per - 1) / per), 128, tiled::SMEM_BYTES, s, nullptr, planes, x + (size_t)m0 * K,
                    w + (size_t)n0 * K, nullptr, nullptr, m, n, K, per);
      launch_kernel(f32_planes_kernel, dim3((unsigned)(((long long)m * n + 255) / 256)), 256, 0, s, out + at, planes, bias != nullptr ? bias + n0 : nullptr,
                    residual != nullptr ? residual + at : nullptr, segments, m, n, N);
    }
  return check_launch("linear_f32");
}

// x_dtype, w_dtype, out_dtype: 0 float32, 1 bfloat16. bias (float32) and residual
// (out_dtype, may be `out` itself) may be null.
PAE_EXPORT int pae_linear_simt(void* out, const void* x, const void* w, const float* bias, const void* residual,
                               int M, int N, int K, int x_dtype, int w_dtype, int out_dtype, void* stream) {
  if (M == 0 || N == 0) return 0;
  if ((long long)((M + BM - 1) / BM) > 65535) return fail(3, "linear_simt: %d rows are more than one launch takes", M);
  cudaStream_t s = (cudaStream_t)stream;
  using bf = __nv_bfloat16;
  const int key = x_dtype * 100 + w_dtype * 10 + out_dtype;
  switch (key) {
    case 0: return launch<float, float, float, double>(out, x, w, bias, residual, M, N, K, s);
    case 111: return launch<bf, bf, bf>(out, x, w, bias, residual, M, N, K, s);
    case 110: return launch<bf, bf, float>(out, x, w, bias, residual, M, N, K, s);
    case 101: return launch<bf, float, bf>(out, x, w, bias, residual, M, N, K, s);
    case 100: return launch<bf, float, float>(out, x, w, bias, residual, M, N, K, s);
    default:
      return fail(1, "linear_simt: element types x=%d w=%d out=%d are not supported", x_dtype, w_dtype, out_dtype);
  }
}

// The grouped product on the CUDA cores: out[row, n] = act(x[row, k] . w[g(row)][n, k]^T) for rows sorted
// by matrix in tiles of `tile` rows (a multiple of 64); tiles int32 [max_tiles + 1, 2]: each tile's matrix
// and how many of its rows count, and in the last entry how many tiles are in use. x and w of one type (float32: sums in double),
// out of that type or float32.
PAE_EXPORT int pae_linear_grouped_simt(void* out, const void* x, const void* w, const int* tiles, int max_tiles, int tile, int n, int k,
                                       int x_dtype, int out_dtype, int activation, void* stream) {
  if (max_tiles == 0 || n == 0) return 0;
  if (tile < BM || tile % BM) return fail(2, "linear_grouped_simt: tiles of %d rows are not a multiple of %d", tile, BM);
  const long long rows = (long long)max_tiles * tile;
  if (rows / BM > 65535) return fail(3, "linear_grouped_simt: %lld rows are more than one launch takes", rows);
  cudaStream_t s = (cudaStream_t)stream;
  using bf = __nv_bfloat16;
  const int M = (int)rows;
  switch (x_dtype * 10 + out_dtype) {
    case 0: return launch<float, float, float, double>(out, x, w, nullptr, nullptr, M, n, k, s, tiles, tile, activation);
    case 11: return launch<bf, bf, bf>(out, x, w, nullptr, nullptr, M, n, k, s, tiles, tile, activation);
    case 10: return launch<bf, bf, float>(out, x, w, nullptr, nullptr, M, n, k, s, tiles, tile, activation);
    default: return fail(1, "linear_grouped_simt: element types x=%d out=%d are not supported", x_dtype, out_dtype);
  }
}

PAE_DEFINE_LAST_ERROR()
