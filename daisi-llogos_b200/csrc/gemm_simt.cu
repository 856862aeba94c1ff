// Matrix product on the CUDA cores: out[n][o] = sum_k x[n][k] * w[o][k], float32 accumulation
// by fused multiply-add only (no tensor cores, no reduced-precision mode).  It is the product
// of the true 32-bit path and the fallback for operand types the tensor-core kernel does not
// take.  Any n, o, k.  The reference sends float32 products to cublasSgemm / cublasSgemv
// (Daisi.Llogos.Cuda/CudaBackend.cs:506-519) and has a one-row-per-block GEMV for 16-bit
// weights (kernels/dequant_matmul.cu:593-619).
#include "common.cuh"
#include "kernel_args.h"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

LLG_API const char* llg_last_error() { return g_llg_error; }

namespace {

constexpr int BM = 64;   // rows of x (tokens) per block
constexpr int BN = 64;   // rows of w (output features) per block
constexpr int BK = 16;

template <typename AT, typename WT, typename CT>
__global__ void __launch_bounds__(256) gemm_tn_kernel(const AT* __restrict__ x, const WT* __restrict__ w,
                                                      CT* __restrict__ out, int n, int o, int k, RowScale scale) {
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;     // 16 x 16 threads, each a 4 x 4 sub-tile
  const int n0 = blockIdx.y * BM, o0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < k; k0 += BK) {
    // 64 rows x 16 k = 1024 elements per operand, 4 per thread
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int idx = tid + e * 256;
      const int r = idx >> 4, c = idx & 15;
      const int kk = k0 + c;
      float xv = 0.f, wv = 0.f;
      if (kk < k) {
        if (n0 + r < n) xv = to_f32(x[(long long)(n0 + r) * k + kk]);
        if (o0 + r < o) wv = to_f32(w[(long long)(o0 + r) * k + kk]);
      }
      xs[c][r] = xv;
      ws[c][r] = wv;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < BK; ++c) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[c][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[c][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = n0 + ty * 4 + i;
    if (r >= n) continue;
    const float rs = row_scale_of(scale, r);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = o0 + tx * 4 + j;
      if (c < o) out[(long long)r * o + c] = from_f32<CT>(scale.ss ? acc[i][j] * rs : acc[i][j]);
    }
  }
}

// Two float32 multiply-adds in one instruction, each rounded as fmaf does: a multiprocessor issues scalar multiply-adds at half of
// its pipes' rate (38 TFLOP/s was the most that the scalar form of the tiles below reached, whatever the shape).  A pair holds
// neighbouring k, so a 16-byte load gives two operand pairs and a sum is kept as two, over the even and the odd k.
typedef unsigned long long pair_t;
__device__ __forceinline__ void fma2(pair_t& acc, pair_t a, pair_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float both(pair_t v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); }

// ---- float32 operands with 16-byte rows: two kernels by the count of rows ------------------------------------------
//
// Few rows (a decode step): a stream of the weights.  A warp keeps F features x NR rows of sums; its lanes take
// neighbouring float4s of k, the next group of weights is on its way while this one is used, and the WK warps of a
// feature group share k.  Bound by the weight stream: a float4 of weights is used for NR products of four, and the rows'
// float4s come from the first-level cache once per F features, so F x NR = 32 keeps the CUDA cores and that cache below
// half of what the memory's rate asks of them.  The weights of the first group do not wait for the kernel before.
// 16,384 x 2,048: 23.3 us for one row (5.8 TB/s), 26.7 for three (5.0), 35.9 for eight (3.7; there the cores bound it); 128,256 x
// 2,048 at three rows 163 us (6.4 TB/s).  gemm_tn_kernel, which took these before, pays for 64 rows: 618 us on average over a 1B
// model's products.
// LIVE of the NR rows are there (the rest of the sums stay zero): three rows 27.9 us with the fourth's multiply-adds, 26.7 without, six 35.9
// with those of eight and 33.1.
template <int NR, int F, int LIVE>
__global__ void __launch_bounds__(256, 2) gemv_rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                        float* __restrict__ out, int n, int o, int k, int wk, RowScale scale) {
  constexpr int NV = NR * F;
  static_assert(NV == 8 || NV == 16 || NV == 32, "the sums of a warp are spread over its lanes");
  __shared__ float part[8][NV];
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = 8 / wk, kp = warp % wk, fg = warp / wk;
  const int chunks = (n + NR - 1) / NR;                  // row chunks of one feature group are neighbours: its weights stay in L2
  const int r0 = (blockIdx.x % chunks) * NR;
  const int f0 = ((blockIdx.x / chunks) * groups + fg) * F;
  const int k4 = k >> 2;
  const float4* wp[F];
#pragma unroll
  for (int f = 0; f < F; ++f) wp[f] = reinterpret_cast<const float4*>(w + (long long)min(f0 + f, o - 1) * k);
  float4 wc[F];
  int c = kp * 32 + lane;
  const int step = wk * 32;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int f = 0; f < F; ++f) wc[f] = c < k4 ? __ldcs(wp[f] + c) : zero;
  pdl_wait();                                            // x is the kernel's before, and what that kernel reads may be `out`
  const float4* xp[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) xp[r] = reinterpret_cast<const float4*>(x + (long long)min(r0 + r, n - 1) * k);
  float acc[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) acc[i] = 0.f;
  for (; c < k4; c += step) {
    float4 wn[F];
    const int cn = c + step;
#pragma unroll
    for (int f = 0; f < F; ++f) wn[f] = cn < k4 ? __ldcs(wp[f] + cn) : zero;
#pragma unroll
    for (int r = 0; r < LIVE; ++r) {
      const float4 xv = xp[r][c];
#pragma unroll
      for (int f = 0; f < F; ++f) {
        float& a = acc[r * F + f];
        a = fmaf(xv.x, wc[f].x, a);
        a = fmaf(xv.y, wc[f].y, a);
        a = fmaf(xv.z, wc[f].z, a);
        a = fmaf(xv.w, wc[f].w, a);
      }
    }
#pragma unroll
    for (int f = 0; f < F; ++f) wc[f] = wn[f];
  }
  // the sums of 32 lanes: every exchange halves the values a lane keeps, so that NV - 1 exchanges and log2(32 / NV) more
  // leave value (lane * NV / 32) in the lane
#pragma unroll
  for (int h = NV / 2, off = 16; off > 0; off >>= 1, h >>= 1) {
    if (h >= 1) {
      const bool up = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < NV / 2; ++i) {
        if (i < h) {
          const float give = up ? acc[i] : acc[i + h];
          const float keep = up ? acc[i + h] : acc[i];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
      }
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    }
  }
  constexpr int LANES_PER = 32 / NV;
  if (lane % LANES_PER == 0) part[warp][lane / LANES_PER] = acc[0];
  __syncthreads();
  const int t = threadIdx.x;
  if (t < groups * NV) {
    const int g = t / NV, v = t % NV;
    float sum = 0.f;
    for (int q = 0; q < wk; ++q) sum += part[g * wk + q][v];
    const int r = r0 + v / F, col = ((blockIdx.x / chunks) * groups + g) * F + v % F;
    if (r < n && col < o) out[(long long)r * o + col] = scale.ss ? sum * row_scale_of(scale, r) : sum;
  }
}

// More rows (a prompt step): tiles of up to 64 rows x 128 features, 256 threads with up to 8 x 4 sums each.  Both operands arrive by
// cp.async as they lie in memory, 32 k of a row at a time, in a ring of three stages: a stage is 24 to 27 KB, so that one block a
// multiprocessor already has the bytes in flight that the memory's latency asks for (with the next stage in registers and
// half as much a step a block waited 2 us a step: 100 x 2,048 x 2,048 81.5 us before, 38.6 in tiles of 64 rows, 34.3 in tiles of 56).  Rows are padded to 36 floats: 16-byte
// reads of consecutive rows at one k fall into different banks.  A thread takes four k at a time, 12 reads for 128
// multiply-adds.  From 300 rows on the multiply-add pipes (two thirds busy) and the 16-byte shared reads bound it: 38 TFLOP/s.  Where a shape has few tiles, the blocks of a cluster
// share the tile's k and add their sums through distributed shared memory, in the order of the ranks.
// A tile has 40, 48, 56 or 64 rows (R = 5 to 8 a thread), by the rows that a count of tokens leaves empty: 44 x 16,384 x 2,048 141 us in
// tiles of 64, 96 in tiles of 48 (two blocks a tile); 44 x 2,048 x 8,192 142 us and 97 (tiles of 40, four blocks).
constexpr int TF = 128, TK = 32, TLD = TK + 4, TSTAGES = 3;
__host__ __device__ constexpr int tile_smem(int rows) { return TSTAGES * (rows + TF) * TLD * (int)sizeof(float); }

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(there ? 16 : 0) : "memory");
}

template <int R>
__global__ void __launch_bounds__(256, 2) gemm_tile_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                        float* __restrict__ out, int n, int o, int k, RowScale scale) {
  constexpr int TM = 8 * R;                              // rows of a tile, R a thread
  static_assert(TM * TF * (int)sizeof(float) <= tile_smem(TM) && TM <= 64, "the sums fit where the stages were");
  extern __shared__ __align__(16) float sm[];            // the stages, then the tile's sums
  pdl_launch_dependents();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  // rows ty + 8 i, features tx + 32 j: a warp reads two rows and sixteen features at a time
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (lane & 15) + 16 * (warp & 1), ty = (lane >> 4) + 2 * (warp >> 1);
  const int n0 = blockIdx.y * TM, o0 = (blockIdx.x / ranks) * TF;
  const int steps_all = (k + TK - 1) / TK, per = (steps_all + ranks - 1) / ranks;
  const int s0 = min(rank * per, steps_all), steps = min(s0 + per, steps_all) - s0;
  const int lr = tid >> 3, lc = (tid & 7) * 4;           // copying: 32 rows of 32 k at a time
  auto fetch_w = [&](int s) {
    const int kk = (s0 + s) * TK + lc;
    float* dst = sm + (s % TSTAGES) * (TM + TF) * TLD + TM * TLD + lr * TLD + lc;
#pragma unroll
    for (int i = 0; i < TF / 32; ++i) {
      const int r = o0 + i * 32 + lr;
      const bool there = kk < k && r < o;
      copy16(dst + i * 32 * TLD, w + (there ? (long long)r * k + kk : 0), there);
    }
  };
  auto fetch_x = [&](int s) {
    const int kk = (s0 + s) * TK + lc;
    float* dst = sm + (s % TSTAGES) * (TM + TF) * TLD + lr * TLD + lc;
#pragma unroll
    for (int i = 0; i < (TM + 31) / 32; ++i) {
      const int r = n0 + i * 32 + lr;
      const bool there = kk < k && r < n;
      if (i * 32 + lr < TM) copy16(dst + i * 32 * TLD, x + (there ? (long long)r * k + kk : 0), there);
    }
  };
  auto close = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };
  pair_t sums[R][4];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[i][j] = 0;
  // the first stages' weights do not wait for the kernel before
  for (int s = 0; s < TSTAGES - 1 && s < steps; ++s) fetch_w(s);
  pdl_wait();
  for (int s = 0; s < TSTAGES - 1; ++s) {
    if (s < steps) fetch_x(s);
    close();                                             // the first group holds the weights of both stages: only earlier, never late
  }
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(TSTAGES - 2) : "memory");
    __syncthreads();                                     // stage s is there, and everybody is done with stage s - 1
    if (s + TSTAGES - 1 < steps) {
      fetch_w(s + TSTAGES - 1);
      fetch_x(s + TSTAGES - 1);
    }
    close();
    const float* xs = sm + (s % TSTAGES) * (TM + TF) * TLD + ty * TLD;
    const float* ws = sm + (s % TSTAGES) * (TM + TF) * TLD + (TM + tx) * TLD;
#pragma unroll 2
    for (int kk = 0; kk < TK; kk += 4) {
      ulonglong2 a[R];
#pragma unroll
      for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * 8 * TLD + kk);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(ws + j * 32 * TLD + kk);
#pragma unroll
        for (int i = 0; i < R; ++i) fma2(sums[i][j], a[i].x, f.x);
#pragma unroll
        for (int i = 0; i < R; ++i) fma2(sums[i][j], a[i].y, f.y);
      }
    }
  }
  if (ranks == 1) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = n0 + ty + 8 * i;
      if (r >= n) continue;
      const float rs = scale.ss ? row_scale_of(scale, r) : 1.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = o0 + tx + 32 * j;
        if (c < o) out[(long long)r * o + c] = both(sums[i][j]) * rs;
      }
    }
    return;
  }
  __syncthreads();                                       // the sums go where the last stage was read
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sm[(ty + 8 * i) * TF + tx + 32 * j] = both(sums[i][j]);
  cluster.sync();
  const int rows = TM / ranks;                           // rows of the tile that this block adds up and stores
  for (int i = tid; i < rows * (TF / 4); i += 256) {
    const int row = rank * rows + i / (TF / 4), c = (i % (TF / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < ranks; ++q) {
      const float4 t = *reinterpret_cast<const float4*>(cluster.map_shared_rank(sm, q) + row * TF + c);
      v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
    }
    const int r = n0 + row;
    if (r < n) {
      const float rs = scale.ss ? row_scale_of(scale, r) : 1.0f;
      const float e[4] = {v.x * rs, v.y * rs, v.z * rs, v.w * rs};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (o0 + c + j < o) out[(long long)r * o + o0 + c + j] = e[j];
    }
  }
  cluster.sync();                                        // nobody leaves while its sums may still be read
}

template <int NR, int F, int LIVE = NR>
int run_gemv(const float* x, const float* w, float* out, int n, int o, int k, const RowScale& rs, cudaStream_t stream) {
  // warps that share k: enough for about 32 a multiprocessor, each with a float4 a lane at least
  int wk = 1;
  const long long groups = (o + F - 1) / F, want = 32LL * llg_sm_count();
  while (wk < 8 && groups * ((n + NR - 1) / NR) * wk < want && k / 4 > wk * 32) wk *= 2;
  const long long per = (long long)F * (8 / wk);
  const long long blocks = ((o + per - 1) / per) * ((n + NR - 1) / NR);
  LLG_REQUIRE(blocks <= 2147483647LL, "gemm_simt: too many blocks");
  cudaError_t e = llg_launch(gemv_rows_kernel<NR, F, LIVE>, dim3((unsigned)blocks), dim3(256), 0, stream, x, w, out, n, o, k, wk, rs);
  if (e != cudaSuccess) return llg_fail("gemm_simt: launch: %s", cudaGetErrorString(e));
  return llg_check_launch("gemm_simt");
}

template <int R>
int launch_tile(const float* x, const float* w, float* out, int n, int o, int k, int ranks, const RowScale& rs, cudaStream_t stream) {
  const long long gx = (long long)((o + TF - 1) / TF) * ranks, sms = llg_sm_count();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)gx, (unsigned)((n + 8 * R - 1) / (8 * R)));
  cfg.blockDim = dim3(256);
  // where every block can have a multiprocessor of its own it asks for more than half of one's shared memory: blocks of a
  // cluster are placed densely otherwise, two on a multiprocessor beside an idle one
  constexpr int ALONE_SMEM = 120 * 1024;
  cfg.dynamicSmemBytes = gx * cfg.gridDim.y <= sms ? ALONE_SMEM : tile_smem(8 * R);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = llg_pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaFuncSetAttribute(gemm_tile_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, ALONE_SMEM);
  if (e != cudaSuccess) return llg_fail("gemm_simt: cannot have %d bytes of shared memory: %s", ALONE_SMEM, cudaGetErrorString(e));
  e = cudaLaunchKernelEx(&cfg, gemm_tile_kernel<R>, x, w, out, n, o, k, rs);
  if (e != cudaSuccess) return llg_fail("gemm_simt: launch: %s", cudaGetErrorString(e));
  return llg_check_launch("gemm_simt");
}

// Rows of a tile (40, 48, 56 or 64) and the blocks that share a tile's k: the multiprocessor with the most blocks has their steps to do, each as
// long as the tile has rows and four more, for its features (two blocks a multiprocessor take as long as one with twice the steps, to 5 %),
// and every block a fixed cost.  Clusters of four leave some multiprocessors out (288 blocks, 100 x 3,072 x 2,048: 68 us, where 144 in
// clusters of two take 51), clusters of eight more (42 us at 64 x 2,048 x 2,048).  Of the twelve forms, timed at 309 sizes (33 to 2,048
// rows, twelve matrices from 1,000 x 1,024 to 128,256 x 2,048), it takes 1.1 % more than the fastest on average and 21 % at worst, and nowhere
// more than tiles of 64 rows alone, which take 25 % more on average; with steps as long as the rows alone it took lower tiles where those of 64
// were 2 to 8 % faster (300 x 4,096 x 4,096: 339 us in tiles of 40, 319 in tiles of 64, four blocks each).
struct TileForm { int rows, ranks; };
constexpr int MAX_ROW_TILES = 65535;
TileForm tile_form(int n, int o, int k, long long sms) {
  const int steps = (k + TK - 1) / TK;
  TileForm best{64, 1};
  double best_cost = 0;
  for (int rows = 64; rows >= 40; rows -= 8) {
    if ((n + rows - 1) / rows > MAX_ROW_TILES) break;    // a grid's y: lower tiles would be more than it takes
    const long long tiles = (long long)((n + rows - 1) / rows) * ((o + TF - 1) / TF);
    for (int s = 1; s <= 4; s *= 2) {
      if (s > 1 && steps < 2 * s) break;
      const long long places = s == 4 ? sms - sms / 14 : sms, per_sm = (tiles * s + places - 1) / places;
      const double cost = (rows + 4) / 68.0 * (per_sm == 1 ? 1.0 : 0.95 * per_sm) * ((steps + s - 1) / s) + 3.0 + (s > 1 ? 2.0 : 0.0);
      if (best_cost == 0 || cost < best_cost * 0.999) {
        best_cost = cost;
        best = {rows, s};
      }
    }
  }
  return best;
}

int run_tile(const float* x, const float* w, float* out, int n, int o, int k, TileForm form, const RowScale& rs, cudaStream_t stream) {
  switch (form.rows) {
    case 40: return launch_tile<5>(x, w, out, n, o, k, form.ranks, rs, stream);
    case 48: return launch_tile<6>(x, w, out, n, o, k, form.ranks, rs, stream);
    case 56: return launch_tile<7>(x, w, out, n, o, k, form.ranks, rs, stream);
    default: return launch_tile<8>(x, w, out, n, o, k, form.ranks, rs, stream);
  }
}

// Rows up to which the weight stream is taken: its time rises with every eight rows, that of tiles of 40 does not.  At 24 and 32 rows 80 and
// 94 us at 16,384 x 2,048, where the tiles take 95; 43 and 55 (96) at 2,048 x 8,192; 18.5 and 23 (27) at 3,072 x 2,048; 13.7 and 17.6 (26.8)
// at 2,048 x 2,048.  Even at 32 for the widest, which is the most of a model's time.
constexpr int GEMV_ROWS_MAX = 32;

}  // namespace

// With `scale` (may be null) row r of the result is multiplied by the scale that a norm left for row r of x.
LLG_API int llg_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                          int n, int o, int k, const RowScale* scale, cudaStream_t stream) {
  LLG_REQUIRE(n >= 0 && o > 0 && k > 0, "gemm_simt: bad sizes n=%d o=%d k=%d", n, o, k);
  if (n == 0) return 0;
  dim3 grid((o + BN - 1) / BN, (n + BM - 1) / BM);
  LLG_REQUIRE(grid.y <= MAX_ROW_TILES, "gemm_simt: %d rows need more than 65535 row blocks", n);
  const RowScale rs = scale ? *scale : RowScale{nullptr, 0, 0.f, 0.f};
  if (x_dtype == LLG_F32 && w_dtype == LLG_F32 && out_dtype == LLG_F32 && k % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15u) == 0) {
    const float *xf = (const float*)x, *wf = (const float*)w;
    float* of = (float*)out;
    if (n == 1) return run_gemv<1, 8>(xf, wf, of, n, o, k, rs, stream);
    if (n == 2) return run_gemv<2, 8>(xf, wf, of, n, o, k, rs, stream);
    if (n == 3) return run_gemv<4, 8, 3>(xf, wf, of, n, o, k, rs, stream);
    if (n == 4) return run_gemv<4, 8>(xf, wf, of, n, o, k, rs, stream);
    if (n <= 6) return run_gemv<8, 4, 6>(xf, wf, of, n, o, k, rs, stream);
    if (n <= GEMV_ROWS_MAX) return run_gemv<8, 4>(xf, wf, of, n, o, k, rs, stream);
    return run_tile(xf, wf, of, n, o, k, tile_form(n, o, k, llg_sm_count()), rs, stream);
  }
#define LAUNCH(AT, WT, CT) \
  gemm_tn_kernel<AT, WT, CT><<<grid, 256, 0, stream>>>((const AT*)x, (const WT*)w, (CT*)out, n, o, k, rs)
  const int key = x_dtype * 4 + w_dtype * 2 + out_dtype;
  switch (key) {
    case 0: LAUNCH(float, float, float); break;
    case 1: LAUNCH(float, float, __nv_bfloat16); break;
    case 2: LAUNCH(float, __nv_bfloat16, float); break;
    case 3: LAUNCH(float, __nv_bfloat16, __nv_bfloat16); break;
    case 4: LAUNCH(__nv_bfloat16, float, float); break;
    case 5: LAUNCH(__nv_bfloat16, float, __nv_bfloat16); break;
    case 6: LAUNCH(__nv_bfloat16, __nv_bfloat16, float); break;
    case 7: LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16); break;
    default: return llg_fail("gemm_simt: unknown dtypes x=%d w=%d out=%d", x_dtype, w_dtype, out_dtype);
  }
#undef LAUNCH
  return llg_check_launch("gemm_simt");
}

// The float32 product in tiles of `rows` rows (40, 48, 56 or 64), `ranks` blocks (1, 2 or 4) sharing a tile's k: the form that llg_gemm_simt
// chooses by itself above some rows.  k in whole fours, operands on 16 bytes.
LLG_API int llg_gemm_simt_tile(const float* x, const float* w, float* out, int n, int o, int k, int rows, int ranks, const RowScale* scale,
                               cudaStream_t stream) {
  LLG_REQUIRE(n > 0 && o > 0 && k > 0 && k % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15u) == 0, "gemm_simt_tile: n=%d o=%d k=%d", n, o, k);
  LLG_REQUIRE((rows == 40 || rows == 48 || rows == 56 || rows == 64) && (ranks == 1 || ranks == 2 || ranks == 4) &&
                  (ranks == 1 || (k + TK - 1) / TK >= 2 * ranks) && (n + rows - 1) / rows <= MAX_ROW_TILES,
              "gemm_simt_tile: tiles of %d rows, %d blocks", rows, ranks);
  return run_tile(x, w, out, n, o, k, TileForm{rows, ranks}, scale ? *scale : RowScale{nullptr, 0, 0.f, 0.f}, stream);
}

// The form that llg_gemm_simt takes for these sizes above the rows of its weight stream: rows + 1,000 times the blocks of a tile.
LLG_API int llg_gemm_simt_form(int n, int o, int k, int sms) {
  const TileForm f = tile_form(n, o, k, sms);
  return f.rows + 1000 * f.ranks;
}
