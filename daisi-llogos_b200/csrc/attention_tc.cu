// Causal attention for prompt steps on the 5th-generation tensor cores (tcgen05), bfloat16, head
// sizes 64 and 128.
//
//   per 64-key tile (one cache page):   S = Q K^T      tcgen05.mma, accumulator S[128 x 64] in TMEM
//                                       each thread reads its row of S (tcgen05.ld), masks, updates the
//                                       running maximum and sum, writes P (bfloat16) over S (tcgen05.st)
//                                       O += P V       tcgen05.mma, P from TMEM, accumulator O[128 x head] in TMEM
//
// A block owns 256 queries of one head as two tiles of 128.  Each tile has a group of four softmax
// warps: thread r of a group owns query row r of its tile, which is lane r of tensor memory, so the
// softmax of a row needs no exchange between threads.  Four more warps serve the groups: a lane each
// issues a group's products, one warp copies the key tiles and one the value tiles (TMA boxes from the
// step's packed buffer or from a cache page; the one tile per sequence that lies partly in each row by
// row with cp.async; four stages each).
// The roles meet only at mbarriers: tiles full / free between the copying warps and the issuing lanes,
// scores ready, weights ready and accumulator updated between a group and its issuing lane.  Each
// group has two score buffers in tensor memory, so that the tensor core computes the next tile's
// scores and the previous tile's O += P V while the group runs the softmax of the current one; the
// scores of tile j + 1 are issued when O += P(j-1) V(j-1) has finished with the buffer they go into.
//
// Q and K are K-major operands in shared memory with the 128-byte swizzle; V is stored as it lies in
// memory ([key][dim], dim contiguous), which makes it the MN-major second operand of the second product;
// P never leaves tensor memory.
// A row's accumulator is rescaled in place (tcgen05.ld / tcgen05.st) only when a tile's weights add up to more than
// 2^14, warp by warp and only when some row of the warp needs it; only then are the tile's maxima worked out.
//
// A key tile's time is a softmax warp's chain of it, about 2,000 cycles: 64 exponentials a row (700 cycles with the other
// group's beside them 980; the special-function unit and the tensor cores are each busy 44 % of the time), the way in and out of
// tensor memory, and 100 to 200 cycles for each barrier that is passed.  So a tile has no maximum and no wait that it
// can do without.  8,192 tokens x 32 heads of 128, ten launches after a pause: 646 us with a lane for both groups' products, a maximum and a
// wait for the accumulator in every tile, 597 now (launch after launch under the power cap 648 at 1,920 MHz and 615 at 1,860); 2,048 tokens
// launch after launch 80 and 67, heads of 64 72 and 60; four prompts of 1,100 tokens, heads of 64, 128 and 98.
// (Taking turns with the exponentials, group by group: 650 us at 8,192 tokens where this form took 584, 82 at 2,048.)
//
// Tiles of at most 128 queries (short prompts, the next turn of a chat) leave the second group without queries.  It then takes
// part in one of two ways, which every block finds from its own tile.  SPLIT (two key tiles or more): the groups share the keys,
// the first takes the even tiles and the second the odd ones, and the threads of a row join the two accumulators at the end: a
// block's time is the chain of its key tiles (scores, softmax, product).  TWO_HEADS (one key tile, and more
// blocks than multiprocessors): the second group takes the next query head of the same key/value head and that head's own block
// ends at once; such blocks cost their set-up, so half as many are half the time.  Four sequences of 83 queries behind 1,000 to
// 4,000 keys, 32 heads of 128: 46 us (two groups of queries a block: 63); five prompts of 3 to 90 tokens, 32 heads of 64: 15 us (19).
//
// FEW, an instance of its own: a step whose time is the chain of a few long blocks (the next turns of a few long chats).  The query heads of a
// key/value head see the same keys, so their queries are rows of one list, a head's behind the last head's, that its blocks take 128 at a
// time, all of them SPLIT; and the keys of a tile may go to the blocks of a cluster, a consecutive run each, which leave their
// accumulators in shared memory and join them there, each block some of the columns, in the blocks' order.  few_form chooses by the
// step's lengths, for the step as a whole: all its tiles have as many parts.
//
// With MAPS (differential attention) the two halves of a query and of a key are two maps over the same values: the block's
// two groups are the two maps of ONE tile of 128 queries, whose scores are products over their half of the head; keys,
// values and queries arrive once for both.  At the end every thread reads a half of its row of both accumulators, takes
// the difference, and the two threads of a row exchange their sums of squares for the head's unit norm.
//
// Every mbarrier wait is bounded; on expiry the thread records an error (llg_attn_tc_status) and
// raises a flag that ends the other roles' waits; every role waits for its own copies in flight,
// and the block frees its tensor memory and returns.
#include "common.cuh"
#include "kernel_args.h"

#include <cuda.h>

#include <map>
#include <mutex>
#include <tuple>

LLG_API const char* llg_last_error() { return g_llg_error; }

namespace {

typedef __nv_bfloat16 bf16;
constexpr int BQ = 128;      // queries per tile (rows of a product, lanes of tensor memory)
constexpr int TK = 64;       // keys per tile = one cache page
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;
constexpr float LOG2E = 1.4426950408889634f;

// 2^x by the special-function unit alone (float32, about 2 ulp, denormal results flushed to zero, +inf past the range);
// exp2f() adds range handling that the softmax does not need: weights that are kept lie below 2^14, and a tile with an argument of any
// size ahead of its maximum, or a weight that has run over, fails the bound on its sum and is worked out again.
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^d for a whole number d <= 0 (or -inf), exactly.
__device__ __forceinline__ float pow2_whole(float d) {
  return d < -126.f ? 0.f : __int_as_float((127 + (int)d) << 23);
}

// the largest of three (one instruction on sm_100)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ int g_error = 0;  // 0 ok; waits that ran out: 1 scores, 2 accumulator, 4 free stage, 5 tile copied, 6 weights, 7 copies at the end; 3 shared memory not aligned to 1024 bytes

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  int spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 1023) == 0) {
      if (*abort_flag) return false;
      if (now_ns() - t0 > WAIT_LIMIT_NS) return false;
    }
  }
  return true;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// shared memory written by threads (cp.async, st.shared) becomes visible to the tensor core's reads
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// K-major operand, rows of 128 bytes with the 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// MN-major operand: 64 elements of the MN dimension are contiguous (one swizzled 128-byte row per k),
// 8-k groups 1024 bytes apart, the next 64 MN elements `lbo_bytes` further
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t addr, uint32_t lbo_bytes) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// first operand from tensor memory (lane = row, one 32-bit column per two k), second from shared memory
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// byte offset of 16-byte chunk `chunk` (0..7) of row `row` in a tile of 128-byte rows with the 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int row, int chunk) { return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4)); }

constexpr int GROUPS = 2;                     // query tiles of 128 rows per block, each with its own softmax warps
constexpr int KST = 4, VST = 4;               // stages of keys and of values
static_assert(KST % 2 == 0 && VST % 2 == 0, "where the groups take turns with the key tiles, a stage belongs to one of them: a wait for its next phase "
              "by parity means something only to who has seen the last one");
constexpr int WORKERS = GROUPS * BQ;          // softmax threads: thread r of group g owns query row r of tile g
constexpr int ISSUE_WARP = WORKERS / 32;      // one lane of this warp issues the first group's products
constexpr int K_LOAD_WARP = ISSUE_WARP + 1;   // copies key tiles
constexpr int V_LOAD_WARP = ISSUE_WARP + 2;   // copies value tiles
constexpr int ISSUE_WARP_2 = ISSUE_WARP + 3;  // issues the second group's products
constexpr int THREADS = (ISSUE_WARP_2 + 1) * 32;

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// What a block knows about its two query tiles and the key tiles they need.
struct TileInfo {
  int b, tok0, lb, slot, k_begin;
  int nq[GROUPS], pos0[GROUPS], n_tiles[GROUPS], n_max;
};

// What the second group does (above): queries of its own; the odd key tiles of the first group's; the next query head.
enum { PLAIN = 0, SPLIT = 1, TWO_HEADS = 2 };

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// an address of this block's shared memory, in the cluster's block `rank`
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 peer_ld4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 peer_ld2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
constexpr int MAX_PARTS = 8;                  // blocks of a cluster that share a tile's keys

template <int HD, bool MAPS, bool FEW>
__global__ void __launch_bounds__(384, 1) attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_k_pages,
                                                                 const __grid_constant__ CUtensorMap map_v_pages,
                                                                 const __grid_constant__ CUtensorMap map_k_new,
                                                                 const __grid_constant__ CUtensorMap map_v_new, PrefillArgs a) {
  constexpr int KB = HD / 64;                 // 64-wide blocks of the head dimension
  constexpr int Q_BYTES = KB * BQ * 128;      // [KB][128 rows][128 bytes]
  constexpr int KV_BYTES = KB * TK * 128;     // [KB][64 keys][128 bytes]
  constexpr int TMEM_COLS = 512;              // per group 256: S 2 x 64 columns, O HD columns from column 128
  constexpr uint32_t G_COLS = 256, O_COL = 128;
  constexpr int CPR = HD / 8;                 // 16-byte chunks per row of the head
  // The tiles need 1024-byte alignment (swizzle); the declaration asks for it and the kernel checks it.
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int Q_TILES = MAPS || FEW ? 1 : GROUPS;
  static_assert(!(MAPS && FEW), "two maps are two groups of one tile of queries");
  unsigned char* Qs = smem;                          // [Q_TILES]
  unsigned char* Ks = Qs + Q_TILES * Q_BYTES;        // [KST]
  unsigned char* Vs = Ks + KST * KV_BYTES;           // [VST]
  __shared__ uint64_t k_full[KST], k_free[KST], v_full[VST], v_free[VST];
  __shared__ uint64_t s_full[GROUPS][2], p_ready[GROUPS][2], o_done[GROUPS], q_ready;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ float split_share[MAPS ? 1 : GROUPS][2][MAPS ? 1 : BQ];     // SPLIT: each group's maximum and sum of a row
  __shared__ float2 part_share[FEW ? BQ : 1];                            // this block's maximum and sum of a row
  __shared__ float map_share[MAPS ? 2 * GROUPS : 1][MAPS ? BQ : 1];      // 1 / sum of each map's weights, sums of squares

  if (!FEW) pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) LLG_STAMP(5, 0, 0, blockIdx.x + gridDim.x * blockIdx.y);
  // Blocks start in the order of blockIdx.x, then blockIdx.y: all heads of the list's first tile, then all
  // heads of its second ...  The caller lists the tiles with the most keys first, so that the long blocks
  // start first and the short ones fill the gaps at the end.
  // (lengths and tiles are the step's, written before its first kernel: they need not wait for the kernel before this one)
  TileInfo ti;
  int mode = PLAIN;
  const int parts = FEW ? (int)gridDim.z : 1, heads_per_kv = a.nh / a.nkv;
  int queries = 0, row0 = 0, q_off_few = 0;   // FEW: the tile's queries, the block's first row of the list, the tile's first query
  if constexpr (FEW) {
    const int blocks = (int)gridDim.x / a.nkv;            // of a key/value head
    ti.b = a.tiles[2 * blockIdx.y];
    q_off_few = a.tiles[2 * blockIdx.y + 1];
    ti.tok0 = a.cu_tokens[ti.b];
    ti.lb = a.len_before[ti.b];
    ti.slot = a.slots[ti.b];
    queries = min(GROUPS * BQ, a.cu_tokens[ti.b + 1] - ti.tok0 - q_off_few);
    row0 = (int)blockIdx.x % blocks * BQ;
    const int rows = min(BQ, queries * heads_per_kv - row0);
    if (rows <= 0) return;                                // (all blocks of a cluster alike)
    // the rows' first and last query: all of the tile's where the rows are not one head's
    const bool one_head = row0 / queries == (row0 + rows - 1) / queries;
    const int q_first = one_head ? row0 % queries : 0, q_last = one_head ? (row0 + rows - 1) % queries : queries - 1;
    mode = SPLIT;
    for (int g = 0; g < GROUPS; ++g) {
      ti.nq[g] = rows;
      ti.pos0[g] = ti.lb + q_off_few + q_first;
      ti.n_tiles[g] = 0;                                  // (SPLIT: by n_max)
    }
    ti.k_begin = mask_first(ti.pos0[0], a.window, a.chunked) / TK * TK;
    ti.n_max = (ti.lb + q_off_few + q_last + 1 - ti.k_begin + TK - 1) / TK;
    // this block's run of the key tiles (the last blocks may find none left)
    const int run = (ti.n_max + parts - 1) / parts, t0 = min((int)blockIdx.z * run, ti.n_max);
    ti.k_begin += t0 * TK;
    ti.n_max = min(run, ti.n_max - t0);
  } else {
    const int tile_id = (int)blockIdx.y;
    ti.b = a.tiles[2 * tile_id];
    const int q_off = a.tiles[2 * tile_id + 1];
    ti.tok0 = a.cu_tokens[ti.b];
    const int total = a.cu_tokens[ti.b + 1] - ti.tok0;
    ti.lb = a.len_before[ti.b];
    ti.slot = a.slots[ti.b];
    ti.n_max = 0;
    for (int g = 0; g < GROUPS; ++g) {
      ti.nq[g] = max(0, min(BQ, total - q_off - g * (MAPS ? 0 : BQ)));
      ti.pos0[g] = ti.lb + q_off + g * (MAPS ? 0 : BQ);
    }
    if (!MAPS && ti.nq[0] > 0 && ti.nq[1] == 0) {
      const int n_keys = ti.pos0[0] + ti.nq[0] - mask_first(ti.pos0[0], a.window, a.chunked) / TK * TK;
      uint32_t sms;
      asm("mov.u32 %0, %%nsmid;" : "=r"(sms));
      if (n_keys > TK) mode = SPLIT;
      else if ((a.nh / a.nkv) % 2 == 0 && gridDim.x * gridDim.y > sms) mode = TWO_HEADS;
      if (mode != PLAIN) {
        ti.nq[1] = ti.nq[0];
        ti.pos0[1] = ti.pos0[0];
      }
    }
    // the first group's window starts earliest; the second masks the tiles that lie before its own
    int kb = mask_first(ti.pos0[0], a.window, a.chunked);
    ti.k_begin = (kb / TK) * TK;
    for (int g = 0; g < GROUPS; ++g) {
      ti.n_tiles[g] = ti.nq[g] > 0 ? (ti.pos0[g] + ti.nq[g] - ti.k_begin + TK - 1) / TK : 0;
      ti.n_max = max(ti.n_max, ti.n_tiles[g]);
    }
  }
  if (mode == TWO_HEADS && (blockIdx.x & 1)) return;       // the block of the head before takes this one along
  const int g_step = MAPS || mode != PLAIN ? 0 : BQ;       // queries from one group's tile to the next one's
  const bool one_q = MAPS || mode == SPLIT;                // the groups read one tile of queries

  if ((smem_u32(smem) & 1023u) != 0) {          // uniform over the block
    if (tid == 0) atomicCAS(&g_error, 0, 3);
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < KST; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_free[s], mode == SPLIT ? 1 : GROUPS);       // who reads a tile: one group, or both
    }
    for (int s = 0; s < VST; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_free[s], mode == SPLIT ? 1 : GROUPS);
    }
    for (int g = 0; g < GROUPS; ++g) {
      mbar_init(&s_full[g][0], 1);
      mbar_init(&s_full[g][1], 1);
      mbar_init(&p_ready[g][0], BQ / 32);
      mbar_init(&p_ready[g][1], BQ / 32);
      mbar_init(&o_done[g], 1);
    }
    mbar_init(&q_ready, WORKERS);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    warp_whole();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // (a cluster's blocks come together: a block of a later kernel must not take tensor memory ahead of one of theirs and then wait for it; nor
  // may another cluster's block, see block_smem)
  if (FEW) pdl_launch_dependents();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_slot;
  volatile int* abortp = &abort_flag;
  pdl_wait();
  if (tid == 0) LLG_STAMP(5, 1, 0, blockIdx.x + gridDim.x * blockIdx.y);

  const int h = blockIdx.x, kvh = FEW ? (int)blockIdx.x / ((int)gridDim.x / a.nkv) : h / heads_per_kv;
  const int k_end = FEW ? ti.lb + q_off_few + queries : ti.pos0[0] + (ti.nq[1] > 0 ? g_step + ti.nq[1] : ti.nq[0]);   // keys past it are never copied
  const int q_tok0 = FEW ? ti.tok0 + q_off_few : ti.tok0 + ti.pos0[0] - ti.lb;  // first token of the first query tile
  // FEW: a row's query among the tile's, and its head
  auto row_query = [&](int row) { return (row0 + row) % queries; };
  auto row_head = [&](int row) { return kvh * heads_per_kv + (row0 + row) / queries; };

  // queries: thread r of group g copies its part of tile g; the issuing lane waits for all of them,
  // the copying warps start on the keys and values meanwhile
  if (tid < WORKERS) {
    const int g = tid / BQ, r = tid % BQ;
    const int ch = r % CPR;
    constexpr int ROWS = BQ / CPR;                   // rows a group copies side by side; with one tile the groups share its rows
    const int head = h + (mode == TWO_HEADS ? g : 0);
    for (int row = r / CPR + (one_q ? g * ROWS : 0); row < BQ; row += one_q ? GROUPS * ROWS : ROWS) {
      const bool valid = row < ti.nq[g];
      const int at = valid ? row : 0;
      const bf16* src = (const bf16*)a.q + ch * 8 +
                        (FEW ? (long long)(q_tok0 + row_query(at)) * a.nh + row_head(at) : (long long)(q_tok0 + g * g_step + at) * a.nh + head) * HD;
      cp_async16(smem_u32(Qs + (one_q ? 0 : g * Q_BYTES)) + (uint32_t)((ch >> 3) * (BQ * 128)) + swz(row, ch & 7), src, valid);
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_async_smem();
    mbar_arrive(&q_ready);
  }

  if (warp == K_LOAD_WARP || warp == V_LOAD_WARP) {
    // ---- copies: one warp per operand.  A tile that lies in one cache page, or in this step's packed rows,
    // is two TMA boxes (64 keys x 64 dimensions, 128-byte swizzle) that one lane requests; the one tile per
    // sequence that lies partly in each is copied row by row with cp.async by the whole warp. ------------
    const bool keys = warp == K_LOAD_WARP;
    const int stages = keys ? KST : VST;
    unsigned char* base = keys ? Ks : Vs;
    uint64_t* full = keys ? k_full : v_full;
    uint64_t* freeb = keys ? k_free : v_free;
    const CUtensorMap* map_pages = keys ? &map_k_pages : &map_v_pages;
    const CUtensorMap* map_new = keys ? &map_k_new : &map_v_new;
    const bf16* fresh_src = (const bf16*)(keys ? a.k_new : a.v_new);
    const bf16* page_src = (const bf16*)(keys ? a.k_pages : a.v_pages);
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(map_pages) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(map_new) : "memory");
    }
    const int ch = lane % CPR;
    constexpr int RSTEP = 32 / CPR;
    int requested = 0;                          // tiles whose copies have been requested
    for (int t = 0; t < ti.n_max; ++t) {
      const int st = t % stages;
      const bool left = t < stages || mbar_wait(&freeb[st], (t / stages - 1) & 1, abortp);
      if (!left && !*abortp) { *abortp = 1; atomicCAS(&g_error, 0, 4); }
      if (!warp_all(left)) break;          // one answer for the warp: its lanes meet again below
      requested = t + 1;
      const int kt = ti.k_begin + t * TK;
      const uint32_t dst = smem_u32(base + st * KV_BYTES);
      if (kt >= ti.lb) {
        // rows past the sequence's last token are another sequence's, or zeros past the buffer: no query sees them
        if (lane == 0) {
          mbar_expect_tx(&full[st], KV_BYTES);
#pragma unroll
          for (int blk = 0; blk < KB; ++blk)
            tma_load_3d(dst + blk * (TK * 128), map_new, blk * 64, kvh, ti.tok0 + kt - ti.lb, &full[st]);
        }
      } else if (kt + TK <= ti.lb) {
        if (lane == 0) {
          const int row0 = (int)kv_row(a.page_table, a.table_width, a.ring_pages, ti.slot, kt, kvh, a.nkv);
          mbar_expect_tx(&full[st], KV_BYTES);
#pragma unroll
          for (int blk = 0; blk < KB; ++blk) tma_load_2d(dst + blk * (TK * 128), map_pages, blk * 64, row0, &full[st]);
        }
      } else {
        const long long old_base = kv_row(a.page_table, a.table_width, a.ring_pages, ti.slot, kt, kvh, a.nkv) * HD;
        const long long new_base = ((long long)(ti.tok0 + kt - ti.lb) * a.nkv + kvh) * HD;
        for (int row = lane / CPR; row < TK; row += RSTEP) {
          const int pos = kt + row;
          const bool valid = pos < k_end, fresh = pos >= ti.lb;
          const long long off = (fresh ? new_base + (long long)row * a.nkv * HD : old_base + (long long)row * HD) + ch * 8;
          cp_async16(dst + (uint32_t)((ch >> 3) * (TK * 128)) + swz(row, ch & 7), (fresh ? fresh_src : page_src) + (valid ? off : 0),
                     valid);
        }
        cp_async_commit();
        cp_async_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[st]);
      }
      __syncwarp();
    }
    // Copies still write into this block's shared memory until their barrier completes: before the block
    // may end, see the last tile of every stage arrive (at once, unless a wait ran out somewhere).
    if (lane == 0) {
      for (int t = max(0, requested - stages); t < requested; ++t) {
        const unsigned long long t0 = now_ns();
        while (!mbar_try_wait(&full[t % stages], (t / stages) & 1)) {
          if (now_ns() - t0 > WAIT_LIMIT_NS) { atomicCAS(&g_error, 0, 7); break; }
        }
      }
    }
  } else if (warp == ISSUE_WARP || warp == ISSUE_WARP_2) {
    // ---- products: one lane per group issues them.  The tensor core takes them one after the other, and a lane that issues is
    // held up while its queue is full, which is why no softmax warp does this; one lane for both groups let each group's next
    // scores wait for the other group's weights. ------
    if (elect_one()) {
      const int g = warp == ISSUE_WARP ? 0 : 1;
      const bool split = !MAPS && mode == SPLIT;
      constexpr uint32_t IDESC_S = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TK >> 3) << 17) | ((uint32_t)(BQ >> 4) << 24);
      constexpr uint32_t IDESC_O = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(BQ >> 4) << 24);
      bool ok = true;
      auto wait_or_fail = [&](uint64_t* bar, uint32_t parity, int code) {
        if (!ok) return;
        if (!mbar_wait(bar, parity, abortp)) {
          if (!*abortp) { *abortp = 1; atomicCAS(&g_error, 0, code); }
          ok = false;
        }
      };
      // the group's own tile i is key tile i, or (SPLIT) every second one
      const int n_own = split ? (ti.n_max + 1 - g) >> 1 : ti.n_tiles[g];
      auto tile_of = [&](int i) { return split ? 2 * i + g : i; };
      // scores of the group's tile i into its score buffer i % 2
      auto issue_scores = [&](int i) {
        const int t = tile_of(i);
        wait_or_fail(&k_full[t % KST], (t / KST) & 1, 5);
        if (i >= 2) wait_or_fail(&o_done[g], i & 1, 6);            // O += P(i-2) V(i-2) has read the buffer
        if (!ok) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t qa = smem_u32(Qs + (one_q ? 0 : g * Q_BYTES)), ka = smem_u32(Ks + (t % KST) * KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < (MAPS ? HD / 32 : HD / 16); ++ks) {
          const int at = MAPS ? g * (HD / 32) + ks : ks;
          const uint32_t blk = at >> 2, kk = at & 3;      // 64-wide block, 16-wide step inside it (32 bytes)
          umma_bf16(tmem + g * G_COLS + (uint32_t)(i & 1) * TK, desc_kmajor(qa + blk * (BQ * 128) + kk * 32),
                    desc_kmajor(ka + blk * (TK * 128) + kk * 32), IDESC_S, ks != 0);
        }
        umma_commit(&s_full[g][i & 1]);
        umma_commit(&k_free[t % KST]);
      };
      wait_or_fail(&q_ready, 0, 5);
      if (n_own > 0) issue_scores(0);
      // Step i: the scores of tile i + 1; then, once the group has turned S(i) into P(i) (written over S(i) in tensor memory),
      // O += P(i) V(i).
      for (int i = 0; i < n_own && ok; ++i) {
        const int t = tile_of(i);
        if (i + 1 < n_own) issue_scores(i + 1);
        wait_or_fail(&v_full[t % VST], (t / VST) & 1, 5);
        wait_or_fail(&p_ready[g][i & 1], (i >> 1) & 1, 6);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t pa = tmem + g * G_COLS + (uint32_t)(i & 1) * TK, va = smem_u32(Vs + (t % VST) * KV_BYTES);
#pragma unroll
        for (int kk = 0; kk < TK / 16; ++kk) {
          // 16 keys further: 8 columns of packed weights, 16 rows (2048 bytes) down V
          umma_bf16_ts(tmem + g * G_COLS + O_COL, pa + kk * 8, desc_mnmajor(va + kk * 2048, TK * 128), IDESC_O, (i | kk) != 0);
        }
        umma_commit(&o_done[g]);
        umma_commit(&v_free[t % VST]);
      }
      // tiles that only the other group sees: given back as they arrive
      if (!split) {
        for (int t = n_own; t < ti.n_max && ok; ++t) {
          wait_or_fail(&k_full[t % KST], (t / KST) & 1, 5);
          if (ok) mbar_arrive(&k_free[t % KST]);
          wait_or_fail(&v_full[t % VST], (t / VST) & 1, 5);
          if (ok) mbar_arrive(&v_free[t % VST]);
        }
      }
    }
  } else if (tid < WORKERS && ti.nq[tid / BQ] > 0) {
    // ---- softmax: thread r of group g owns query row r of tile g ------------------------------------
    const int g = tid / BQ, r = tid % BQ, gw = (tid % BQ) >> 5;       // gw: warp inside the group = its lane quarter
    const uint32_t lane_base = tmem + g * G_COLS + ((uint32_t)(gw * 32) << 16);
    const bool split = !MAPS && mode == SPLIT;
    const int n_tiles = split ? (ti.n_max + 1 - g) >> 1 : ti.n_tiles[g], pos0 = ti.pos0[g];
    const float sc = a.scale * LOG2E;
    // A row's weights are 2^(x - M) with x = score * scale * log2 e and M a whole number that is raised (to the
    // tile's maximum, rounded up) only when a tile's weights add up to more than 2^14, so some weight is above 2^8: no weight
    // exceeds 2^14 and the accumulator is rescaled rarely, by an exact power of two.  The common factor cancels in the final division.
    // A weight rounded to bfloat16 has the same digits for any whole M but for the rounding of x - M itself (float32, at a magnitude that
    // depends on M): now and then, where 2^(x - M) lies next to the middle of two bfloat16 numbers, it goes the other way.  So how the
    // keys are cut into tiles or steps shows in a last bit of some weights and in no error: against 64 bits 2.289e-3 to 2.342e-3 at 2,048
    // tokens and scores of standard deviation 0.3 to 8, to four digits the same under a rule that raised M by every tile's maximum.
    const float sum_bound = 16384.0f;
    const int qpos = FEW ? ti.lb + q_off_few + row_query(r) : pos0 + r;
    // positions of the warp's first and last row, for the tiles that need no mask (FEW: of the block's)
    const int warp_first = FEW ? pos0 : pos0 + gw * 32, warp_last = FEW ? ti.lb + q_off_few + queries - 1 : pos0 + gw * 32 + 31;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const bool scored = mbar_wait(&s_full[g][j & 1], (j >> 1) & 1, abortp);
      if (!scored && !*abortp) { *abortp = 1; atomicCAS(&g_error, 0, 1); }
      ok = warp_all(scored);
      if (!ok) break;                      // uniform: one answer for the warp, tensor memory's instructions want all of its lanes
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int kt = ti.k_begin + (split ? 2 * j + g : j) * TK;
      float sv[TK];
      {
        uint32_t r0_[16], r1_[16], r2_[16], r3_[16];
        const uint32_t sa = lane_base + (uint32_t)(j & 1) * TK;
        tmem_ld16(sa, r0_);
        tmem_ld16(sa + 16, r1_);
        tmem_ld16(sa + 32, r2_);
        tmem_ld16(sa + 48, r3_);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          sv[c] = __uint_as_float(r0_[c]);
          sv[16 + c] = __uint_as_float(r1_[c]);
          sv[32 + c] = __uint_as_float(r2_[c]);
          sv[48 + c] = __uint_as_float(r3_[c]);
        }
      }
      const bool need_mask = (kt + TK - 1 > warp_first) || (a.window > 0 && kt < mask_first(warp_last, a.window, a.chunked));
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < TK; ++c) {
          const int key = kt + c;
          const bool valid = key <= qpos && key >= mask_first(qpos, a.window, a.chunked);
          sv[c] = valid ? sv[c] : -INFINITY;
        }
      }
      // The weights of the tile at the M there is, and their sum: a sum within the bound says that no weight is far out of
      // range, so most tiles need no maximum (its 32 instructions a row took a quarter of a tile's time).
      // Two elements per instruction where the arithmetic allows it (fma.rn.f32x2, add.rn.f32x2).
      uint32_t pk[TK / 2];
      float psum;
      auto weights = [&](float m) {
        const float ms = m == -INFINITY ? 0.f : m;
        const float2 sc2 = make_float2(sc, sc), nms2 = make_float2(-ms, -ms);
        float2 ps2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int e = 0; e < TK / 2; ++e) {
          const float2 x = __ffma2_rn(make_float2(sv[2 * e], sv[2 * e + 1]), sc2, nms2);
          const float2 w = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          ps2[e & 1] = __fadd2_rn(ps2[e & 1], w);
          pk[e] = pack_bf16(w.x, w.y);
        }
        psum = (ps2[0].x + ps2[0].y) + (ps2[1].x + ps2[1].y);
      };
      float corr = 1.f;
      bool fits = false, rescale = false;                // the latter one answer for the warp
#pragma unroll 1
      for (int pass = j == 0; ; ++pass) {
        if (pass == 1) {
          // the first tile, one whose scores rise, rows that have seen no key yet
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < TK; c += 8) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mx4[k] = max3(mx4[k], sv[c + 2 * k], sv[c + 2 * k + 1]);
          }
          const float mxs = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sc;
          const float m_new = fits ? m_run : fmaxf(m_run, ceilf(mxs));
          corr = m_new == m_run || m_new == -INFINITY ? 1.f : pow2_whole(m_run - m_new);
          m_run = m_new;
          rescale = !warp_all(corr == 1.f);
        }
        weights(m_run);
        fits = m_run != -INFINITY && psum <= sum_bound;
        if (pass == 1 || warp_all(fits)) break;          // uniform
      }
      // P(j) takes the place of S(j) in tensor memory: 64 weights of a row in 32 columns
      warp_whole();
#pragma unroll
      for (int c16 = 0; c16 < TK / 32; ++c16)          // uniform
        tmem_st16(lane_base + (uint32_t)(j & 1) * TK + c16 * 16, reinterpret_cast<const uint32_t(&)[16]>(pk[c16 * 16]));
      l_run = l_run * corr + psum;

      // A rescaled accumulator, and the last tile's: O += P(j-1) V(j-1) has finished.  (Scores of tile j mean that O += P(j-2) V(j-2) has, so a
      // wait by parity is for that product's end and no other.)
      const bool rescale_now = j > 0 && rescale;
      if (rescale_now || (j > 0 && j + 1 == n_tiles)) {
        const bool added = mbar_wait(&o_done[g], (j - 1) & 1, abortp);
        if (!added && !*abortp) { *abortp = 1; atomicCAS(&g_error, 0, 2); }
        ok = warp_all(added);
        if (!ok) break;                                // uniform
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (rescale_now) {                             // uniform: rescale is one answer for the warp
#pragma unroll
          for (int c0 = 0; c0 < HD; c0 += 16) {        // uniform
            uint32_t rr[16];
            tmem_ld16(lane_base + O_COL + c0, rr);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 16; ++c) rr[c] = __float_as_uint(__uint_as_float(rr[c]) * corr);
            tmem_st16(lane_base + O_COL + c0, rr);
          }
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[g][j & 1]);      // one arrival a warp: 128 on one barrier stand in line
    }
    if (ok) {
      const bool added = mbar_wait(&o_done[g], (n_tiles - 1) & 1, abortp);
      if (!added && !*abortp) { *abortp = 1; atomicCAS(&g_error, 0, 2); }
      ok = warp_all(added);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (MAPS) {
      // the two groups meet (both have the same queries, so all 256 threads come here, also after a wait that ran out)
      map_share[g][r] = l_run > 0.f ? 1.0f / l_run : 0.f;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool whole = !*abortp;                       // uniform behind the barrier: no wait is left that could run out
      float o[HD / 2], ss = 0.f;
      if (whole) {
        const float w1 = map_share[0][r], w2 = -a.map_lambda * map_share[GROUPS - 1][r];
        const uint32_t row = tmem + O_COL + ((uint32_t)(gw * 32) << 16) + (uint32_t)(g * (HD / 2));
#pragma unroll
        for (int c0 = 0; c0 < HD / 2; c0 += 16) {
          uint32_t r1[16], r2[16];
          warp_whole();
          tmem_ld16(row + c0, r1);
          tmem_ld16(row + G_COLS + c0, r2);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const float v = fmaf(w2, __uint_as_float(r2[c]), w1 * __uint_as_float(r1[c]));
            o[c0 + c] = v;
            ss = fmaf(v, v, ss);
          }
        }
      }
      map_share[GROUPS + g][r] = ss;
      asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
      if (whole && r < ti.nq[g]) {
        const float f = a.map_scale / sqrtf((map_share[GROUPS][r] + map_share[2 * GROUPS - 1][r]) / (float)HD + a.map_eps);
        bf16* dst = (bf16*)a.out + ((long long)(q_tok0 + r) * a.nh + h) * HD + g * (HD / 2);
#pragma unroll
        for (int c0 = 0; c0 < HD / 2; c0 += 8) {
          uint4 v;
          v.x = pack_bf16(o[c0] * f, o[c0 + 1] * f);
          v.y = pack_bf16(o[c0 + 2] * f, o[c0 + 3] * f);
          v.z = pack_bf16(o[c0 + 4] * f, o[c0 + 5] * f);
          v.w = pack_bf16(o[c0 + 6] * f, o[c0 + 7] * f);
          *reinterpret_cast<uint4*>(dst + c0) = v;
        }
      }
    } else if (FEW) {
      // the two groups meet, as above: every thread joins a half of its row's two accumulators and writes them out, or, where the
      // keys are in parts, leaves them where queries, keys and values were (all products have read those): four columns of all rows
      // after four columns
      split_share[g][0][r] = m_run;
      split_share[g][1][r] = l_run;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool whole = warp_all(!*abortp);
      const float m0 = split_share[0][0][r], m1 = split_share[1][0][r], m = fmaxf(m0, m1);
      float w0 = m0 == -INFINITY ? 0.f : fast_exp2(m0 - m), w1 = m1 == -INFINITY ? 0.f : fast_exp2(m1 - m);
      float l = split_share[0][1][r] * w0 + split_share[1][1][r] * w1;
      if (g == 0) part_share[FEW ? r : 0] = make_float2(m, l);
      const bool live = r < ti.nq[g];
      const int head = live ? row_head(r) : 0, tok = q_tok0 + row_query(r);
      if (parts == 1) {
        if (a.has_sink) l += fast_exp2((a.sinks ? a.sinks[head] : a.sink_score) * LOG2E - m);
        float inv = l > 0.f ? 1.0f / l : 0.f;
        if (a.gate && live) inv *= a.gate[(long long)tok * a.nh + head];
        w0 *= inv;
        w1 *= inv;
      }
      const bool some0 = ti.n_max > 0, some1 = ti.n_max > 1;      // an accumulator that no tile went into holds anything
      bf16* dst = (bf16*)a.out + ((long long)tok * a.nh + head) * HD;
      const uint32_t row = tmem + O_COL + ((uint32_t)(gw * 32) << 16);
#pragma unroll 1
      for (int c0 = g * (HD / 2); c0 < (g + 1) * (HD / 2); c0 += 16) {
        uint32_t r0_[16], r1_[16];
        warp_whole();                                     // (the last columns' stores are those of the queries that there are)
        if (whole) {                                      // uniform
          tmem_ld16(row + c0, r0_);
          tmem_ld16(row + G_COLS + c0, r1_);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float o[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          o[c] = some0 ? w0 * __uint_as_float(r0_[c]) : 0.f;
          if (some1) o[c] = fmaf(w1, __uint_as_float(r1_[c]), o[c]);
        }
        if (parts > 1) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            reinterpret_cast<float4*>(smem)[(c0 / 4 + q) * BQ + r] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        } else if (live && whole) {
          uint4 v0, v1;
          v0.x = pack_bf16(o[0], o[1]); v0.y = pack_bf16(o[2], o[3]); v0.z = pack_bf16(o[4], o[5]); v0.w = pack_bf16(o[6], o[7]);
          v1.x = pack_bf16(o[8], o[9]); v1.y = pack_bf16(o[10], o[11]); v1.z = pack_bf16(o[12], o[13]); v1.w = pack_bf16(o[14], o[15]);
          *reinterpret_cast<uint4*>(dst + c0) = v0;
          *reinterpret_cast<uint4*>(dst + c0 + 8) = v1;
        }
      }
    } else if (split) {
      // the two groups meet, as above: every thread joins a half of its row's two accumulators
      split_share[g][0][r] = m_run;
      split_share[g][1][r] = l_run;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!*abortp) {
        const float m0 = split_share[0][0][r], m1 = split_share[1][0][r], m = fmaxf(m0, m1);
        float w0 = m0 == -INFINITY ? 0.f : fast_exp2(m0 - m), w1 = m1 == -INFINITY ? 0.f : fast_exp2(m1 - m);
        float l = split_share[0][1][r] * w0 + split_share[1][1][r] * w1;
        if (a.has_sink) l += fast_exp2((a.sinks ? a.sinks[h] : a.sink_score) * LOG2E - m);
        float inv = l > 0.f ? 1.0f / l : 0.f;
        if (a.gate && r < ti.nq[g]) inv *= a.gate[(long long)(q_tok0 + r) * a.nh + h];
        w0 *= inv;
        w1 *= inv;
        const uint32_t row = tmem + O_COL + ((uint32_t)(gw * 32) << 16) + (uint32_t)(g * (HD / 2));
        bf16* dst = (bf16*)a.out + ((long long)(q_tok0 + r) * a.nh + h) * HD + g * (HD / 2);
#pragma unroll
        for (int c0 = 0; c0 < HD / 2; c0 += 16) {
          uint32_t r0_[16], r1_[16];
          warp_whole();                                   // (the last columns' stores are those of the queries that there are)
          tmem_ld16(row + c0, r0_);
          tmem_ld16(row + G_COLS + c0, r1_);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (r < ti.nq[g]) {
            float o[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) o[c] = fmaf(w1, __uint_as_float(r1_[c]), w0 * __uint_as_float(r0_[c]));
            uint4 v0, v1;
            v0.x = pack_bf16(o[0], o[1]); v0.y = pack_bf16(o[2], o[3]); v0.z = pack_bf16(o[4], o[5]); v0.w = pack_bf16(o[6], o[7]);
            v1.x = pack_bf16(o[8], o[9]); v1.y = pack_bf16(o[10], o[11]); v1.z = pack_bf16(o[12], o[13]); v1.w = pack_bf16(o[14], o[15]);
            *reinterpret_cast<uint4*>(dst + c0) = v0;
            *reinterpret_cast<uint4*>(dst + c0 + 8) = v1;
          }
        }
      }
    } else if (warp_all(ok && !*abortp)) {
      const int head = h + (mode == TWO_HEADS ? g : 0);
      // a sink joins the sum with its own weight 2^(sink - M) and carries no value; a gate scales the head's output
      if (a.has_sink) l_run += fast_exp2((a.sinks ? a.sinks[head] : a.sink_score) * LOG2E - m_run);
      float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      if (a.gate && r < ti.nq[g]) inv *= a.gate[(long long)(q_tok0 + g * g_step + r) * a.nh + head];
      bf16* dst = (bf16*)a.out + ((long long)(q_tok0 + g * g_step + r) * a.nh + head) * HD;
#pragma unroll
      for (int c0 = 0; c0 < HD; c0 += 16) {
        uint32_t rr[16];
        warp_whole();                                     // (the last columns' stores are those of the queries that there are)
        tmem_ld16(lane_base + O_COL + c0, rr);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (r < ti.nq[g]) {
          uint4 v0, v1;
          v0.x = pack_bf16(__uint_as_float(rr[0]) * inv, __uint_as_float(rr[1]) * inv);
          v0.y = pack_bf16(__uint_as_float(rr[2]) * inv, __uint_as_float(rr[3]) * inv);
          v0.z = pack_bf16(__uint_as_float(rr[4]) * inv, __uint_as_float(rr[5]) * inv);
          v0.w = pack_bf16(__uint_as_float(rr[6]) * inv, __uint_as_float(rr[7]) * inv);
          v1.x = pack_bf16(__uint_as_float(rr[8]) * inv, __uint_as_float(rr[9]) * inv);
          v1.y = pack_bf16(__uint_as_float(rr[10]) * inv, __uint_as_float(rr[11]) * inv);
          v1.z = pack_bf16(__uint_as_float(rr[12]) * inv, __uint_as_float(rr[13]) * inv);
          v1.w = pack_bf16(__uint_as_float(rr[14]) * inv, __uint_as_float(rr[15]) * inv);
          *reinterpret_cast<uint4*>(dst + c0) = v0;
          *reinterpret_cast<uint4*>(dst + c0 + 8) = v1;
        }
      }
    }
  }

  if (FEW && parts > 1) {
    // every block of the cluster has left its accumulators and its rows' maxima and sums; this one joins some of the columns
    __syncwarp();
    cluster_barrier();
    const int g = tid / BQ, r = tid % BQ;
    if (tid < WORKERS && r < ti.nq[0]) {
      const uint32_t ml = smem_u32(&part_share[FEW ? r : 0]), acc = smem_u32(smem) + (uint32_t)r * 16;
      float w[MAX_PARTS], m = -INFINITY, l = 0.f;
      float2 mls[MAX_PARTS];
#pragma unroll
      for (int p = 0; p < MAX_PARTS; ++p) {
        mls[p] = p < parts ? peer_ld2(peer_smem(ml, p)) : make_float2(-INFINITY, 0.f);
        m = fmaxf(m, mls[p].x);
      }
#pragma unroll
      for (int p = 0; p < MAX_PARTS; ++p) {
        w[p] = mls[p].x == -INFINITY ? 0.f : fast_exp2(mls[p].x - m);
        l = fmaf(mls[p].y, w[p], l);
      }
      const int head = row_head(r), tok = q_tok0 + row_query(r);
      if (a.has_sink) l += fast_exp2((a.sinks ? a.sinks[head] : a.sink_score) * LOG2E - m);
      float inv = l > 0.f ? 1.0f / l : 0.f;
      if (a.gate) inv *= a.gate[(long long)tok * a.nh + head];
      bf16* dst = (bf16*)a.out + ((long long)tok * a.nh + head) * HD;
      // runs of eight columns, the row's two threads in turn
      for (int c8 = (int)blockIdx.z * (HD / 8 / parts) + g; c8 < ((int)blockIdx.z + 1) * (HD / 8 / parts); c8 += GROUPS) {
        float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int p = 0; p < MAX_PARTS; ++p) {
          if (p < parts) {
            const uint32_t from = peer_smem(acc + (uint32_t)(2 * c8 * BQ) * 16, p);
            const float4 u = peer_ld4(from), v = peer_ld4(from + BQ * 16);
            o[0] = fmaf(w[p], u.x, o[0]); o[1] = fmaf(w[p], u.y, o[1]); o[2] = fmaf(w[p], u.z, o[2]); o[3] = fmaf(w[p], u.w, o[3]);
            o[4] = fmaf(w[p], v.x, o[4]); o[5] = fmaf(w[p], v.y, o[5]); o[6] = fmaf(w[p], v.z, o[6]); o[7] = fmaf(w[p], v.w, o[7]);
          }
        }
        uint4 v;
        v.x = pack_bf16(o[0] * inv, o[1] * inv);
        v.y = pack_bf16(o[2] * inv, o[3] * inv);
        v.z = pack_bf16(o[4] * inv, o[5] * inv);
        v.w = pack_bf16(o[6] * inv, o[7] * inv);
        *reinterpret_cast<uint4*>(dst + 8 * c8) = v;
      }
    }
    __syncwarp();
    cluster_barrier();                                      // nobody leaves while another block reads its shared memory
  }
  // every role comes here, also after a wait that ran out: copies in flight have been waited for above
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0) LLG_STAMP(5, 3, 0, blockIdx.x + gridDim.x * blockIdx.y);
  if (warp == 1) {
    warp_whole();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
  }
}

// ---- host side: tensor maps of the key/value sources ------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

// Boxes of 64 rows x 64 head dimensions (128 bytes, swizzled) out of [rows][hd] (cache pages: rows = pages x kv
// heads x 64 positions) or, with nkv > 0, out of [rows][nkv][hd] for one kv head (the step's packed keys or values).
bool kv_map(const void* base, long long rows, int nkv, int hd, CUtensorMap* result) {
  static std::map<std::tuple<const void*, long long, int, int>, CUtensorMap> cache;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  auto key = std::make_tuple(base, rows, nkv, hd);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *result = it->second;
    return true;
  }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  CUtensorMap m;
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r;
  if (nkv > 0) {
    cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)nkv, (cuuint64_t)rows};
    cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)nkv * hd * 2};
    cuuint32_t box[3] = {64, 1, (cuuint32_t)TK};
    r = fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    cuuint64_t dims[2] = {(cuuint64_t)hd, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)hd * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)TK};
    r = fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS) return false;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, m);
  *result = m;
  return true;
}

// Whether a step takes the FEW instance, and in what form: `parts` blocks that share a tile's keys (0: the other instance), `blocks` of 128 rows a
// key/value head.  From the tiles' keys and queries on the host (a.host_tiles; without them the other instance): the form whose blocks, spread over the
// multiprocessors, end soonest by the measured times below (us: a block, a key tile of a SPLIT block and of a PLAIN one, what parts add).  Parts only
// where all clusters are resident at once: in two rounds of them a step takes longer than with whole keys (96 blocks of 1,399 to 2,813
// keys: 39 us, in two parts 45; 16 of 810: 16 us, in four parts 13, in eight 25, as not quite sixteen clusters of eight fit).
// Measured, 32 query and 8 key/value heads of 128 (of 64): 83 queries behind 4,000 keys 41 us (40) in the other instance, 21 (19) in four parts; 5
// behind 6,000 (40 heads) 56 (54) and 16 (15) in eight; 300 behind 6,000 117 (111) and 65 (63) whole, behind 1,000 38 (35) and 24 (22); two
// of 200 behind 3,000 and 2,000 67 (64) and 43 (40); a prompt of 300 17 (15) and 12 (11), five of 11 to 51 10.8 (9.8) and 10.1 (8.9).  Where
// the rule stays with the other instance: a prompt of 2,048 67 us against 75, four of 1,100 (heads of 64) 98 against 110.  The times
// of a block and of a tile are those of heads of 128; heads of 64 are 5 to 15 % faster in both instances, so the comparison stands for them.
// Four turns of 83 queries behind 1,400 to 2,800 keys come out level by these times (33 us; 37 measured) and keep the other instance: with
// one count of parts for the step the longest sequence's blocks are as many as the shortest's.
struct FewForm { int parts, blocks; };
constexpr float BLOCK_US = 7.0f, SPLIT_TILE_US = 0.57f, PLAIN_TILE_US = 1.15f, JOIN_US = 4.5f;
FewForm few_form(const PrefillArgs& a, int sms) {
  const int per_kv = a.nh / a.nkv;
  FewForm best{0, 0};
  if (!a.host_tiles || (long long)a.nh * a.n_tiles > 8LL * sms) return best;
  // the grid goes by the sizes on the host, the kernel's rows by the device's: sizes that are not the step's must not leave rows out
  long long step_rows = 0;
  for (int t = 0; t < a.n_tiles; ++t) step_rows += a.host_tiles[2 * t + 1];
  if (step_rows != a.n_tokens) return best;
  float best_us = 0.f;
  int most = 0;
  for (int parts = 0; parts <= MAX_PARTS; parts = parts ? 2 * parts : 1) {
    float all = 0.f, longest = 0.f;
    long long blocks = 0;
    for (int t = 0; t < a.n_tiles; ++t) {
      const int end = a.host_tiles[2 * t], queries = a.host_tiles[2 * t + 1], pos0 = end - queries;
      const int first = a.window <= 0 ? 0 : a.chunked ? pos0 / a.window * a.window : (pos0 - a.window + 1 > 0 ? pos0 - a.window + 1 : 0);
      const int tiles = (end - first / TK * TK + TK - 1) / TK, n = (queries * per_kv + BQ - 1) / BQ;
      const long long same = parts ? (long long)parts * n * a.nkv : a.nh;
      const float us = BLOCK_US + (parts > 1 ? JOIN_US : 0.f) +
                       (parts ? (tiles + parts - 1) / parts * SPLIT_TILE_US : tiles * (queries > BQ ? PLAIN_TILE_US : SPLIT_TILE_US));
      all += us * same;
      blocks += same;
      if (us > longest) longest = us;
      if (n > most) most = n;
    }
    if (parts > 1 && blocks > (parts == 2 ? sms - sms / 16 : parts == 4 ? sms - sms / 7 : sms - sms * 3 / 10)) break;
    const float us = blocks <= sms ? longest : fmaxf(longest, all / sms) + 0.3f * longest;
    if (parts == 0 || us < 0.95f * best_us) {
      best.parts = parts;
      best_us = us;
    }
  }
  best.blocks = most;
  return best;
}

// Shared memory of a block: queries, keys and values.  The blocks of a cluster wait for one another while each holds all of its multiprocessor's
// tensor memory, so no two such blocks may share a multiprocessor (each could wait for ever for what the other's cluster holds, and
// tcgen05.alloc and the cluster's barrier have no limit): they ask for more than half of its 228 KB.  (The pair products, the other kernel
// whose blocks wait for one another with tensor memory in hand, take more than half too.)
constexpr int ALONE_SMEM = 120 * 1024;
constexpr int block_smem(int hd, int q_tiles, int parts) {
  const int tiles = hd / 64 * 128 * (q_tiles * BQ + (KST + VST) * TK);
  return parts > 1 && tiles < ALONE_SMEM ? ALONE_SMEM : tiles;
}

template <int HD, bool MAPS, bool FEW>
int launch(const PrefillArgs& a, FewForm form, cudaStream_t stream) {
  constexpr int Q_TILES = MAPS || FEW ? 1 : GROUPS, MOST_SMEM = block_smem(HD, Q_TILES, FEW ? MAX_PARTS : 1);
  static_assert(!FEW || BQ * HD * 4 <= block_smem(HD, Q_TILES, 1), "a block's accumulators take the place of its queries, keys and values");
  const int smem = block_smem(HD, Q_TILES, form.parts);
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel<HD, MAPS, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SMEM);
    if (e != cudaSuccess) return llg_fail("attn_prefill_tc: shared memory %d: %s", MOST_SMEM, cudaGetErrorString(e));
    configured = true;
  }
  CUtensorMap mkp, mvp, mkn, mvn;
  const long long page_rows = (long long)a.n_pages * a.nkv * TK;
  if (!kv_map(a.k_pages, page_rows, 0, HD, &mkp) || !kv_map(a.v_pages, page_rows, 0, HD, &mvp) ||
      !kv_map(a.k_new, a.n_tokens, a.nkv, HD, &mkn) || !kv_map(a.v_new, a.n_tokens, a.nkv, HD, &mvn))
    return llg_fail("attn_prefill_tc: cuTensorMapEncodeTiled failed or is not available");
  cudaError_t le;
  if (FEW) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.nkv * form.blocks), a.n_tiles, form.parts);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = form.parts;
    cfg.attrs = llg_pdl_enabled() ? attr : attr + 1;
    cfg.numAttrs = (llg_pdl_enabled() ? 1 : 0) + (form.parts > 1 ? 1 : 0);
    le = cudaLaunchKernelEx(&cfg, attn_prefill_tc_kernel<HD, MAPS, FEW>, mkp, mvp, mkn, mvn, a);
  } else {
    le = llg_launch(attn_prefill_tc_kernel<HD, MAPS, FEW>, dim3(a.nh, a.n_tiles), dim3(THREADS), (size_t)smem, stream, mkp, mvp, mkn, mvn, a);
  }
  if (le != cudaSuccess) return llg_fail("attn_prefill_tc: launch: %s", cudaGetErrorString(le));
  return llg_check_launch("attn_prefill_tc");
}

}  // namespace

// 1 when this kernel takes the head size (bfloat16 only): 64 or 128.
LLG_API int llg_attn_tc_supported(int hd) { return hd == 64 || hd == 128; }

// Blocks that share a tile's keys for these sizes (n_tiles, n_tokens, nh, nkv, window, chunked and host_tiles of `args`) on a GPU of `sms` multiprocessors;
// 0 where the step takes the instance for long prompts.
LLG_API int llg_attn_prefill_parts(const PrefillArgs* args, int sms) { return few_form(*args, sms).parts; }

// Bytes of shared memory that such a block asks for.
LLG_API int llg_attn_prefill_few_smem(int hd, int parts) { return block_smem(hd, 1, parts); }

LLG_API int llg_attn_prefill_tc(const PrefillArgs* args, cudaStream_t stream) {
  const PrefillArgs& a = *args;
  LLG_REQUIRE(llg_attn_tc_supported(a.hd), "attn_prefill_tc: head_dim %d is neither 64 nor 128", a.hd);
  LLG_REQUIRE(a.nh > 0 && a.nkv > 0 && a.nh % a.nkv == 0, "attn_prefill_tc: %d heads are no multiple of %d key/value heads",
              a.nh, a.nkv);
  LLG_REQUIRE(a.window >= 0 && a.ring_pages > 0 && a.table_width >= a.ring_pages, "attn_prefill_tc: bad cache geometry");
  LLG_REQUIRE(a.n_tiles <= 65535, "attn_prefill_tc: %d query tiles in one step are more than a grid takes (65535)", a.n_tiles);
  LLG_REQUIRE(a.scale > 0.f, "attn_prefill_tc: the softmax scale must be positive");
  LLG_REQUIRE(a.vd == 0 || a.vd == a.hd, "attn_prefill_tc: value heads of %d elements beside key heads of %d", a.vd, a.hd);
  LLG_REQUIRE(a.n_tokens > 0 && a.n_pages > 0, "attn_prefill_tc: needs the sizes of the packed rows and of the pages");
  LLG_REQUIRE(((uintptr_t)a.k_new % 16) == 0 && ((uintptr_t)a.v_new % 16) == 0 && ((uintptr_t)a.k_pages % 16) == 0 &&
                  ((uintptr_t)a.v_pages % 16) == 0,
              "attn_prefill_tc: keys and values must be 16-byte aligned");
  if (a.n_tiles <= 0) return 0;
  LLG_REQUIRE(a.maps == 0 || a.maps == 2, "attn_prefill_tc: %d maps (0 or 2)", a.maps);
  if (a.maps == 2) {
    LLG_REQUIRE(!a.has_sink && !a.gate && a.map_eps > 0.f, "attn_prefill_tc: two maps go with neither a sink nor gates");
    return a.hd == 64 ? launch<64, true, false>(a, {}, stream) : launch<128, true, false>(a, {}, stream);
  }
  const FewForm form = few_form(a, llg_sm_count());
  if (form.parts > 0) return a.hd == 64 ? launch<64, false, true>(a, form, stream) : launch<128, false, true>(a, form, stream);
  return a.hd == 64 ? launch<64, false, false>(a, {}, stream) : launch<128, false, false>(a, {}, stream);
}

// Error code recorded when a wait ran out (0 = none); clears it.  Synchronises the device.
LLG_API int llg_attn_tc_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(g_error, &zero, sizeof(int));
  return v;
}
