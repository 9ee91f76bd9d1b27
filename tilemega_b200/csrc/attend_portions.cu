// Attention of prompt portions in bf16 ragged steps on tcgen05: scores and weighted sums of 128 rows against 128 keys at a
// time, accumulators (and the weights, as an operand) in tensor memory.
#include <algorithm>

#include "attend.cuh"
#include "tensor_map.h"
#include "umma.cuh"
#include "wide.cuh"

namespace tmb {
namespace {

constexpr int kTileKeys = 128;                 // keys per block
constexpr int kChunk = 128 * 128;              // bytes of 128 rows x 64 columns, 128-byte swizzled
constexpr int kHalfKeys = kTileKeys / 2, kHalfChunk = kChunk / 2;   // values come and go by half blocks
constexpr int kRun = kRaggedBlock;             // keys that lie together: one copy's rows
constexpr int kRuns = kTileKeys / kRun;
constexpr float kSlack = 8.f;                  // log2 of how far a row's weights may grow before its sums are scaled down
constexpr uint32_t kUmmaBTransposed = 1u << 16;   // instruction descriptor: B lies transposed
constexpr unsigned kWaitLoader = 0xA7700001u, kWaitMma = 0xA7700002u, kWaitSoftmax = 0xA7700003u;

template <int KC, int VC, int TILES> struct PortionShape {
  static constexpr int kThreads = 32 * 4 * (TILES + 1);
  static constexpr int kKeyStages = 2, kValueStages = KC > 2 && TILES > 1 ? 2 : 4;   // (values by half blocks)
  static constexpr int kSmem = (TILES * KC + kKeyStages * KC) * kChunk + kValueStages * VC * kHalfChunk + 1024;   // (registers allow one CTA an SM in any form)
  static constexpr int kColumns = TILES == 2 ? 512 : 256;
  static constexpr int kSums = 128 * TILES;                                  // first column of the weighted sums
};

// Tensor memory by 32 columns, with the wait apart, so that several are in flight; what was loaded may be used behind
// loads_done() and loaded().
__device__ __forceinline__ void load_columns(uint32_t at, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(at)
      : "memory");
}
__device__ __forceinline__ void loads_done() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void loaded(float* v) {     // (keeps uses of v behind the wait)
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+f"(v[i]));
}
__device__ __forceinline__ void store_columns(uint32_t at, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(at),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void store_columns16(uint32_t at, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(at), "f"(v[0]),
      "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]),
      "f"(v[14]), "f"(v[15])
      : "memory");
}
__device__ __forceinline__ void stores_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Two fp32 numbers at a time.
__device__ __forceinline__ uint64_t two(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void apart(uint64_t v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
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

// Rows of a tile are (token, query head of the unit) pairs, token-major, as in attend_tiles; a CTA holds TILES tiles of 128
// rows. KC, VC: 64-column chunks of keys and values. Warps 0 .. 4 TILES - 1: a thread a row, softmax and output. Of the last
// four, one issues the products, one copies keys and values (runs of 16 keys, as the pools hold them), K one block ahead of V.
//
// A row's weights go back into the columns of its scores, 32 keys as 16 words of bf16 heads and 16 words of remainders, and
// enter the second product from there, head and remainder one after the other: about 16 bits of every weight. What a row's
// weights are relative to follows its maximum only in steps of 2^8, so that its sums are seldom scaled.
//
// Bound by the tensor pipe and the softmax between its two products: the pipe is active half of the time behind 4096 positions, 30 % at 2048
// rows from the start, where a CTA's start and end weigh more; a third of the products are the remainders'. 2048 tokens, 32 heads of
// 128 over 8 key heads: 75 us where attend_tiles takes 337; 2048 tokens behind 4096, 32 heads of 192 and 128: 290 us for 1770 (300 GFLOP executed;
// two rounds of CTAs). What that took: keys by TMA instead of 16-byte copies of three warps (98 and 518 us with those), a warp that stays together
// around the issuing lane (90 and 340 without), values by half blocks where shared memory holds just one, output rows written by eight lanes each.
template <int KC, int VC, int TILES>
__global__ void __launch_bounds__(PortionShape<KC, VC, TILES>::kThreads, 1) attend_portions(StepRows r, AttendParams p, const __grid_constant__ CUtensorMap k_map,
                                                                                           const __grid_constant__ CUtensorMap v_map, unsigned* status, bool vector_rows) {
  using Shape = PortionShape<KC, VC, TILES>;
  constexpr int KS = Shape::kKeyStages, VS = Shape::kValueStages;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t k_full[KS], k_empty[KS], v_full[VS], v_empty[VS], v_landed, s_full[TILES], p_full[TILES], o_full[TILES], q_full[TILES];
  __shared__ uint32_t tmem_slot;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* ks = smem + TILES * KC * kChunk;
  unsigned char* vs = ks + KS * KC * kChunk;
  dependency_wait();
  allow_dependents();
  const Entry e = r.entry[blockIdx.z];
  if (e.rows == 1) return;
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int group = blockIdx.x / p.subs, first_head = (blockIdx.x % p.subs) * p.sub_heads;
  const int gq = min(p.sub_heads, p.heads / p.kv_heads - first_head);
  const int head0 = group * (p.heads / p.kv_heads) + first_head;
  const int per_tile = 128 / gq;
  const int t0 = (gridDim.y - 1 - blockIdx.y) * TILES * per_tile;      // (the last tokens see the most keys: their CTAs start first)
  if (t0 >= e.rows) return;
  const int tokens = min(TILES * per_tile, e.rows - t0);
  const int p0 = e.first_position + t0, p1 = p0 + tokens - 1;
  const int low = max(0, p0 - p.window + 1), kept = min(p.keep, low);
  const int start = p.context ? low : low / kRun * kRun;               // (pools are read by whole runs)
  const int kept_blocks = (kept + kTileKeys - 1) / kTileKeys, blocks = kept_blocks + (p1 + 1 - start + kTileKeys - 1) / kTileKeys;
  auto block_base = [&](int b) { return b < kept_blocks ? b * kTileKeys : start + (b - kept_blocks) * kTileKeys; };
  auto block_limit = [&](int b) { return b < kept_blocks ? kept : p1 + 1; };
  // does any row of the tile see keys of the block
  auto active = [&](int tile, int b) {
    if (tile * per_tile >= tokens) return false;
    if (b < kept_blocks) return true;
    const int first = block_base(b), q0 = p0 + tile * per_tile, q1 = min(q0 + per_tile - 1, p1);
    return first <= q1 && (q0 - (first + kTileKeys - 1) < p.window || first < p.keep);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < KS; ++i) mbar_init(&k_full[i], 1), mbar_init(&k_empty[i], 1);
    for (int i = 0; i < VS; ++i) mbar_init(&v_full[i], 1), mbar_init(&v_empty[i], 1);
    for (int i = 0; i < TILES; ++i) mbar_init(&s_full[i], 1), mbar_init(&p_full[i], 128), mbar_init(&o_full[i], 1), mbar_init(&q_full[i], 128);
    mbar_init(&v_landed, 1);
    mbar_fence_init();
    prefetch_map(&k_map);
    prefetch_map(&v_map);
  }
  if (warp == 4 * TILES) tmem_alloc(&tmem_slot, Shape::kColumns);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;

  // (twelve warps of 168 registers share them out: 208 for softmax, 88 for the others)
  if (warp >= 4 * TILES) {
    if constexpr (TILES == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 4 * TILES + 1) {
      // ---- keys and values: a lane a run ----
      const int* table = r.block_table + size_t(e.slot) * r.max_blocks;
      const int context = p.context ? p.context[blockIdx.z] - max(0, e.first_position - p.window + 1) : 0;
      auto place = [&](int b) {                        // of the lane's run of a block: head of a pool block, or row of the context
        const int j = block_base(b) + kRun * (lane % kRuns);
        if (p.context) return context + j;
        return key_row(table, j, r) / kRun * p.kv_heads + group;
      };
      // up to `most` runs of a block from its run `first` on, as `chunks` pieces of 64 columns
      auto issue = [&](const CUtensorMap* map, unsigned char* to, int chunks, int chunk_bytes, uint64_t* full, int b, int first, int most, int at) {
        const int runs = min(max((block_limit(b) - block_base(b) + kRun - 1) / kRun - first, 0), most);
        if (lane == 0) mbar_expect_tx(full, uint32_t(runs * chunks * kRun * 128));
        __syncwarp();
        const int run = lane - first;
        if (run >= 0 && run < runs)
          for (int c = 0; c < chunks; ++c) tma_load_3d(to + c * chunk_bytes + run * kRun * 128, map, 64 * c, p.context ? group : 0, at, full);
      };
      auto there = [&](int b, int half) { return max(0, block_limit(b) - block_base(b) - half * kHalfKeys); };      // values of a half
      auto wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_bounded(bar, parity, status, kWaitLoader)) != 0; };
      int at_value = 0, at_key = place(0), at_next = blocks > 1 ? place(1) : 0;      // places are fetched one turn ahead
      fill_blocks<KS, VS>(
          blocks, [&](int b, int s) { issue(&k_map, ks + s * KC * kChunk, KC, kChunk, &k_full[s], b, 0, kRuns, at_key); },
          [&](int b, int half, int s) {
            const bool part = there(b, half) < kHalfKeys;
            issue(&v_map, vs + s * VC * kHalfChunk, VC, kHalfChunk, part ? &v_landed : &v_full[s], b, half * kRuns / 2, kRuns / 2, at_value);
            return part;
          },
          [&](uint32_t parity) { return wait(&v_landed, parity); },
          [&](int b, int half, int s) {                // what lies behind the last key, or was there before, may be no number
            const int held = there(b, half);
            for (int i = lane; i < (kHalfKeys - held) * 8 * VC; i += 32)
              *reinterpret_cast<uint4*>(vs + s * VC * kHalfChunk + (i / 8 % VC) * kHalfChunk + (held + i / (8 * VC)) * 128 + (i & 7) * 16) = make_uint4(0, 0, 0, 0);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&v_full[s]);
          },
          [&](int b) {
            at_value = at_key;
            at_key = at_next;
            at_next = b + 3 < blocks ? place(b + 3) : 0;
          },
          [&](int s, uint32_t parity) { return wait(&k_empty[s], parity); }, [&](int s, uint32_t parity) { return wait(&v_empty[s], parity); },
          [&](int s, uint32_t parity) { drained(&k_full[s], parity); }, [&](int s, uint32_t parity) { drained(&v_full[s], parity); },
          [&](uint32_t parity) { drained(&v_landed, parity); });
    } else if (warp == 4 * TILES) {
      // ---- products: the warp walks along together, one lane issues (what decides its way is taken from votes and shuffles, so that
      // the compiler knows it to be the warp's: operands of the products are then formed once, not per lane) ----
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
      const int count = __shfl_sync(0xffffffffu, blocks, 0);
      const uint32_t score_idesc = umma_idesc_bf16(128, kTileKeys), sum_idesc = umma_idesc_bf16(128, VC * 64) | kUmmaBTransposed;
      const uint64_t q_desc = umma_desc_k_sw128(smem_u32(smem), 1024), k_desc = umma_desc_k_sw128(smem_u32(ks), 1024);
      const uint64_t v_desc = umma_desc_mn_sw128(smem_u32(vs), kHalfChunk, 1024);
      const uint32_t q_low = uint32_t(q_desc), k_low = uint32_t(k_desc), v_low = uint32_t(v_desc), high = uint32_t(k_desc >> 32);   // (the same for all)
      bool ok = true;
      for (int t = 0; t < TILES; ++t) ok = __all_sync(0xffffffffu, ok && wait_bounded(&q_full[t], 0, status, kWaitMma));
      unsigned started = 0;                            // bit per tile: its sums hold something
      int waits[TILES] = {};
      for (int b = 0; b <= count && ok; ++b) {
        if (b < count) ok = wait_bounded(&k_full[b % KS], (b / KS) & 1, status, kWaitMma);
        ok = __all_sync(0xffffffffu, ok);
#pragma unroll
        for (int t = 0; t < TILES; ++t) {
          const bool sum = b > 0 && __any_sync(0xffffffffu, active(t, b - 1));
          if (ok && sum) {
            ok = __all_sync(0xffffffffu, wait_bounded(&p_full[t], waits[t] & 1, status, kWaitMma));
            ++waits[t];
          }
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (b == 0 || !ok) break;
            const int stage = (2 * b - 2 + half) % VS, turn = (2 * b - 2 + half) / VS;
            if (t == 0) ok = __all_sync(0xffffffffu, wait_bounded(&v_full[stage], turn & 1, status, kWaitMma));   // (before the first tile that reads them)
            if (!ok) break;
            tcgen05_fence_after();
            if (elect_one()) {
              if (sum) {
                const uint32_t v = v_low + stage * (VC * kHalfChunk / 16), weights = tmem + t * 128 + 64 * half, sums = tmem + Shape::kSums + t * VC * 64;
#pragma unroll
                for (int step = 0; step < kHalfKeys / 16; ++step) {
                  umma_step_tmem(sums, weights + 32 * (step / 2) + 8 * (step & 1), v + step * (2048 / 16), high, sum_idesc, half || step || (started >> t & 1u));
                  umma_step_tmem(sums, weights + 32 * (step / 2) + 8 * (step & 1) + 16, v + step * (2048 / 16), high, sum_idesc, true);
                }
              }
              if (t == TILES - 1) umma_commit(&v_empty[stage]);
            }
            __syncwarp();
          }
          if (!ok) break;
          if (sum) started |= 1u << t;
          if (b < count && __any_sync(0xffffffffu, active(t, b))) {
            if (elect_one()) {
              const uint32_t q = q_low + t * (KC * kChunk / 16), k = k_low + (b % KS) * (KC * kChunk / 16);
#pragma unroll
              for (int step = 0; step < KC * 4; ++step)
                umma_step(tmem + t * 128, q + (step / 4) * (kChunk / 16) + 2 * (step % 4), k + (step / 4) * (kChunk / 16) + 2 * (step % 4), high, score_idesc, step != 0);
              umma_commit(&s_full[t]);
            }
            __syncwarp();
          }
        }
        if (b < count && elect_one()) umma_commit(&k_empty[b % KS]);
        __syncwarp();
      }
      if (elect_one())
        for (int t = 0; t < TILES; ++t) umma_commit(&o_full[t]);
      __syncwarp();
      // (also behind a wait that gave up: tensor memory is freed once no product runs)
      for (int t = 0; t < TILES; ++t) drained(&o_full[t], 0);
      __syncwarp();
    }
  } else {
    if constexpr (TILES == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // ---- softmax and output: a thread a row; first a warp brings its rows' queries ----
    const int tile = warp / 4, m = (warp % 4) * 32 + lane;
    {
      constexpr int kLanes = KC > 2 ? 32 : KC * 8, kAtOnce = 32 / kLanes;      // lanes and rows of a load
      const bool wide = (p.dim & 7) == 0 && (p.q_head & 7) == 0 && (p.proj_stride & 7) == 0 && (reinterpret_cast<uintptr_t>(p.proj) & 15) == 0;
      const int piece = lane % kLanes, c = piece * 8;
#pragma unroll 8
      for (int i = 0; i < 32; i += kAtOnce) {
        const int row = (warp % 4) * 32 + i + lane / kLanes, token = row / gq, t = tile * per_tile + token;
        const bf16* head = p.proj + size_t(e.first_row + t0 + min(t, tokens - 1)) * p.proj_stride + size_t(head0 + row - token * gq) * p.q_head;
        uint4 word = make_uint4(0, 0, 0, 0);
        if (token < per_tile && t < tokens && c < p.dim) {
          if (wide) {
            word = *reinterpret_cast<const uint4*>(head + c);
          } else {
            bf16 e8[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) e8[j] = c + j >= p.dim ? __float2bfloat16_rn(0.f) : head[c + j];
            word = *reinterpret_cast<uint4*>(e8);
          }
        }
        if (piece < KC * 8) *reinterpret_cast<uint4*>(smem + (tile * KC + piece / 8) * kChunk + row * 128 + (((piece & 7) ^ (row & 7)) << 4)) = word;
      }
      fence_proxy_async();
      mbar_arrive(&q_full[tile]);
    }
    const uint32_t scores = tmem + (uint32_t((warp % 4) * 32) << 16) + tile * 128, sums = scores - tile * 128 + Shape::kSums + tile * VC * 64;
    const int t = tile * per_tile + m / gq;
    const bool live = m / gq < per_tile && t < tokens;
    const int position = p0 + min(t, tokens - 1);
    const int least = __reduce_min_sync(0xffffffffu, position), most = __reduce_max_sync(0xffffffffu, position);
    float ref = -INFINITY, sum = 0.f;
    bool ok = true, first = true;
    int waits = 0;
    for (int b = 0; b < blocks; ++b) {
      if (!active(tile, b)) continue;
      ok = ok && wait_bounded(&s_full[tile], waits & 1, status, kWaitSoftmax);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ++waits;
      tcgen05_fence_after();
      const int base = block_base(b), limit = block_limit(b), begin = b < kept_blocks ? 0 : low;
      const bool whole = base >= begin && base + kTileKeys <= limit && base + kTileKeys - 1 <= least && most - base < p.window;
      // which of 32 keys from `at` the row sees
      auto seen = [&](int at) {
        auto below = [](int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; };
        const uint32_t there = below(min(limit, position + 1) - at) & ~below(begin - at);
        return there & (~below(position - p.window + 1 - at) | below(p.keep - at));
      };
      float v[kTileKeys];
#pragma unroll
      for (int c = 0; c < kTileKeys; c += 32) load_columns(scores + c, v + c);
      loads_done();
#pragma unroll
      for (int c = 0; c < kTileKeys; c += 32) loaded(v + c);
      if (!whole) {
#pragma unroll
        for (int c = 0; c < kTileKeys; c += 32) {
          const uint32_t bits = seen(base + c);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[c + i] = bits >> i & 1u ? v[c + i] : -INFINITY;
        }
      }
      float h[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
      for (int i = 4; i < kTileKeys; ++i) h[i & 3] = fmaxf(h[i & 3], v[i]);
      const float high = fmaxf(fmaxf(h[0], h[1]), fmaxf(h[2], h[3])) * p.scale_log2;
      if (__any_sync(0xffffffffu, high > ref + kSlack)) {
        const float now = fmaxf(high, ref), fade = ref == -INFINITY ? 0.f : ex2(ref - now);
        sum *= fade;
        if (!first) {
#pragma unroll 1
          for (int c = 0; c < VC * 64; c += 16) {
            float o[16];
            tmem_load_16(sums + c, o);
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] *= fade;
            store_columns16(sums + c, o);
          }
        }
        ref = now;
      }
      first = false;
      const float shift = ref == -INFINITY ? 0.f : ref;      // (masked scores of -inf weigh nothing)
      const uint64_t scale2 = two(p.scale_log2, p.scale_log2), shift2 = two(-shift, -shift);
      uint64_t add[4] = {};
#pragma unroll
      for (int c = 0; c < kTileKeys; c += 32) {
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float x, y;
          apart(fma2(two(v[c + 2 * i], v[c + 2 * i + 1]), scale2, shift2), x, y);
          const uint64_t weight = two(ex2(x), ex2(y));
          apart(weight, x, y);
          add[i & 3] = add2(add[i & 3], weight);
          const uint32_t head = pack(x, y);
          float rx, ry;
          apart(add2(weight, two(-bf_lo(head), -bf_hi(head))), rx, ry);
          w[i] = head;
          w[16 + i] = pack(rx, ry);
        }
        store_columns(scores + c, w);
      }
      stores_done();
      float s0, s1;
      apart(add2(add2(add[0], add[1]), add2(add[2], add[3])), s0, s1);
      sum += s0 + s1;
      tcgen05_fence_before();
      mbar_arrive(&p_full[tile]);
    }
    if (tile * per_tile < tokens) {
      ok = ok && wait_bounded(&o_full[tile], 0, status, kWaitSoftmax);
      ok = __all_sync(0xffffffffu, ok);
      tcgen05_fence_after();
      const int head = head0 + m % gq;
      const float sink = p.sink_of(head);
      float inv = 1.f / sum;
      if (sink != -INFINITY) {                       // (a null key that stands above every key takes the maximum's place)
        const float high = fmaxf(ref, sink), f = ex2(ref - high);
        inv = f / fmaf(sum, f, ex2(sink - high));
      }
      const size_t row = size_t(e.first_row + t0 + (live ? t : 0)), column = size_t(head) * p.vdim;
      bf16* dst = p.out + row * p.out_stride + column;
      const bf16* gate = p.proj + row * p.proj_stride + (p.gate_at >= 0 ? p.gate_at : 0) + column;
      // rows pass through the tile's queries' place, 32 columns at a time, so that eight lanes write a row
      unsigned char* own = smem + tile * KC * kChunk + (warp % 4) * 4096;
      bf16* to[8];                                     // of rows lane / 8, lane / 8 + 4, ... of the warp's
      const bf16* gate_at[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m4 = (warp % 4) * 32 + 4 * i + (lane >> 3), token = m4 / gq, t4 = tile * per_tile + token, head4 = head0 + m4 - token * gq;
        const bool there = ok && token < per_tile && t4 < tokens;
        const size_t row4 = size_t(e.first_row + t0 + (there ? t4 : 0)), column4 = size_t(head4) * p.vdim + 4 * (lane & 7);
        to[i] = there ? p.out + row4 * p.out_stride + column4 : nullptr;
        gate_at[i] = p.proj + row4 * p.proj_stride + max(p.gate_at, 0) + column4;
      }
#pragma unroll 1
      for (int c = 0; c < VC * 64 && c < p.vdim; c += 32) {
        float v[32];
        uint2 gates[8];
        const bool here = c + 4 * (lane & 7) < p.vdim;
        if (vector_rows && p.gate_at >= 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (to[i] && here) gates[i] = *reinterpret_cast<const uint2*>(gate_at[i] + c);
        }
        tmem_load_32(sums + c, v);
        if (vector_rows) {
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(own + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_float4(v[4 * i] * inv, v[4 * i + 1] * inv, v[4 * i + 2] * inv, v[4 * i + 3] * inv);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row4 = 4 * i + (lane >> 3);
            float4 y = *reinterpret_cast<const float4*>(own + row4 * 128 + (((lane & 7) ^ (row4 & 7)) << 4));
            if (p.gate_at >= 0) {
              y.x = __fdividef(y.x, 1.f + ex2(-1.4426950408889634f * bf_lo(gates[i].x)));
              y.y = __fdividef(y.y, 1.f + ex2(-1.4426950408889634f * bf_hi(gates[i].x)));
              y.z = __fdividef(y.z, 1.f + ex2(-1.4426950408889634f * bf_lo(gates[i].y)));
              y.w = __fdividef(y.w, 1.f + ex2(-1.4426950408889634f * bf_hi(gates[i].y)));
            }
            if (to[i] && here) *reinterpret_cast<uint2*>(to[i] + c) = make_uint2(pack(y.x, y.y), pack(y.z, y.w));
          }
        } else if (live && ok) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c + i < p.vdim) {
              float y = v[i] * inv;
              if (p.gate_at >= 0) y *= sigmoid(__bfloat162float(gate[c + i]));
              dst[c + i] = __float2bfloat16_rn(y);
            }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 4 * TILES) {
    __syncwarp();
    tmem_dealloc(tmem, Shape::kColumns);
  }
}

template <int KC, int VC, int TILES>
int LaunchPortions(const Queue& q, const StepRows& r, const AttendParams& p, const CUtensorMap& k_map, const CUtensorMap& v_map, int tiles) {
  auto aligned = [](const void* at) { return (reinterpret_cast<uintptr_t>(at) & 7) == 0; };
  const bool vector_rows = p.vdim % 4 == 0 && p.out_stride % 4 == 0 && p.proj_stride % 4 == 0 && (p.gate_at < 0 || p.gate_at % 4 == 0) && aligned(p.out) &&
                           aligned(p.proj);
  return int(Launch(attend_portions<KC, VC, TILES>, dim3(unsigned(p.kv_heads * p.subs), unsigned((tiles + TILES - 1) / TILES), unsigned(r.entries)),
                    dim3(PortionShape<KC, VC, TILES>::kThreads), PortionShape<KC, VC, TILES>::kSmem, q.stream, q.chained, r, p, k_map, v_map, q.status,
                    vector_rows));
}

template <int KC, int VC> int PortionsWith(const Queue& q, const StepRows& r, const AttendParams& p, const CUtensorMap& k_map, const CUtensorMap& v_map) {
  const int per_tile = 128 / p.sub_heads, tiles = (r.longest + per_tile - 1) / per_tile;
  // Two tiles a CTA share its keys and overlap one's softmax with the other's products. Where both ways are one round of CTAs, two take
  // 1.1 to 1.2 times as long as one (8B shape, 431 rows 33 us for 30, behind 2000 67 for 59; 16 heads of 192, 1000 rows 68 for 58): one tile
  // each. At half the rounds 0.6 to 0.9 times (2048 rows 75 for 125, 1000 rows 43 for 53; 32 heads of 192, 700 rows 42 for 47): two.
  const int units = p.kv_heads * p.subs * std::max(1, r.entries - r.singles);
  auto rounds = [&](int count) { return (count + q.sm_count - 1) / q.sm_count; };
  if (16 * rounds((tiles + 1) / 2 * units) <= 10 * rounds(tiles * units)) return LaunchPortions<KC, VC, 2>(q, r, p, k_map, v_map, tiles);
  return LaunchPortions<KC, VC, 1>(q, r, p, k_map, v_map, tiles);
}

template <int KC, int VC> cudaError_t RaisePortions() {
  const cudaError_t err = cudaFuncSetAttribute(attend_portions<KC, VC, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, PortionShape<KC, VC, 1>::kSmem);
  if (err != cudaSuccess) return err;
  return cudaFuncSetAttribute(attend_portions<KC, VC, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, PortionShape<KC, VC, 2>::kSmem);
}

// [z][y][dim] as boxes of 64 columns and 16 rows along y or z; columns behind `dim` arrive as zeros.
bool EncodeRuns(CUtensorMap* map, const void* base, uint64_t dim, uint64_t y, uint64_t y_stride, uint64_t z, uint64_t z_stride, uint32_t box_y, uint32_t box_z) {
  EncodeTiled encode = TensorMapEncoder();
  if (!encode) return false;
  const cuuint64_t dims[3] = {dim, y, z}, strides[2] = {y_stride * 2, z_stride * 2};
  const cuuint32_t box[3] = {64, box_y, box_z}, steps[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool EncodePool(CUtensorMap* map, const void* pool, uint64_t heads, uint64_t dim) {
  return EncodeRuns(map, pool, dim, kRaggedBlock, dim, heads, dim * kRaggedBlock, kRaggedBlock, 1);
}
bool EncodeContext(CUtensorMap* map, const void* rows, uint64_t heads, uint64_t dim, uint64_t count, uint64_t stride) {
  return EncodeRuns(map, rows, dim, heads, dim, count, stride, 1, kRaggedBlock);
}

int AttendPortions(const Queue& q, const StepRows& r, const AttendParams& given, const CUtensorMap* k_map, const CUtensorMap* v_map, bool* done) {
  *done = false;
  if (!k_map || !v_map) return 0;
  AttendParams p = given;
  p.window = std::min(p.window, 1 << 29);            // (differences of positions and windows stay in range)
  if (!(p.scale_log2 > 0.f) || p.pool_dim > 192 || p.v_pool_dim > 128) return 0;
  *done = true;
  if (p.pool_dim <= 64 && p.v_pool_dim <= 64) return PortionsWith<1, 1>(q, r, p, *k_map, *v_map);
  return p.pool_dim <= 128 ? PortionsWith<2, 2>(q, r, p, *k_map, *v_map) : PortionsWith<3, 2>(q, r, p, *k_map, *v_map);
}

int PreparePortions() {
  cudaError_t err = RaisePortions<1, 1>();
  if (err == cudaSuccess) err = RaisePortions<2, 2>();
  if (err == cudaSuccess) err = RaisePortions<3, 2>();
  return int(err);
}

}  // namespace tmb
