// The FastScan sums of a batch of queries as an integer contraction on the
// tensor cores (sm_100a).
//
// A vector's LUT sum for a query is sum_g LUT[q][g][code(v, g)]: a row of the
// one-hot matrix of its nibbles (16 columns per nibble, a single 1 each) times
// the query's LUT bytes, which already lie K-major in the order [group][high
// nibble's 16 entries, low nibble's 16]. u8 x u8 products with s32 accumulation
// (tcgen05.mma kind::i8) give exactly the integers the lookup kernels add up,
// and the epilogue flushes them into f32 every 256 byte groups with the same
// fused multiply-add (search_avx2.cpp:24-48), so scores and top-k are equal bit
// for bit to tq_scan.cu's.
//
// A pair of CTAs (cta_group::2) owns a tile of 256 vectors (128 per CTA) x N
// queries (N <= 192). Per stage of 8 byte groups (256 bytes of K; 512 for at most
// 64 queries, and 3-bit codes take half the K per group):
//   * TMA loads bring each CTA's half of the N queries' LUT bytes to shared
//     memory (K-major, 128-byte swizzle);
//   * eight producer warps, two sets of four, read the codes, build each vector's
//     one-hot row in registers (its own TMEM lane) and store it to TMEM;
//   * one thread of the pair issues a K = 32 MMA per byte group (A in TMEM, B in
//     shared memory).
// The one-hot operand lives in TMEM because shared memory could not carry it as
// well: writing and reading it there next to the LUT tiles takes all of the 128
// bytes per clock at N = 256 (measured: 631 clocks per stage instead of 512).
// Accumulators are double-buffered in TMEM per 256-group batch (2 x 192 columns,
// the other 128 hold two one-hot stages); eight warps per CTA read them back,
// keep the f32 sums in registers across batches (96 queries each), and append
// scores at or above the query's threshold to a list, cut back to the top k when
// it fills up.
#include <cfloat>
#include <algorithm>

#include <cuda.h>

#include "tq_bucket.h"
#include "tq_device.cuh"
#include "tq_kernels.h"
#include "tq_tc.cuh"

namespace vcb {
namespace {

constexpr int kMaxN = 192;              // queries per tile
constexpr int kHalfN = kMaxN / 2;       // LUT rows per CTA; queries per epilogue warp
constexpr int kTileB = kHalfN * 128;    // LUT bytes per CTA and 128 bytes of K
constexpr int kStagesB = 6;
constexpr int kMaxStagesA = 4;
constexpr int kPieceCols = 16;          // TMEM columns a producer stores at a time
// Codes: 32 byte groups (32 words of 128 vectors each) per chunk.
constexpr int kChunkGroups = 32;
constexpr int kTileC = kChunkGroups * 128;
constexpr int kStagesC = 4;
constexpr int kTmemCols = 512;
constexpr int kPairVectors = 256;
// Warps 0-7 build one-hot rows (two sets of four, a TMEM quadrant each), 8-15
// are the epilogue, 16 loads LUT tiles, 17 issues MMAs, 18 loads codes (in bucket
// mode 16, 18, 20 and 21 gather LUT rows and 19 prepares items).
//   kOne: rows of a single 256-group batch, whose sums need no registers between
//     batches: fewer registers per epilogue warp, and four more warps.
//   kSmall: at most 64 queries. The MMAs take a third of the time then and the
//     hand-over of the stages bounds the kernel: 430 of 580 clocks per 256 bytes
//     of K are left with a quarter of the MMAs and no one-hot stores. So stages
//     hold 512 bytes of K, and the one-hot and LUT stages share one ring: one wait
//     and one commit instead of two. (Twice the producer warps instead: 1M x 1536,
//     16 queries 1625 -> 1792 us.)
// A stage holds 256 bytes of K otherwise: the issuing warp spends about 400 clocks
// per stage on its waits and commits whatever it holds, so it has to be worth more
// than that (8 MMAs are 768 clocks at N = 192).
enum Variant { kMulti, kOne, kSmall };
template <int V>
struct Config {
  static constexpr int kThreads = V == kOne ? 768 : 640;
  static constexpr int kRegsLaunch = V == kOne ? 80 : 96;
  static constexpr int kRegsProducer = 64, kRegsEpilogue = V == kOne ? 128 : 152;
  static constexpr int kRegsIssue = V == kOne ? 48 : 40;
  static_assert(256 * (kRegsProducer + kRegsEpilogue) + (kThreads - 512) * kRegsIssue <= kThreads * kRegsLaunch,
                "the register split must fit what the block is launched with");
  static constexpr int kGatherTeams = V == kOne ? 2 : 1;    // pairs of warps that gather LUT rows
  static constexpr int kCols = V == kSmall ? 64 : kMaxN;    // accumulator columns (queries)
  static constexpr int kStageBytes = V == kSmall ? 512 : 256;
  static constexpr int kTiles = kStageBytes / 128;          // LUT tiles of a stage
  static constexpr int kTileBytes = V == kSmall ? 32 * 128 : kTileB;
  static constexpr int kRingB = V == kSmall ? 3 : kStagesB; // kSmall: the one-hot ring as well
  static constexpr int kStageCols = kStageBytes / 4;        // TMEM columns of a stage's one-hot rows
};
// Byte groups of a stage. A byte group takes 32 bytes of K, or 16 with 3-bit
// codes (N8): their nibbles are below 8, so half of a one-hot row and of the LUT
// never meets a 1 and is left out (compact_luts_kernel).
template <bool N8, int V>
struct Groups {
  static constexpr int kBytes = N8 ? 16 : 32;
  static constexpr int kStage = Config<V>::kStageBytes / kBytes;
  static constexpr int kHalf = kStage / 2;        // a producer set's share
  static constexpr int kTile = 128 / kBytes;      // per LUT tile
  static constexpr int kPiece = 4 * kPieceCols / kBytes;
  static constexpr int kBatchStages = kFlushGroups / kStage;
  static constexpr int kChunkStages = kChunkGroups / kStage;
};

enum Mode { kSample, kTopK, kBucket };

// One item's queries and vectors (bucket mode: three items in flight).
constexpr int kParams = 3;
struct Params {
  float scale[kMaxN], init[kMaxN], thr[kMaxN], off[kMaxN];
  int q[kMaxN];
  uint32_t row[kMaxN + 32];  // byte offset of the query's LUT row (read in eights)
  int tiles, cols, size, vt0;
};

struct Shared {
  uint64_t full_b[kStagesB], empty_b[kStagesB];
  uint64_t full_a[kMaxStagesA], empty_a[kMaxStagesA];
  uint64_t full_c[kStagesC], empty_c[kStagesC];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t full_p[kParams], empty_p[kParams];
  uint64_t landed_b[kStagesB];
  uint32_t tmem;
  uint32_t pad[3];
  Params par[kParams];
  int cnt[kMaxN];
  // 32 queries' scores of an epilogue warp's 32 vectors.
  float stage[8][32][32];
};
constexpr size_t kSmemBytes = 1024 + static_cast<size_t>(kStagesB) * 2 * kTileB + kStagesC * kTileC + sizeof(Shared);

__device__ __forceinline__ uint32_t order_key(float s) {
  const uint32_t u = __float_as_uint(s);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_score(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Descending bitonic sort of 32 * E keys of a warp, entry lane * E + e.
template <int E>
__device__ __forceinline__ void warp_sort_keys(unsigned long long (&key)[E], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= E) {
        const int m = stride / E;
        const bool lower = (lane & m) == 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const unsigned long long o = __shfl_xor_sync(full_mask(), key[e], m);
          const bool desc = ((lane * E + e) & size) == 0;
          const bool take_max = lower == desc;
          key[e] = ((key[e] > o) == take_max) ? key[e] : o;
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if ((e & stride) == 0) {
            const bool desc = ((lane * E + e) & size) == 0;
            const unsigned long long x = key[e], y = key[e | stride];
            const bool keep = (x > y) == desc;
            key[e] = keep ? x : y;
            key[e | stride] = keep ? y : x;
          }
        }
      }
    }
  }
}

// Cuts a list of n (<= 32 * E) entries to its best min(k, n), best first, in
// place; returns the k-th key.
template <int E>
__device__ __noinline__ unsigned long long cut_list(unsigned long long* list, int n, int k, int lane) {
  unsigned long long key[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = lane * E + e;
    key[e] = i < n ? __ldcg(list + i) : 0ull;
  }
  warp_sort_keys<E>(key, lane);
  unsigned long long kth = 0ull;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = lane * E + e;
    if (i < k && i < n) list[i] = key[e];
    const unsigned long long c = __shfl_sync(full_mask(), key[e], (k - 1) / E);
    if ((k - 1) % E == e) kth = c;
  }
  return kth;
}

template <int CAP>
__device__ __forceinline__ unsigned long long cut_any(unsigned long long* list, int n, int k, int lane) {
  const int m = n > k ? n : k;
  if (m <= 128) return cut_list<4>(list, n, k, lane);
  if (CAP == 256 || m <= 256) return cut_list<8>(list, n, k, lane);
  return cut_list<16>(list, n, k, lane);
}

// The 8 one-hot bytes of a 3-bit code in bits 3..5 of x.
__device__ __forceinline__ void onehot8(uint32_t x, uint32_t* out) {
  uint64_t v;
  asm("shl.b64 %0, %1, %2;" : "=l"(v) : "l"(uint64_t{1}), "r"(x & 0x38u));
  out[0] = static_cast<uint32_t>(v);
  out[1] = static_cast<uint32_t>(v >> 32);
}
// The 16 one-hot bytes of the nibble in bits 3..6 of x, as two 64-bit shifts of a
// 1 by 8 * nibble and 8 * nibble - 64; a shift of 64 or more gives 0.
__device__ __forceinline__ void onehot16(uint32_t x, uint32_t* out) {
  uint64_t lo, hi;
  asm("shl.b64 %0, %1, %2;" : "=l"(lo) : "l"(uint64_t{1}), "r"(x & 0x78u));
  asm("shl.b64 %0, %1, %2;" : "=l"(hi) : "l"(uint64_t{1}), "r"((x & 0x78u) ^ 0x40u));
  out[0] = static_cast<uint32_t>(lo);
  out[1] = static_cast<uint32_t>(lo >> 32);
  out[2] = static_cast<uint32_t>(hi);
  out[3] = static_cast<uint32_t>(hi >> 32);
}

// One role's view of a work item.
struct Item {
  int tiles;    // 256-vector tiles
  int vt0, step;
  int cols;     // queries (a multiple of 32)
  int y;        // first LUT row (consecutive rows; not in bucket mode)
};

// kSample: write every score of the sampled tiles (thresholds come from them).
// kTopK: keep each query's top k of the item's range; CAP entries per list.
// kBucket: items are (bucket, up to 192 of its probing queries); the LUT rows are
// gathered by cp.async, and scores at or above the query's floor are appended to its region.
template <int MODE, int CAP, int V, bool N8>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Config<V>::kThreads, 1)
    onehot_scan_kernel(const __grid_constant__ CUtensorMap lut_map, const __grid_constant__ CUtensorMap code_map,
                       const __grid_constant__ OneHotArgs a) {
  constexpr bool SAMPLE = MODE == kSample, ONE = V == kOne;
  constexpr int kChunks = Config<V>::kCols / 2 / 32;  // of 32 queries per epilogue warp
  using G = Groups<N8, V>;
  constexpr int kStageGroupsTc = G::kStage, kHalfGroups = G::kHalf;
  constexpr int kBatchStages = G::kBatchStages, kChunkStages = G::kChunkStages;
  constexpr int kTiles = Config<V>::kTiles, kTileBytes = Config<V>::kTileBytes, kRingB = Config<V>::kRingB;
  constexpr int kStageColsA = Config<V>::kStageCols, kHalfColsA = kStageColsA / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // An offset, not integer arithmetic on the pointer: the compiler has to see that
  // everything below lies in shared memory.
  unsigned char* base = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* codes_smem = base + static_cast<size_t>(kStagesB) * 2 * kTileB;
  Shared& sh = *reinterpret_cast<Shared*>(codes_smem + kStagesC * kTileC);
  const uint32_t sB = tc::smem_u32(base), sC = tc::smem_u32(codes_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = tc::cta_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int n_stages = (a.nbg + kStageGroupsTc - 1) / kStageGroupsTc;
  const int n_batches = (a.nbg + kFlushGroups - 1) / kFlushGroups;
  const int items = MODE == kBucket ? static_cast<int>(*a.n_items) : a.q_tiles * a.n_ranges;
  // TMEM: two accumulators of acc_cols columns, then the one-hot stages.
  const uint32_t acc_cols = V == kSmall ? 64 : (MODE != kBucket && a.tile_queries <= 128 ? 128 : kMaxN);
  const int stages_a = V == kSmall ? kRingB : (acc_cols == 128 ? 4 : 2);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesB; ++s) {
      tc::mbar_init(tc::smem_u32(&sh.full_b[s]), MODE == kBucket ? 2 : 1);  // bucket mode: each CTA's relay
      tc::mbar_init(tc::smem_u32(&sh.landed_b[s]), 64);  // two gathering warps
      tc::mbar_init(tc::smem_u32(&sh.empty_b[s]), 1);
    }
    for (int s = 0; s < kMaxStagesA; ++s) {
      // eight producer warps of each CTA (and, sharing the ring, the LUT bytes)
      tc::mbar_init(tc::smem_u32(&sh.full_a[s]), V == kSmall ? 17 : 16);
      tc::mbar_init(tc::smem_u32(&sh.empty_a[s]), 1);
    }
    for (int s = 0; s < kStagesC; ++s) {
      tc::mbar_init(tc::smem_u32(&sh.full_c[s]), 1);
      tc::mbar_init(tc::smem_u32(&sh.empty_c[s]), 8);  // this CTA's producer warps
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(tc::smem_u32(&sh.acc_full[b]), 1);
      tc::mbar_init(tc::smem_u32(&sh.acc_empty[b]), 16);  // eight epilogue warps of each CTA
    }
    for (int b = 0; b < kParams; ++b) {
      tc::mbar_init(tc::smem_u32(&sh.full_p[b]), 1);
      // eight producer, eight epilogue and the gathering warps, and the issuing one
      tc::mbar_init(tc::smem_u32(&sh.empty_p[b]), 16 + 2 * Config<V>::kGatherTeams + (rank == 0 ? 1 : 0));
    }
    tc::mbar_init_fence();
    tc::prefetch_map(&lut_map);
    tc::prefetch_map(&code_map);
  }
  if (warp == 17) {
    tc::tmem_alloc2(tc::smem_u32(&sh.tmem), kTmemCols);
    tc::tmem_relinquish2();
    tc::fence_before();
  }
  __syncthreads();
  tc::cluster_sync();
  tc::fence_after();
  const uint32_t tmem = sh.tmem;
  bool alive = true;  // false: a wait gave up; this role stops
  uint64_t* const full_b = V == kSmall ? sh.full_a : sh.full_b;
  uint64_t* const empty_b = V == kSmall ? sh.empty_a : sh.empty_b;

  // Every role walks the same items: number pair, pair + pairs, ... In bucket mode
  // their parameters come through shared memory (warp 19 fills them in).
  int pb = 0;
  uint32_t pp = 0;
  auto open_item = [&](int it) -> Item {
    Item x{};
    if constexpr (MODE == kBucket) {
      if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.full_p[pb]), pp))) {
        alive = false;
        return x;
      }
      x.tiles = sh.par[pb].tiles;
      x.vt0 = sh.par[pb].vt0;
      x.step = 1;
      x.cols = sh.par[pb].cols;
    } else {
      const int qt = it / a.n_ranges, t0 = (it % a.n_ranges) * a.range_tiles;
      x.tiles = min(a.range_tiles, a.tiles - t0);
      x.step = a.tile_step > 0 ? a.tile_step : 1;
      x.vt0 = t0 * x.step;
      x.cols = a.tile_queries;
      x.y = qt * a.tile_queries;
    }
    return x;
  };
  auto close_item = [&]() {
    if constexpr (MODE == kBucket) {
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_u32(&sh.empty_p[pb]));
      if (++pb == kParams) {
        pb = 0;
        pp ^= 1u;
      }
    }
  };

  if (warp < 8) {
    // ---- one-hot rows: set `set` builds its half of every stage; TMEM lane
    // 32 quad + lane holds vector 4 lane + quad of this CTA's 128.
    tc::reg_dec<Config<V>::kRegsProducer>();
    const int quad = warp & 3, set = warp >> 2;
    const uint32_t dst0 = tmem + 2 * acc_cols + set * kHalfColsA + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t src0 = sC + set * kHalfGroups * 128 + lane * 4;
    const unsigned rot = (4 * quad + 29) & 31;  // brings the quad's nibbles to bits 3..6 and 19..22
    int slot = 0, sc = 0;
    uint32_t ph = 0, pc = 0;
    for (int it = pair; it < items && alive; it += pairs) {
      const Item x = open_item(it);
      for (int t = 0; t < x.tiles && alive; ++t) {
        for (int s0 = 0; s0 < n_stages && alive; s0 += kChunkStages) {
          if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.full_c[sc]), pc))) {
            alive = false;
            break;
          }
          const int s1 = min(kChunkStages, n_stages - s0);
          uint32_t src = src0 + sc * kTileC;
          for (int s = 0; s < s1; ++s, src += kStageGroupsTc * 128) {
            // The first look at the slot runs under the shifts, the first
            // half's columns are stored while the second half is built.
            const uint32_t bar = tc::smem_u32(&sh.empty_a[slot]);
            const bool ready = tc::mbar_test(bar, ph ^ 1u);
            uint32_t w[kHalfGroups];
#pragma unroll
            for (int g = 0; g < kHalfGroups; ++g) {
              asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[g]) : "r"(src + g * 128));
            }
            // The set's rows in pieces of 16 columns: high nibble (first half of
            // the LUT row), then the low one.
            auto build = [&](int piece, uint32_t (&out)[kPieceCols]) {
#pragma unroll
              for (int g = 0; g < G::kPiece; ++g) {
                const uint32_t word = w[piece * G::kPiece + g];
                const uint32_t v = __funnelshift_r(word, word, rot);
                if constexpr (N8) {
                  onehot8(v >> 16, out + 4 * g);
                  onehot8(v, out + 4 * g + 2);
                } else {
                  onehot16(v >> 16, out + 8 * g);
                  onehot16(v, out + 8 * g + 4);
                }
              }
            };
            uint32_t row[2][kPieceCols];
            build(0, row[0]);
            if (!__all_sync(full_mask(), ready || tc::mbar_wait(bar, ph ^ 1u))) {
              alive = false;
              break;
            }
            tc::fence_after();
#pragma unroll
            for (int piece = 0; piece < kHalfColsA / kPieceCols; ++piece) {
              if (piece > 0) build(piece, row[piece & 1]);
              tc::tmem_st16(dst0 + slot * kStageColsA + piece * kPieceCols, row[piece & 1]);
            }
            tc::tmem_wait_st();
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_cluster(tc::mapa(tc::smem_u32(&sh.full_a[slot]), 0));
            if (++slot == stages_a) {
              slot = 0;
              ph ^= 1u;
            }
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(tc::smem_u32(&sh.empty_c[sc]));
          if (++sc == kStagesC) {
            sc = 0;
            pc ^= 1u;
          }
        }
      }
      close_item();
    }
    __syncwarp();
  } else if (warp >= 16) {
    tc::reg_dec<Config<V>::kRegsIssue>();
    if (MODE == kBucket && (warp == 16 || warp == 18 || (ONE && (warp == 20 || warp == 21)))) {
      // ---- LUT rows of the item's queries: warp 16 copies the first 128 bytes
      // of K of every stage, warp 18 the second, 16 bytes a lane, eight lanes a
      // row, in the 128-byte swizzle (16-byte chunk c of row r at c ^ (r % 8)); the
      // copies arrive at landed_b themselves and warp 19 passes them on.
      // A one-row-box TMA gather (tile::gather4) took about 77 clocks per four
      // rows and bound the kernel (far scan of 10k queries x 464 probes of 1.2M x
      // 100: 8.8 ms, 4.9 ms with the copies). Warp 16 also loads the code chunks.
      // Two pairs of warps (ONE) take the stages in turn.
      const int which = warp == 18 || warp == 21;
      const int team = warp >= 20;
      const uint32_t rl = lane >> 3, cl = lane & 7;
      const uint32_t dst_even = rl * 128 + ((cl ^ rl) << 4), dst_odd = rl * 128 + ((cl ^ (rl + 4)) << 4);
      const uint32_t row_bytes = static_cast<uint32_t>(a.nbg) * Groups<N8, V>::kBytes;
      int st = 0, sc = 0;
      uint32_t ph = 0, pc = 0;
      for (int it = pair; it < items && alive; it += pairs) {
        const Item x = open_item(it);
        const int groups4 = x.cols / 8;  // four rows at a time
        const uint32_t* row = &sh.par[pb].row[rank * kHalfN + rl];
        for (int t = 0; t < x.tiles && alive; ++t) {
          for (int s = 0; s < n_stages && alive; ++s) {
            if (warp == 16 && s % kChunkStages == 0) {
              if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.empty_c[sc]), pc ^ 1u))) alive = false;
              if (alive && tc::elect_one()) {
                const uint32_t bar = tc::smem_u32(&sh.full_c[sc]);
                tc::mbar_arrive_expect_tx(bar, kTileC);
                tc::tma_load_2d(sC + sc * kTileC, &code_map, ((x.vt0 + t) & 1) * 64 + static_cast<int>(rank) * 32,
                                ((x.vt0 + t) >> 1) * a.nbg + s * kStageGroupsTc, bar);
              }
              __syncwarp();
              if (++sc == kStagesC) {
                sc = 0;
                pc ^= 1u;
              }
            }
            if (!alive) break;
            if (st % Config<V>::kGatherTeams == team) {
              if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.empty_b[st]), ph ^ 1u))) alive = false;
              if (!alive) break;
              const uint32_t at = static_cast<uint32_t>(s) * 256 + which * 128 + cl * 16;
              const uint32_t bytes = at < row_bytes ? 16u : 0u;  // zero past the row's end
              const uint8_t* src = a.luts + (bytes ? at : 0u);
              uint32_t dst = sB + (st * kTiles + which) * kTileBytes;
              // Eight rows' offsets first: read one by one between the copies, their
              // latency added up to 76 clocks a copy.
              for (int i = 0; i < groups4; i += 8, dst += 4096) {
                uint32_t off[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) off[u] = row[4 * (i + u)];
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                  if (i + u < groups4) {
                    tc::cp_async16_zfill(dst + u * 512 + dst_even, src + off[u], bytes);
                    tc::cp_async16_zfill(dst + u * 512 + 512 + dst_odd, src + off[u + 1], bytes);
                  }
                }
            }
              tc::cp_async_arrive(tc::smem_u32(&sh.landed_b[st]));
            }
            if (++st == kStagesB) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
        close_item();
      }
    } else if (warp == 16) {
      // ---- LUT tiles -------------------------------------------------------
      int st = 0;
      uint32_t ph = 0;
      for (int it = pair; it < items && alive; it += pairs) {
        const Item x = open_item(it);
        const int half_rows = x.cols / 2;
        for (int t = 0; t < x.tiles && alive; ++t) {
          for (int s = 0; s < n_stages; ++s) {
            if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&empty_b[st]), ph ^ 1u))) {
              alive = false;
              break;
            }
            const uint32_t bar = tc::smem_u32(&full_b[st]);
            const uint32_t dst = sB + st * kTiles * kTileBytes, cbar = tc::mapa(bar, 0);
            if (tc::elect_one()) {
              const int y = x.y + static_cast<int>(rank) * half_rows;
              if (rank == 0) tc::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(x.cols) * Config<V>::kStageBytes);
#pragma unroll
              for (int j = 0; j < kTiles; ++j) {  // tiles past the row are zero
                tc::tma_load_2d_pair(dst + j * kTileBytes, &lut_map, (s * kTiles + j) * 128, y, cbar);
              }
            }
            __syncwarp();
            if (++st == kRingB) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
        close_item();
      }
    } else if (warp == 18) {
      // ---- code chunks: 32 rows (byte groups) x 32 words of the scan layout.
      // Rows past the tile's last byte group meet zero LUT bytes.
      int sc = 0;
      uint32_t ph = 0;
      for (int it = pair; it < items && alive; it += pairs) {
        const Item x = open_item(it);
        for (int t = 0; t < x.tiles && alive; ++t) {
          const int vt = x.vt0 + t * x.step;
          for (int g0 = 0; g0 < a.nbg; g0 += kChunkGroups) {
            if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.empty_c[sc]), ph ^ 1u))) {
              alive = false;
              break;
            }
            const uint32_t bar = tc::smem_u32(&sh.full_c[sc]);
            if (tc::elect_one()) {
              tc::mbar_arrive_expect_tx(bar, kTileC);
              tc::tma_load_2d(sC + sc * kTileC, &code_map, (vt & 1) * 64 + static_cast<int>(rank) * 32,
                              (vt >> 1) * a.nbg + g0, bar);
            }
            __syncwarp();
            if (++sc == kStagesC) {
              sc = 0;
              ph ^= 1u;
            }
          }
        }
        close_item();
      }
    } else if (warp == 17 && rank == 0) {
      // ---- MMA ---------------------------------------------------------------
      int sa = 0, sb = 0;
      uint32_t pa = 0, pb = 0, batch = 0;
      bool seen = false;
      for (int it = pair; it < items && alive; it += pairs) {
        const Item x = open_item(it);
        const uint32_t idesc = (2u << 4) | (static_cast<uint32_t>(x.cols >> 3) << 17) | (16u << 24);
        for (int t = 0; t < x.tiles && alive; ++t) {
          for (int s0 = 0; s0 < n_stages && alive; s0 += kBatchStages, ++batch) {
            const uint32_t buf = batch & 1u;
            const uint32_t d = tmem + buf * acc_cols;
            if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.acc_empty[buf]), ((batch >> 1) & 1u) ^ 1u))) {
              alive = false;
              break;
            }
            const int s1 = min(s0 + kBatchStages, n_stages);
            for (int s = s0; s < s1; ++s) {
              // `seen`: the stage was found ready while the one before was issued.
              if (!seen && !__all_sync(full_mask(), (V == kSmall || tc::mbar_wait(tc::smem_u32(&full_b[sb]), pb)) &&
                                                        tc::mbar_wait(tc::smem_u32(&sh.full_a[sa]), pa))) {
                alive = false;
                break;
              }
              tc::fence_after();
              const uint32_t ta = tmem + 2 * acc_cols + sa * kStageColsA;
              const uint64_t db = tc::desc_k128(sB + sb * kTiles * kTileBytes);
              const int groups_left = a.nbg - s * kStageGroupsTc;  // tiles past the row are skipped
              const int na = sa + 1 == stages_a ? 0 : sa + 1, nb = sb + 1 == kRingB ? 0 : sb + 1;
              const uint32_t npa = pa ^ (na == 0 ? 1u : 0u), npb = pb ^ (nb == 0 ? 1u : 0u);
              // kSmall: look at the next stage while this one is issued (with longer
              // MMAs the look only costs: 1000 x 100k x 128 150 -> 160 us).
              const bool peek = V == kSmall && tc::mbar_test(tc::smem_u32(&sh.full_a[na]), npa);
              if (tc::elect_one()) {
#pragma unroll
                for (int i = 0; i < kTiles; ++i) {
                  if (i > 0 && groups_left <= i * G::kTile) break;
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    tc::mma_i8_pair_ta(d, ta + 32u * i + 8u * j, db + (kTileBytes >> 4) * i + 2u * j, idesc,
                                       (i > 0 || j > 0) ? 1u : (s > s0 ? 1u : 0u));
                  }
                }
                tc::commit2(tc::smem_u32(&sh.empty_a[sa]));
                if (V != kSmall) tc::commit2(tc::smem_u32(&sh.empty_b[sb]));
                if (s + 1 == s1) tc::commit2(tc::smem_u32(&sh.acc_full[buf]));
              }
              __syncwarp();
              if (V == kSmall) seen = __all_sync(full_mask(), peek);
              sa = na;
              sb = nb;
              pa = npa;
              pb = npb;
            }
          }
        }
        close_item();
      }
    } else if (MODE == kBucket && warp == 19) {
      // ---- bucket items: the queries' constants, up to three items ahead, and
      // the relay of landed LUT stages: fenced to the async proxy here (a fence in
      // the gathering warps waits for all their copies in flight), then passed to
      // the issuing CTA.
      int next = pair;  // the next item to prepare
      auto prepare_item = [&]() {
        Params& p = sh.par[pb];
        const uint4 e = a.items[next];  // bucket, first pair, pairs
        const int count = static_cast<int>(e.z), cols = (count + 31) / 32 * 32;
        for (int c = lane; c < cols; c += kWarp) {
          const int at = c < cols / 2 ? c : kHalfN + c - cols / 2;
          int q = 0;
          float scale = 0.f, init = 0.f, off = 0.f, thr = INFINITY;  // a column of no query
          if (c < count) {
            const uint32_t pr = a.pairs[e.y + c];
            q = static_cast<int>(pr / static_cast<uint32_t>(a.max_probe));
            scale = a.lut_scale[q];
            init = a.fa_init[q];
            off = a.offsets[pr];
            thr = fmaxf(-FLT_MAX, a.floor[q]);
          }
          p.q[at] = q;
          p.row[at] = static_cast<uint32_t>(q) * static_cast<uint32_t>(a.nbg * Groups<N8, V>::kBytes);
          p.scale[at] = scale;
          p.init[at] = init;
          p.off[at] = off;
          p.thr[at] = thr;
        }
        if (lane == 0) {
          p.size = static_cast<int>(a.bucket_size[e.x]);
          p.tiles = (p.size + kPairVectors - 1) / kPairVectors;
          p.vt0 = static_cast<int>(a.slot_start[e.x] / kPairVectors);
          p.cols = cols;
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(tc::smem_u32(&sh.full_p[pb]));
        next += pairs;
        if (++pb == kParams) {
          pb = 0;
          pp ^= 1u;
        }
      };
      int rb = 0, st = 0;  // the relayed item's parameters, the next stage
      uint32_t ph = 0;
      for (int it = pair; it < items && alive; it += pairs) {
        if (next == it) {
          if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.empty_p[pb]), pp ^ 1u))) {
            alive = false;
            break;
          }
          prepare_item();
        }
        const int stages = sh.par[rb].tiles * n_stages;
        for (int s = 0; s < stages; ++s) {
          if (next < items && next - it < kParams * pairs &&
              __all_sync(full_mask(), tc::mbar_test(tc::smem_u32(&sh.empty_p[pb]), pp ^ 1u))) {
            prepare_item();
          }
          if (!__all_sync(full_mask(), tc::mbar_wait(tc::smem_u32(&sh.landed_b[st]), ph))) {
            alive = false;
            break;
          }
          tc::fence_async_shared();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive_release(tc::mapa(tc::smem_u32(&sh.full_b[st]), 0));
          if (++st == kStagesB) {
            st = 0;
            ph ^= 1u;
          }
        }
        if (++rb == kParams) rb = 0;
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue: warp quadrant = 32 vectors, half = N / 2 queries ------------
    tc::reg_inc<Config<V>::kRegsEpilogue>();
    const int quad = warp & 3, half = (warp - 8) >> 2;
    const long long list0 = (static_cast<long long>(blockIdx.x) * a.tile_queries + half * (a.tile_queries / 2)) * CAP;
    unsigned long long* lists = MODE == kTopK ? a.lists + list0 : nullptr;
    int* s_cnt = sh.cnt + half * kHalfN;
    float* stage = &sh.stage[warp - 8][0][lane];
    const int ht = (warp & 3) * 32 + lane;  // thread of the half
    uint32_t batch = 0;
    // A warp whose wait gave up goes on through the barriers it shares.
    for (int it = pair; it < items && (alive || MODE != kBucket); it += pairs) {
      const Item x = open_item(it);
      const int cols = x.cols / 2;  // this half's queries, a multiple of 16
      const int c0 = half * cols;
      const uint32_t t_base = tmem + (static_cast<uint32_t>(quad * 32) << 16) + c0;
      const Params& par = sh.par[pb];
      const float* s_scale = par.scale + half * kHalfN;
      const float* s_init = par.init + half * kHalfN;
      float* s_thr = sh.par[pb].thr + half * kHalfN;
      const long long q0 = x.y + c0;
      if constexpr (MODE != kBucket) {
        tc::named_sync(1 + half, 128);
        if (ht < cols) {
          const bool ok = q0 + ht < a.nq;
          sh.par[0].scale[half * kHalfN + ht] = ok ? a.lut_scale[q0 + ht] : 0.f;
          sh.par[0].init[half * kHalfN + ht] = ok ? a.fa_init[q0 + ht] : 0.f;
          // -FLT_MAX admits every score above -inf; NaN never compares >=.
          float th = -FLT_MAX;
          if (!SAMPLE && ok && a.floor) th = fmaxf(th, a.floor[q0 + ht]);
          s_thr[ht] = ok ? th : INFINITY;
          s_cnt[ht] = 0;
        }
        tc::named_sync(1 + half, 128);
      }
      // A lane's vector of tile t: its alpha (NaN past the end: no score compares)
      // and id, loaded one tile ahead.
      auto slot_of = [&](int t) {
        return (static_cast<long long>(x.vt0) + t * x.step) * kPairVectors + rank * 128 + 4 * lane + quad;
      };
      auto load_vector = [&](int t, float* al, uint32_t* id) {
        const long long v = slot_of(t);
        *al = NAN;
        *id = static_cast<uint32_t>(v);
        if (t >= x.tiles) return;
        if constexpr (MODE == kBucket) {
          if (v - static_cast<long long>(x.vt0) * kPairVectors < par.size) {
            *al = __ldg(a.alpha + v);
            *id = __ldg(a.slot_ids + v);
          }
        } else {
          if (v < a.n) *al = __ldg(a.alpha + v);
        }
      };
      float al, al_next;
      uint32_t id, id_next;
      load_vector(0, &al_next, &id_next);
      for (int t = 0; t < x.tiles; ++t) {
        al = al_next;
        id = id_next;
        load_vector(t + 1, &al_next, &id_next);
        // fa of 32 queries (chunk c) -> scores: written out (sample), or one mask
        // bit per score at or above its threshold, by straight-line code. Only
        // when some lane has one do the scores go through shared memory
        // (registers cannot be indexed) to the lists. NaN never compares >=.
        auto take_scores = [&](int c, tc::F2 (&f)[16]) {
          const tc::F2 al2{al, al};
          if constexpr (SAMPLE) {
            const long long at =
                (static_cast<long long>(it % a.n_ranges) * a.range_tiles + t) * kPairVectors + rank * 128 + quad * 32 + lane;
            const bool valid = slot_of(t) < a.n;
            const int left = static_cast<int>(min(static_cast<long long>(cols), a.nq - q0)) - c * 32;
            float* out = a.dense + (q0 + c * 32) * a.dense_stride + at;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float v = (i & 1) ? f[i / 2].y : f[i / 2].x;
              if (i < left) *out = valid ? __fadd_rn(__fmul_rn(v, al), 0.f) : -INFINITY;
              out += a.dense_stride;
            }
          } else {
            unsigned part[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 th = *reinterpret_cast<const float4*>(s_thr + c * 32 + i);
              tc::F2 s0 = tc::mul2(f[i / 2], al2), s1 = tc::mul2(f[i / 2 + 1], al2);
              if constexpr (MODE == kBucket) {
                const float4 o = *reinterpret_cast<const float4*>(par.off + half * kHalfN + c * 32 + i);
                // One by one: ptxas 12.9 fused a packed add (.rn, -fmad=false) with the
                // packed multiply before it, which rounds once instead of twice.
                s0 = {__fadd_rn(s0.x, o.x), __fadd_rn(s0.y, o.y)};
                s1 = {__fadd_rn(s1.x, o.z), __fadd_rn(s1.y, o.w)};
              }
              if (s0.x >= th.x) part[0] |= 1u << i;
              if (s0.y >= th.y) part[1] |= 2u << i;
              if (s1.x >= th.z) part[2] |= 4u << i;
              if (s1.y >= th.w) part[3] |= 8u << i;
              f[i / 2] = s0;
              f[i / 2 + 1] = s1;
            }
            unsigned hits = part[0] | part[1] | part[2] | part[3];
            if (cols - c * 32 < 32) hits &= 0xffffu;  // the last 16 queries
            if (__any_sync(full_mask(), hits != 0u)) {
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                stage[2 * i * 32] = f[i].x;
                stage[(2 * i + 1) * 32] = f[i].y;
              }
              while (hits) {
                const int i = __ffs(hits) - 1;
                hits &= hits - 1;
                if constexpr (MODE == kBucket) {
                  // Past the region's end nothing is written; the count says so.
                  const int q = par.q[half * kHalfN + c * 32 + i];
                  const uint32_t pos = atomicAdd(a.append_count + q, 1u);
                  if (pos < a.region) {
                    const long long at = static_cast<long long>(q) * a.region + pos;
                    a.cand_score[at] = stage[i * 32];
                    a.cand_id[at] = id;
                  }
                } else {
                  const float score = __fadd_rn(stage[i * 32], 0.f);
                  const int pos = atomicAdd(&s_cnt[c * 32 + i], 1);
                  lists[static_cast<long long>(c * 32 + i) * CAP + pos] =
                      (static_cast<unsigned long long>(order_key(score)) << 32) | static_cast<uint32_t>(~id);
                }
              }
              __syncwarp();
            }
          }
        };
        // The batch sums are below 2^23: 2^23 + sum is exact in f32, and so is
        // taking the 2^23 off again.
        auto flush_sums = [&](int c, const uint32_t (&acc)[32], tc::F2 (&f)[16]) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 sc = *reinterpret_cast<const float4*>(s_scale + c * 32 + i);
            const tc::F2 big{-8388608.f, -8388608.f};
            const tc::F2 v0 = tc::add2({__uint_as_float(acc[i] | 0x4b000000u), __uint_as_float(acc[i + 1] | 0x4b000000u)}, big);
            const tc::F2 v1 =
                tc::add2({__uint_as_float(acc[i + 2] | 0x4b000000u), __uint_as_float(acc[i + 3] | 0x4b000000u)}, big);
            if constexpr (ONE) {  // the only batch: from the initial value
              const float4 in = *reinterpret_cast<const float4*>(s_init + c * 32 + i);
              f[i / 2] = tc::fma2({sc.x, sc.y}, v0, {in.x, in.y});
              f[i / 2 + 1] = tc::fma2({sc.z, sc.w}, v1, {in.z, in.w});
            } else {
              f[i / 2] = tc::fma2({sc.x, sc.y}, v0, f[i / 2]);
              f[i / 2 + 1] = tc::fma2({sc.z, sc.w}, v1, f[i / 2 + 1]);
            }
          }
        };
        auto load_init = [&](int c, tc::F2 (&f)[16]) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 v = *reinterpret_cast<const float4*>(s_init + c * 32 + i);
            f[i / 2] = {v.x, v.y};
            f[i / 2 + 1] = {v.z, v.w};
          }
        };
        auto wait_acc = [&]() {
          const uint32_t buf = batch & 1u;
          if (alive) alive = __all_sync(full_mask(), tc::mbar_wait_long(tc::smem_u32(&sh.acc_full[buf]), (batch >> 1) & 1u));
          tc::fence_after();
          return t_base + buf * acc_cols;
        };
        auto free_acc = [&]() {
          tc::fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive_cluster(tc::mapa(tc::smem_u32(&sh.acc_empty[batch & 1u]), 0));
          ++batch;
        };
        // TMEM columns past `cols` in a chunk belong to the other half or are unused.
        if constexpr (ONE) {
          // One batch: 32 queries at a time from sums to lists. (The next 32 sums
          // loaded meanwhile: 224 bytes of spills per thread and tile, slower.)
          const uint32_t acc_at = wait_acc();
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            if (c * 32 < cols) {
              uint32_t acc[32];
              tc::tmem_ld32(acc_at + c * 32, acc);
              tc::tmem_wait_ld32(acc);
              if (c + 1 == kChunks || (c + 1) * 32 >= cols) free_acc();
              tc::F2 f[16];
              flush_sums(c, acc, f);
              take_scores(c, f);
            }
          }
        } else {
          tc::F2 fa[kChunks][16];
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            if (c * 32 < cols) load_init(c, fa[c]);
          }
          for (int b = 0; b < n_batches; ++b) {
            const uint32_t acc_at = wait_acc();
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
              if (c * 32 < cols) {
                uint32_t acc[32];
                tc::tmem_ld32(acc_at + c * 32, acc);
                tc::tmem_wait_ld32(acc);
                flush_sums(c, acc, fa[c]);
              }
            }
            free_acc();
          }
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            if (c * 32 < cols) take_scores(c, fa[c]);
          }
        }
        {
          if constexpr (MODE == kTopK) {
          // A tile adds at most 128 entries per list: cut the lists that might
          // overflow on the next one to their top k and raise the threshold.
          tc::named_sync(1 + half, 128);
          const int mine = lane * 4 + quad;
          unsigned need = __ballot_sync(full_mask(), mine < cols && s_cnt[mine] > CAP - 128);
          while (need) {
            const int c = (__ffs(need) - 1) * 4 + quad;
            need &= need - 1;
            const int n = s_cnt[c];
            const unsigned long long kth = cut_any<CAP>(lists + static_cast<long long>(c) * CAP, n, a.k, lane);
            __syncwarp();
            if (lane == 0) {
              s_cnt[c] = min(n, a.k);
              if (n >= a.k) s_thr[c] = key_score(static_cast<uint32_t>(kth >> 32));
            }
          }
          tc::named_sync(1 + half, 128);
          }
        }
      }
      if (MODE == kTopK && alive) {
        const int r = it % a.n_ranges;
        // Publish: lists that fit go out as they are, longer ones cut to the top
        // k; four lists at a time, so that their loads overlap.
        constexpr int kAtOnce = 4;
        for (int base_c = quad; base_c < cols; base_c += 4 * kAtOnce) {
          int n[kAtOnce];
#pragma unroll
          for (int j = 0; j < kAtOnce; ++j) {
            const int c = base_c + 4 * j;
            n[j] = c < cols && q0 + c < a.nq ? s_cnt[c] : -1;
            if (n[j] > a.list_len) {
              cut_any<CAP>(lists + static_cast<long long>(c) * CAP, n[j], a.k, lane);
              __syncwarp();
              n[j] = a.k;
            }
          }
          for (int i = lane; i < a.list_len; i += kWarp) {
            unsigned long long key[kAtOnce];
#pragma unroll
            for (int j = 0; j < kAtOnce; ++j) {
              key[j] = i < n[j] ? __ldcg(lists + static_cast<long long>(base_c + 4 * j) * CAP + i) : 0ull;
            }
#pragma unroll
            for (int j = 0; j < kAtOnce; ++j) {
              if (n[j] >= 0) {
                const long long out = ((q0 + base_c + 4 * j) * (2LL * a.n_ranges) + 2 * r + rank) * a.list_len;
                a.cand_score[out + i] = i < n[j] ? key_score(static_cast<uint32_t>(key[j] >> 32)) : -INFINITY;
                a.cand_id[out + i] = ~static_cast<uint32_t>(key[j]);
              }
            }
          }
        }
      }
      close_item();
    }
  }
  if (!alive && a.status) {  // pinned host memory
    *static_cast<volatile unsigned*>(a.status) = 1u;
    __threadfence_system();
  }
  // A role that gave up waited about two seconds first, so no copy of this
  // CTA is still in flight here; otherwise every load was consumed.
  __syncwarp();
  __syncthreads();
  tc::cluster_sync();
  if (warp == 17) tc::tmem_dealloc2(tmem, kTmemCols);
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      p = nullptr;
    }
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

cudaError_t make_map(CUtensorMapDataType type, const void* p, uint64_t cols, uint64_t rows, uint64_t row_bytes,
                     uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swizzle, CUtensorMap* m) {
  EncodeTiled fn = encode_tiled();
  if (!fn) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {row_bytes};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t es[2] = {1, 1};
  const CUresult r = fn(m, type, 2, const_cast<void*>(p), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// LUT rows of 3-bit codes without the entries no code selects: 16 bytes a byte
// group, entries 0..7 of the high nibble, then of the low one.
__global__ void compact_luts_kernel(const uint2* __restrict__ luts, long long groups, uint4* __restrict__ out) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= groups) return;
  const uint2 hi = luts[4 * i], lo = luts[4 * i + 2];
  out[i] = make_uint4(hi.x, hi.y, lo.x, lo.y);
}

template <int MODE, int CAP, int V, bool N8>
cudaError_t launch_one(const OneHotArgs& a, int ctas, cudaStream_t stream) {
  auto kern = onehot_scan_kernel<MODE, CAP, V, N8>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemBytes));
  if (e != cudaSuccess) return e;
  CUtensorMap luts, codes;
  const uint64_t row_bytes = static_cast<uint64_t>(a.nbg) * Groups<N8, V>::kBytes;
  e = make_map(CU_TENSOR_MAP_DATA_TYPE_UINT8, a.luts, row_bytes, static_cast<uint64_t>(a.nq), row_bytes, 128,
               static_cast<uint32_t>(a.tile_queries / 2),
               CU_TENSOR_MAP_SWIZZLE_128B, &luts);
  if (e != cudaSuccess) return e;
  const uint64_t rows = static_cast<uint64_t>((a.n + kTileVectors - 1) / kTileVectors) * static_cast<uint64_t>(a.nbg);
  e = make_map(CU_TENSOR_MAP_DATA_TYPE_UINT32, a.codes, kTileWords, rows, kTileWords * 4, 32, kChunkGroups,
               CU_TENSOR_MAP_SWIZZLE_NONE, &codes);
  if (e != cudaSuccess) return e;
  kern<<<static_cast<unsigned>(ctas), Config<V>::kThreads, kSmemBytes, stream>>>(luts, codes, a);
  return cudaGetLastError();
}

template <int MODE, int CAP>
cudaError_t launch_t(const OneHotArgs& a, int ctas, cudaStream_t stream) {
  const bool one = a.nbg <= kFlushGroups;
  if constexpr (MODE == kBucket) {
    return one ? launch_one<MODE, CAP, kOne, false>(a, ctas, stream) : launch_one<MODE, CAP, kMulti, false>(a, ctas, stream);
  } else {
    if (a.tile_queries <= Config<kSmall>::kCols) {
      return a.compact ? launch_one<MODE, CAP, kSmall, true>(a, ctas, stream)
                       : launch_one<MODE, CAP, kSmall, false>(a, ctas, stream);
    }
    if (a.compact) {
      return one ? launch_one<MODE, CAP, kOne, true>(a, ctas, stream) : launch_one<MODE, CAP, kMulti, true>(a, ctas, stream);
    }
    return one ? launch_one<MODE, CAP, kOne, false>(a, ctas, stream) : launch_one<MODE, CAP, kMulti, false>(a, ctas, stream);
  }
}

// Ranges per query tile so that the items fill whole waves of CTA pairs: the
// fewest ranges within 1 % of the smallest longest-pair time, but at least a
// third of the pairs each (at most three query tiles' LUTs live in L2 at once).
int choose_ranges(long long q_tiles, long long tiles, int pairs) {
  const long long most = std::min<long long>(tiles, 2LL * pairs);
  auto cost = [&](long long r) {
    const long long per = (tiles + r - 1) / r;
    const long long rr = (tiles + per - 1) / per;
    return ((q_tiles * rr + pairs - 1) / pairs) * per;
  };
  long long best = cost(1);
  for (long long r = 2; r <= most; ++r) best = std::min(best, cost(r));
  const long long from = std::min<long long>(most, (pairs + 2) / 3);
  for (long long r = from; r <= most; ++r) {
    if (cost(r) * 100 <= best * 101) return static_cast<int>(r);
  }
  for (long long r = 1; r <= most; ++r) {
    if (cost(r) * 100 <= best * 101) return static_cast<int>(r);
  }
  return 1;
}

// Whether a batch is faster here than on the lookup scan. Times in us beyond what
// both spend (launches, query preparation, merge), fitted to searches of 8k to 2M
// vectors of 128 to 1536 dimensions:
//   * here, up to 64 queries: 25 for the sample, and 0.43 per 256-vector tile and
//     16 byte groups (0.56 per 32 groups of 3-bit codes) on each CTA pair;
//   * lookups, k <= 32, from three queries on: four queries a CTA over 2048-vector
//     blocks, 0.31 per byte group (3-bit 0.17) and 14 per wave of two CTAs per SM,
//     0.21 (0.11) per group while every CTA has an SM to itself. One and two
//     queries stream the codes at HBM speed and stay there;
//   * lookups, k > 32: lists in shared memory and a longer merge; slower from three
//     queries on nearly everywhere (20k x 128 3-bit, 24 queries of k = 256 82 / 139 us
//     is the worst of the others), for one or two by a fit of its own to 616 searches of
//     8k to 3M vectors, k 33 to 256, that picks the faster side or one at most 10 %
//     slower in all but 33 of them (a third slower at worst).
// Measured (lookup / here): 1M x 1536 4-bit 8 queries 937 / 1155, 12 queries
// 1272 / 1155, 16 queries 1721 / 1155; 100k x 128 4-bit 24 queries 69 / 74, 32
// queries 94 / 74; 2M x 768 3-bit 8 queries 647 / 774, 12 queries 826 / 774;
// 20k x 768 4-bit 4 queries 125 / 85; one query of k = 100 over 1M x 1536 551 / 1137,
// of k = 33 over 3M x 384 398 / 896, two of k = 48 over 8,192 x 128 58 / 39.
bool onehot_pays(long long n, long long nq, int nbg, int bits, int k, int sms) {
  const long long pairs = sms / 2, tiles = (n + kPairVectors - 1) / kPairVectors;
  const double blocks = static_cast<double>((n + kScanBlockVectors - 1) / kScanBlockVectors);
  if (nq > Config<kSmall>::kCols) {
    if (k > 32) return true;
    // Whole searches, fitted to 4,536 of them (66 to 600 queries, k 1 to 32, 8k to 100k
    // vectors of 8 to 768 dims): the side it picks is 0.4 % above the faster one on
    // average, more than 10 % in 68. Small indexes are launches on both sides, and the
    // lookups' grow with k: lookups / here, 128 queries over 8,192 x 64 3-bit, k = 1
    // 31.3 / 45.6 us, k = 5 34.4 / 47.3; 66 over 16,384 x 64 3-bit, k = 3 33.4 / 46.8.
    const long long q_tiles = (nq + kMaxN - 1) / kMaxN;
    const double share = static_cast<double>(((nq + q_tiles - 1) / q_tiles + 31) / 32 * 32) / kMaxN;
    const double waves = std::max(0.0, static_cast<double>((nq + 3) / 4) * blocks / (2.0 * sms) - 0.5);
    const double stages = static_cast<double>((nbg + (bits == 3 ? 15 : 7)) / (bits == 3 ? 16 : 8));
    const double lookups = 22.6 + nbg * (bits == 3 ? 0.128 : 0.226) +
                           waves * (nbg * (bits == 3 ? 0.151 : 0.259) + 10.2 + 1.6 * k) + 1.9 * k + 0.106 * blocks;
    const double here = 36.7 + (bits == 3 ? 4.1 : 0.0) +
                        static_cast<double>((q_tiles * tiles + pairs - 1) / pairs) * share * (0.374 * stages + 3.14) +
                        0.085 * k + 0.019 * static_cast<double>(nq) + 0.72 * stages;
    return lookups > here;
  }
  const double stages = static_cast<double>((nbg + (bits == 3 ? 31 : 15)) / (bits == 3 ? 32 : 16));
  const double scan = static_cast<double>((tiles + pairs - 1) / pairs) * stages * (bits == 3 ? 0.56 : 0.43);
  const double here = 25.0 + scan;
  if (nq <= 2) {
    if (k <= 32) return false;
    const double q = static_cast<double>(nq), nd = static_cast<double>(n);
    return 10.0 + 18.0 * q + nd * nbg / 3.1e6 + 0.03 * nbg * q + blocks * (0.0015 * k * (1.0 + q) + 0.057 * q) + 0.1 * k >
           28.0 + scan + 0.19 * k + 0.04 * nbg + 44e-6 * nd;
  }
  if (k > 32) return true;
  const double ctas = static_cast<double>((nq + 3) / 4) * blocks;
  double lookups = nbg * (bits == 3 ? 0.11 : 0.21);
  if (ctas > sms) lookups = std::max(lookups, ctas / (2.0 * sms) * (nbg * (bits == 3 ? 0.17 : 0.31) + 14.0));
  return lookups > here;
}

}  // namespace

bool plan_onehot(long long n, long long nq, int nbg, int bits, int k, int sms, OneHotPlan* plan) {
  if (n < kOneHotMinVectors || n > 0x7fffffffLL || nq < 1 || k < 1 || k > kMaxK || sms < 2) return false;
  if (!onehot_pays(n, nq, nbg, bits, k, sms)) return false;
  const long long q_tiles = (nq + kMaxN - 1) / kMaxN;
  const long long per = (nq + q_tiles - 1) / q_tiles;
  plan->tile_queries = static_cast<int>((per + 31) / 32 * 32);
  plan->q_tiles = static_cast<int>((nq + plan->tile_queries - 1) / plan->tile_queries);
  plan->tiles = static_cast<int>((n + kPairVectors - 1) / kPairVectors);
  const int pairs = sms / 2;
  int r = choose_ranges(plan->q_tiles, plan->tiles, pairs);
  plan->range_tiles = (plan->tiles + r - 1) / r;
  plan->n_ranges = (plan->tiles + plan->range_tiles - 1) / plan->range_tiles;
  const long long items = static_cast<long long>(plan->q_tiles) * plan->n_ranges;
  plan->ctas = static_cast<int>(2 * std::min<long long>(pairs, items));
  plan->cap = k <= 64 ? 256 : 512;
  // Thresholds: the k-th best of a sample of whole tiles spread over the index.
  // About n k / sample scores per query then pass them and cost the epilogue
  // some hundred clocks each per warp, which rows of few stages (768 clocks of
  // MMA each) do not hide: at least 8192 k / stages vectors, 1/64 of the index,
  // at most 1/16 of it, 32768 vectors and 128 MiB of scores, at least 1024 vectors
  // (128 MiB at kOneHotMaxPass queries). (1000 queries x
  // 100k x 128, k = 10: scan + sample + selection 261 + 23 + 13 us with 1536
  // vectors, 188 + 35 + 25 us with the rule's 6144.)
  const int stage = bits == 3 ? Groups<true, kOne>::kStage : Groups<false, kOne>::kStage;
  const long long n_stages = (nbg + stage - 1) / stage;
  plan->compact = bits == 3;
  long long sample = std::max<long long>(n / 64, 8192LL * k / n_stages);
  sample = std::min<long long>({sample, n / 16, 32768, (128LL << 20) / 4 / nq});
  sample = std::max<long long>(sample, 1024);
  plan->sample_tiles = static_cast<int>(std::min<long long>(plan->tiles, sample / kPairVectors));
  plan->sample_step = plan->tiles / plan->sample_tiles;
  // Published lists: room for what usually passes, so that few need a cut.
  const long long expect = n * k / (static_cast<long long>(plan->sample_tiles) * kPairVectors * 2 * plan->n_ranges);
  plan->list_len = k + (2 * expect <= k ? 0 : 16);
  return true;
}

long long onehot_pass(const OneHotPlan& p, long long nq) {
  const long long per_query = 2LL * p.n_ranges * p.list_len * 8;
  const long long fit = static_cast<long long>(kOneHotListBytes) / per_query / kMaxN * kMaxN;
  return std::min<long long>({nq, kOneHotMaxPass, std::max<long long>(fit, kMaxN)});
}

OneHotScratch onehot_scratch(const OneHotPlan& p, long long nq, int nbg) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  const size_t m = static_cast<size_t>(nq);
  const size_t running = static_cast<size_t>(p.ctas) * p.tile_queries * p.cap * 8;
  const size_t sample = m * p.sample_tiles * kPairVectors * 4;
  const size_t lists = up(m * 2 * p.n_ranges * p.list_len * 4);
  OneHotScratch s;
  s.cand_score = up(std::max(running, sample));
  s.cand_id = s.cand_score + lists;
  s.compact = s.cand_id + lists;
  s.floor = s.compact + (p.compact ? up(m * nbg * 16) : 0);
  s.bytes = s.floor + m * 4;
  return s;
}

cudaError_t launch_compact_luts(const uint8_t* luts, long long nq, int nbg, uint8_t* out, cudaStream_t stream) {
  const long long groups = nq * nbg;
  compact_luts_kernel<<<static_cast<unsigned>((groups + 255) / 256), 256, 0, stream>>>(
      reinterpret_cast<const uint2*>(luts), groups, reinterpret_cast<uint4*>(out));
  return cudaGetLastError();
}

cudaError_t launch_onehot_sample(const OneHotArgs& in, const OneHotPlan& p, int sms, cudaStream_t stream) {
  OneHotArgs a = in;
  a.compact = p.compact;
  a.tile_queries = p.tile_queries;
  a.q_tiles = p.q_tiles;
  a.tiles = p.sample_tiles;
  a.tile_step = p.sample_step;
  a.dense_stride = static_cast<long long>(p.sample_tiles) * kPairVectors;
  const int r = choose_ranges(p.q_tiles, p.sample_tiles, sms / 2);
  a.range_tiles = (a.tiles + r - 1) / r;
  a.n_ranges = (a.tiles + a.range_tiles - 1) / a.range_tiles;
  const long long items = static_cast<long long>(a.q_tiles) * a.n_ranges;
  return launch_t<kSample, 256>(a, static_cast<int>(2 * std::min<long long>(sms / 2, items)), stream);
}

cudaError_t launch_onehot_scan(const OneHotArgs& in, const OneHotPlan& p, cudaStream_t stream) {
  OneHotArgs a = in;
  a.compact = p.compact;
  a.tile_queries = p.tile_queries;
  a.q_tiles = p.q_tiles;
  a.tiles = p.tiles;
  a.tile_step = 0;
  a.range_tiles = p.range_tiles;
  a.n_ranges = p.n_ranges;
  a.list_len = p.list_len;
  return p.cap == 256 ? launch_t<kTopK, 256>(a, p.ctas, stream) : launch_t<kTopK, 512>(a, p.ctas, stream);
}

cudaError_t launch_onehot_buckets(const BucketScanArgs& b, long long nq, long long n_slots, int sms, unsigned* status,
                                  cudaStream_t stream) {
  if (!b.append_count || !b.floor || b.n_items == nullptr || !onehot_buckets_fit(nq, n_slots, b.nbg)) {
    return cudaErrorInvalidValue;
  }
  OneHotArgs a{};
  a.codes = b.codes;
  a.alpha = b.alpha;
  a.luts = b.luts;
  a.lut_scale = b.lut_scale;
  a.fa_init = b.fa_init;
  a.n = n_slots;
  a.nbg = b.nbg;
  a.nq = nq;
  a.k = b.k;
  a.cand_score = b.cand_score;
  a.cand_id = b.cand_id;
  a.floor = b.floor;
  a.status = status;
  a.tile_queries = kMaxN;
  a.items = b.items;
  a.n_items = b.n_items;
  a.pairs = b.pairs;
  a.offsets = b.offsets;
  a.slot_ids = b.slot_ids;
  a.slot_start = b.slot_start;
  a.bucket_size = b.bucket_size;
  a.append_count = b.append_count;
  a.region = static_cast<uint32_t>(b.region);
  a.max_probe = b.max_probe;
  return launch_t<kBucket, 256>(a, sms / 2 * 2, stream);
}

}  // namespace vcb
