// KV-cache decode attention: one new query token per sequence against that sequence's cache.
//
// The reference runs this as 61 tiny launches per layer (per-head M=1 cuBLAS products, 256-byte
// device-to-device appends, one softmax; src/model.cpp:745-790). Here it is ONE kernel per layer
// call, for any number of concurrent sequences. It is bound by HBM where the caches are large and by
// latency where they are not:
//   * a producer thread per CTA streams the cache rows of a (sequence, head) through a ring of 16 KB
//     stages (8 KB of K, 8 KB of V) with bulk copies; four consumer warps read them from shared
//     memory 512 contiguous bytes at a time. What is in flight does not depend on how the arithmetic
//     is getting on: with loads and arithmetic taking turns in the same warps the kernel reached
//     4.75 TB/s on 64 sequences x 12 heads of up to 1024 rows and 4.26 on 4 x 24 of up to 8000 at head
//     size 128, now 5.56-5.7 and 4.85-5.2 (6.8 on 128 x 24 x 128; the lengths are drawn);
//   * q.k partial sums are reduced over a row's D*sizeof(T)/16 lanes with warp shuffles; each lane
//     keeps an online-softmax state (max, sum, D/lanes accumulators) for the rows it has seen. The
//     row groups of a tile are handled without branches so that their latencies overlap: a CTA's
//     rate is the length of that chain (branching on each row: 12-24 % slower);
//   * many (sequence, head) pairs: persistent CTAs, the longest sequences first, items handed out by
//     a counter, the next item's rows already on their way while one is merged. Few pairs: the CTAs
//     of a cluster share one, or the same head of a long and a short sequence, and merge through distributed
//     shared memory. Neither needs records in
//     global memory, and a pair's merge costs no trip through L2 (8 sequences x 8 heads of up to 400
//     rows, early start: 6.9 us a layer with records and tickets, 3.9 now);
//   * the append is fused: the warp that owns row `len` takes k_new/v_new from the token's vectors,
//     uses them, and stores them into the cache;
//   * every CTA draws a ticket once it has copied the lengths; the holder of the last one stores
//     length + 1, while the rows are still streaming. Counters are returned to zero by their last
//     user, also where a bounded wait ran out, so a workspace zeroed once stays usable forever;
//   * launched with programmatic stream serialization: the next decode call's CTAs set themselves up
//     (and, where the caller allows it, fill their rings) while this grid drains.
#include <cfloat>
#include <climits>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace {

constexpr int kDecodeWarps = 4;                         // consumer warps
constexpr int kDecodeThreads = (kDecodeWarps + 1) * 32;  // and one producer warp
constexpr int kTileBytes = 8192;                        // K (and V) bytes of one ring stage
// Ring stages, and CTAs an SM holds with that many: calls of few CTAs get the deeper rings.
constexpr int kFewStages = 4, kFewPerSm = 3;
constexpr int kManyStages = 3, kManyPerSm = 4;
constexpr int kMaxStages = 4;
constexpr int kItemRing = 2;        // items a CTA's producer may be ahead
constexpr unsigned kTicketGroups = 32;  // first-level counters of the "all lengths read" tickets
constexpr int kMaxRanked = 256;     // sequences whose lengths a CTA copies and can rank
constexpr int kMaxCluster = 8;      // CTAs that share a head of one sequence or two (portable cluster size)
constexpr int kMaxPaired = 64;      // sequences of a call up to which clusters share two
constexpr long long kBytesPerRank = 65536;    // and the K + V bytes that are worth one of them

// A 16-byte piece of a row as float pairs, and the softmax's exponential. Scores are kept in units
// that exp_of() takes: natural units and expf for fp32 caches, log2 units and ex2 for bf16 ones
// (whose 2^-9 rounding of the inputs is far above the difference).
template <typename T>
struct Elem;
template <>
struct Elem<float> {
  static constexpr int kPerLane = 4;
  static constexpr float kUnit = 1.0f;
  __device__ static void unpack(float2 (&f)[2], const uint4& raw) {
    f[0] = make_float2(__uint_as_float(raw.x), __uint_as_float(raw.y));
    f[1] = make_float2(__uint_as_float(raw.z), __uint_as_float(raw.w));
  }
  __device__ static float exp_of(float x) { return expf(x); }
  __device__ static float from_float(float x) { return x; }
};
template <>
struct Elem<__nv_bfloat16> {
  static constexpr int kPerLane = 8;
  static constexpr float kUnit = 1.4426950408889634f;
  __device__ static void unpack(float2 (&f)[4], const uint4& raw) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
  }
  __device__ static float exp_of(float x) { return ptx::ex2(x); }
  __device__ static __nv_bfloat16 from_float(float x) { return __float2bfloat16_rn(x); }
};

// Workspace: B*H words, of which the first is the item counter, then the 1 + kTicketGroups counters
// of the "all lengths read" tickets (uint32, all zero between calls), padded to 256 bytes. No more is
// used. The sizes that callers are asked for, and the shapes that the allocation-free entry point
// refuses, are part of the interface and count room for the records of a split-K merge, too, which an
// earlier kernel kept in global memory.
inline size_t record_bytes(int B, int H, int D, int max_len) {
  constexpr long long kTargetCtas = 592, kMinRows = 256;
  const long long pairs = static_cast<long long>(B) * H;
  const long long want = std::max(1LL, (kTargetCtas + pairs - 1) / pairs);
  const long long rows = (std::max((max_len + want - 1) / want, kMinRows) + 127) / 128 * 128;
  const long long splits = (max_len + rows - 1) / rows;
  if (splits == 1) return 0;
  return static_cast<size_t>(pairs) * splits * (D + 2) * sizeof(float);
}
inline size_t ticket_bytes(int B, int H) {
  return (sizeof(uint32_t) * (static_cast<size_t>(B) * H + 1 + kTicketGroups) + 255) / 256 * 256;
}
inline size_t workspace_bytes(int B, int H, int D, int max_len) {
  return ticket_bytes(B, H) + (record_bytes(B, H, D, max_len) + 255) / 256 * 256;
}

// ---- the kernel --------------------------------------------------------------------------------
// How a call's (sequence, head) pairs are dealt out. Each way is an instance of its own: in one kernel that branched on
// it, every one carried the others' registers and branches (bf16, us a layer, one kernel -> instances: 64 sequences x 12
// heads x 64 17.4 -> 17.2, all of 512 rows 18.4 -> 17.7, 1 x 24 heads x 128 of 7900 rows 21.2 -> 20.5, 2 x 12 19.2 -> 18.0).
enum class Deal { kPersistent, kCluster, kPairCluster };
// kPersistent: persistent CTAs take whole (sequence, head) items, the items of longer sequences first
// (`reorder`): CTA c item c, then whatever a global counter hands out. The producer is already loading
// the next item's rows while the consumers finish the current one.
// kCluster: the `ranks` CTAs of a thread-block cluster share the rows of one item and merge
// through distributed shared memory: no records in global memory, no tickets, no second kernel.
// kPairCluster: a cluster shares the same head of two sequences, the longest of the call with the shortest and so on,
// and each gets of its CTAs what its length, read here, asks for. With a cluster for each, the longest ones' read alone at
// the end (bf16, 24 heads x 128, us a layer, before -> now: rows 1000 / 3000 / 5000 / 7000 38.6 -> 35.5, 7900 and three
// of 1000 40.1 -> 29.0, 4 x 4000 35.5 -> 35.2, 7000 / 3000 / 5000 37.7 -> 36.8; 16 x 12 heads, up to 1900 rows 22.7 ->
// 21.2). Parts that ran on from one sequence into the other, all exactly even, were slower: 38.2, 28.8, 38.0 and 23.5.
// A sequence's sums, and with them the last bits of its result, are divided by its partner's length then; in every deal they
// go by the number of (sequence, head) pairs.
template <typename T, int D>
struct DecodeTile {
  static constexpr int kRowBytes = D * static_cast<int>(sizeof(T));
  static constexpr int kRows = kTileBytes / kRowBytes;   // cache rows of one ring stage
  static_assert(kRows >= 1 && kTileBytes % kRowBytes == 0, "a tile is a whole number of rows");
};

struct DecodeShared {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t item_ready[kItemRing], item_free[kItemRing];
  int item[kItemRing];                   // items claimed for this CTA
  int abort_flag;
  float m[kDecodeWarps], l[kDecodeWarps];
  float acc[kDecodeWarps][128];          // [warp][d]
  __align__(16) int lens[kMaxRanked];    // the sequence lengths (calls of up to kMaxRanked sequences)
  int2 member[2];                        // kPairCluster: (sequence or -1, length)
  union {
    struct {
      int place[kMaxRanked];             // reorder: rank of each sequence
      int order[kMaxRanked];             // reorder: sequence of each rank
    };
    float record[kMaxCluster][130];      // clusters: every CTA's partial result, in the CTA that merges it
  };
};

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   ptx::smem_u32(smem_dst)),
               "l"(src), "r"(bytes), "r"(ptx::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// stores to the same shared-memory variable of another CTA of the cluster
__device__ __forceinline__ uint32_t cluster_address(const void* own, int cta) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(ptx::smem_u32(own)), "r"(cta));
  return a;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void consumers_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kDecodeWarps * 32) : "memory");
}
// The same, and whether any consumer thread brought a true one.
__device__ __forceinline__ bool consumers_any(bool mine) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, 2, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"(static_cast<uint32_t>(mine)), "n"(kDecodeWarps * 32)
      : "memory");
  return any != 0;
}

template <typename T, int D, Deal DEAL>
__global__ void __launch_bounds__(kDecodeThreads, kManyPerSm)
decode_kernel(T* __restrict__ out, unsigned* __restrict__ item_counter, unsigned* __restrict__ seq_tickets, const T* __restrict__ q,
              const T* __restrict__ k_new, const T* __restrict__ v_new, T* __restrict__ k_cache,
              T* __restrict__ v_cache, int32_t* __restrict__ lengths, int fixed_len, int B, int H, int max_len,
              int cluster_ctas, int stages, int reorder, int early, float scale, int* __restrict__ status) {
  using namespace ptx;
  using Tile = DecodeTile<T, D>;
  constexpr bool kPersistent = DEAL == Deal::kPersistent, kPairs = DEAL == Deal::kPairCluster;
  const int ranks = kPersistent ? 1 : cluster_ctas;
  constexpr int EPL = Elem<T>::kPerLane;  // elements per lane (16 bytes)
  constexpr int LPK = D / EPL;            // lanes per cache row
  constexpr int KPI = 32 / LPK;           // cache rows per warp instruction
  constexpr int kGroups = Tile::kRows / (kDecodeWarps * KPI);   // row groups of a tile per warp
  static_assert(LPK >= 1 && LPK <= 32 && (LPK & (LPK - 1)) == 0, "row must split over a warp");
  static_assert(kGroups * kDecodeWarps * KPI == Tile::kRows && D <= kDecodeWarps * 32, "tile split");

  extern __shared__ __align__(128) uint8_t smem[];
  DecodeShared& sh = *reinterpret_cast<DecodeShared*>(smem + stages * 2 * kTileBytes);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0);
  const int lane = threadIdx.x % 32;
  const int rank = static_cast<int>(blockIdx.x) % ranks;

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], kDecodeWarps);
    }
    for (int i = 0; i < kItemRing; ++i) {
      mbar_init(&sh.item_ready[i], 1);
      mbar_init(&sh.item_free[i], kDecodeWarps);
    }
    sh.abort_flag = 0;
    fence_mbar_init();
  }
  // Everything this grid reads may have been written by the grid before it — unless the caller
  // has promised (dadattn_set_decode_early_start) that the grid before it does not write this
  // call's caches, lengths and workspace: then the lengths are read, and the ring is filled with
  // the first cache rows, while that grid drains, and only the token vectors wait for it.
  // Dependents are released behind that wait in either case: of several early calls in a row each
  // overlaps the one ahead of it and no other, so that a cache written two calls ago may be read.
  if (!early) {
    pdl_wait();
    pdl_launch_dependents();
  }

  // Up to kMaxRanked lengths are copied to shared memory first; nobody reads the caller's array
  // after that, so it can be advanced as soon as every CTA has its copy.
  const bool snapshot = B <= kMaxRanked;
  if (snapshot)
    for (int i = threadIdx.x; i < kMaxRanked; i += kDecodeThreads) {
      sh.lens[i] = i < B ? (lengths ? lengths[i] : fixed_len) : INT_MIN;
      if (kPersistent && reorder) sh.place[i] = 0;
    }
  if (kPairs && threadIdx.x < 2) sh.member[threadIdx.x] = make_int2(-1, -1);
  __syncthreads();
  if (kPersistent && reorder) {
    // rank(s) = number of sequences that come before s (longer, or as long with a smaller index);
    // with the count padded to a power of two n_pad (32..256; padding is INT_MIN and comes last),
    // 128 threads share out the n_pad^2 comparisons.
    const int t = threadIdx.x;
    if (t < 128) {
      const int lg = 32 - __clz(B - 1);   // n_pad = 1 << lg, 5 <= lg <= 8
      const int n_pad = 1 << lg;
      const int groups = lg < 7 ? 128 >> lg : 1;
      const int per = n_pad / groups, g = (t >> lg) & (groups - 1);
      for (int si = t & (n_pad - 1); si < n_pad; si += 128) {
        const int mine = sh.lens[si];
        int count = 0;
#pragma unroll 4
        for (int j = g * per; j < (g + 1) * per; j += 4) {
          const int4 o = *reinterpret_cast<const int4*>(sh.lens + j);   // broadcast reads
          count += static_cast<int>(o.x > mine) | (static_cast<int>(o.x == mine) & static_cast<int>(j + 0 < si));
          count += static_cast<int>(o.y > mine) | (static_cast<int>(o.y == mine) & static_cast<int>(j + 1 < si));
          count += static_cast<int>(o.z > mine) | (static_cast<int>(o.z == mine) & static_cast<int>(j + 2 < si));
          count += static_cast<int>(o.w > mine) | (static_cast<int>(o.w == mine) & static_cast<int>(j + 3 < si));
        }
        if (count) atomicAdd(&sh.place[si], count);
      }
    }
    __syncthreads();
    for (int i = t; i < B; i += kDecodeThreads) sh.order[sh.place[i]] = i;
    __syncthreads();
  }

  // Item e of the call. A sequence whose length is outside [0, max_len) is skipped (rows = 0) and
  // reported.
  struct Item {
    int b, h, len, row0, row1;
  };
  const int n_items = B * H, n_lanes = static_cast<int>(gridDim.x);   // kPersistent: items taken up by CTAs at the start
  auto rows_of = [&](int len) { return len >= 0 && len < max_len ? len + 1 : 0; };
  int merges = -1;            // which sequence of its cluster a CTA merges, if any, and which CTAs have parts of it
  int part0 = 0, part1 = ranks;
  bool second = false;        // whether the CTA's own part is of its cluster's second sequence
  // CTA `part` of the `parts` that share sequence b's head h
  auto share_of = [&](int b, int h, int len, int part, int parts) -> Item {
    const int rows = rows_of(len), share = (static_cast<unsigned>(rows) + parts - 1) / static_cast<unsigned>(max(parts, 1)), row0 = min(part * share, rows);
    return Item{b, h, len, row0, min(row0 + share, rows)};
  };
  auto item = [&](int e) -> Item {
    const int p = e / H, b = kPersistent && reorder ? sh.order[p] : p;
    return share_of(b, e - p * H, snapshot ? sh.lens[b] : lengths[b], rank, ranks);
  };
  Item first;
  if (!kPairs) {
    first = item(static_cast<int>(blockIdx.x) / ranks);
    if (rank == 0) merges = 0;
  } else {
    // Cluster c takes head c % H of the c / H-th longest and c / H-th shortest sequence (one, in the middle of an odd
    // number). Its CTAs are divided so that the largest part is as small as it can be.
    const int e = static_cast<int>(blockIdx.x) / ranks, g = e / H, t = threadIdx.x;
    if (t < B) {
      const int mine = sh.lens[t];
      int place = 0;
#pragma unroll 4
      for (int j = 0; j < B; ++j)
        place += static_cast<int>(sh.lens[j] > mine) | (static_cast<int>(sh.lens[j] == mine) & static_cast<int>(j < t));
      if (place == g) sh.member[0] = make_int2(t, mine);
      else if (place == B - 1 - g) sh.member[1] = make_int2(t, mine);
    }
    __syncthreads();
    const int2 a = sh.member[0], b = sh.member[1];
    const int rows_a = rows_of(a.y), rows_b = b.x < 0 ? 0 : rows_of(b.y);
    int cut = rows_b == 0 ? ranks : 0;   // CTAs for the first
    if (rows_a > 0 && rows_b > 0) {
      // the whole number below or above what is in proportion, whichever has the smaller largest part
      const float fa = static_cast<float>(rows_a), fb = static_cast<float>(rows_b);
      const int below = min(max(static_cast<int>(__fdividef(fa * ranks, fa + fb)), 1), ranks - 1);
      const int above = min(below + 1, ranks - 1);
      cut = fa * (ranks - above) <= fb * below ? below : above;
    }
    second = rank >= cut;
    first = second ? share_of(b.x, e - g * H, b.y, rank - cut, ranks - cut) : share_of(a.x, e - g * H, a.y, rank, cut);
    if (rank < 2 && (rank == 0 ? a.x : b.x) >= 0) merges = rank;
    part0 = rank == 0 ? 0 : cut;
    part1 = rank == 0 ? cut : ranks;
  }
  // "this CTA has started and looked its item up" (record shares memory with the ranking): waited
  // for before the first remote store
  if (!kPersistent) cluster_arrive();

  // Every CTA of the call draws a ticket once it has read the lengths; whoever holds the last one
  // knows that nobody will read them again and advances them. Two levels keep the atomics off one
  // address: the CTAs are dealt into kTicketGroups groups; the last of each group draws from a
  // second counter, and the last of those advances.
  const unsigned group = blockIdx.x % kTicketGroups;
  auto draw_ticket = [&]() { return atomicAdd(&seq_tickets[1 + group], 1u); };
  auto is_last = [&](unsigned ticket) -> bool {
    const unsigned all_ctas = gridDim.x;
    if (ticket != (all_ctas - group + kTicketGroups - 1) / kTicketGroups - 1) return false;
    seq_tickets[1 + group] = 0;   // ready for the next call
    const unsigned groups = all_ctas < kTicketGroups ? all_ctas : kTicketGroups;
    if (atomicAdd(&seq_tickets[0], 1u) != groups - 1) return false;
    seq_tickets[0] = 0;
    return true;
  };

  volatile int* abort_flag = &sh.abort_flag;
  if (warp == kDecodeWarps) {
    // ------------------------------ producer ------------------------------
    if (elect_one()) {
      // The ticket is drawn now and looked at once the ring is full: its round trip and the advance
      // of the lengths stay off the path to the kernel's end.
      bool ticket_due = lengths != nullptr && snapshot;
      const unsigned ticket = ticket_due ? draw_ticket() : 0;
      auto settle_ticket = [&]() {
        if (ticket_due && is_last(ticket)) {
          if (early) pdl_wait();   // the kernel ahead may still read the lengths
          for (int j = 0; j < B; ++j) {
            const int len = sh.lens[j];
            if (len >= 0 && len < max_len) lengths[j] = len + 1;   // a full or invalid sequence is left alone
          }
        }
        ticket_due = false;
      };
      // One claim per item beyond the CTAs' first ones and one per CTA that finds nothing left: n_items
      // in all, of which the last returns the counter to zero.
      auto claim = [&]() -> int {
        if (!kPersistent || n_lanes >= n_items) return n_items;
        const unsigned c = atomicAdd(item_counter, 1u);
        if (c == static_cast<unsigned>(n_items - 1)) *item_counter = 0;
        return min(static_cast<int>(c) + n_lanes, n_items);
      };
      int st = 0, lap = 0;
      int next = 0;   // the last claim
      Item s = first;
      bool ok = true;
      for (int n = 0; ok; ++n) {
        const size_t base = (static_cast<size_t>(s.b) * H + s.h) * max_len * D;
        const int end = min(s.row1, s.len);   // the row being appended comes from k_new / v_new
        for (int r = s.row0; r < end; r += Tile::kRows) {
          if (lap == 1 && st == 0) settle_ticket();
          if (lap > 0 && !(ok = mbar_wait(&sh.empty[st], (lap - 1) & 1, abort_flag))) break;
          const uint32_t bytes = static_cast<uint32_t>(min(Tile::kRows, end - r)) * Tile::kRowBytes;
          mbar_arrive_expect_tx(&sh.full[st], 2 * bytes);
          bulk_load(smem + st * 2 * kTileBytes, k_cache + base + static_cast<size_t>(r) * D, bytes, &sh.full[st]);
          bulk_load(smem + (st * 2 + 1) * kTileBytes, v_cache + base + static_cast<size_t>(r) * D, bytes, &sh.full[st]);
          if (++st == stages) st = 0, ++lap;
        }
        // The item after this one is claimed only when this one's last rows are on their way: what is
        // in the ring covers the counter's round trip, and a CTA with a long item takes no second one
        // that an idle CTA could have had (64 sequences x 12 heads: 210 us, 240 when claimed an item ahead).
        if (ok) next = claim();
        const int slot = n % kItemRing;
        ok = ok && (n < kItemRing || mbar_wait(&sh.item_free[slot], (n / kItemRing - 1) & 1, abort_flag));
        if (!ok) break;
        *reinterpret_cast<volatile int*>(&sh.item[slot]) = next;
        mbar_arrive(&sh.item_ready[slot]);
        if (next >= n_items) break;
        s = item(next);
      }
      // After a wait that ran out the claims are made all the same: the workspace stays usable.
      while (next < n_items) next = claim();
      settle_ticket();
      settle_ring(sh.full, stages, lap * stages + st);
    }
  } else {
    // ------------------------------ consumers ------------------------------
    if (early) {
      pdl_wait();
      pdl_launch_dependents();
    }
    const int slot = lane / LPK, part = lane % LPK;
    const float scale_unit = scale * Elem<T>::kUnit;
    int st = 0;
    uint32_t phase = 0;
    bool ok = true;
    Item s = first, nxt = first;
    bool have = true;
    // token vectors of an item: fetched an item ahead (k_new / v_new by the warp that appends)
    uint4 q_raw = make_uint4(0, 0, 0, 0), kn_raw = q_raw, vn_raw = q_raw;
    auto fetch_token = [&](const Item& t) {
      const size_t off = (static_cast<size_t>(t.b) * H + t.h) * D + part * EPL;
      q_raw = *reinterpret_cast<const uint4*>(q + off);
      if (warp == 0 && slot == 0) {
        kn_raw = *reinterpret_cast<const uint4*>(k_new + off);
        vn_raw = *reinterpret_cast<const uint4*>(v_new + off);
      }
    };
    fetch_token(s);
    for (int n = 0; have; ++n, s = nxt) {
      const size_t bh = static_cast<size_t>(s.b) * H + s.h;
      float m = -FLT_MAX, l = 0.f;
      float2 acc[EPL / 2], qf[EPL / 2];
      Elem<T>::unpack(qf, q_raw);
#pragma unroll
      for (int e = 0; e < EPL / 2; ++e) acc[e] = make_float2(0.f, 0.f);

      // NR row groups' worth of K / V registers into the lane's online-softmax state. No branches:
      // the groups' chains (shuffles, exponentials, sums) have to overlap, a CTA's rate is their
      // latency. Rows that do not count (`valid`, read only when !ALL) come in as zeros.
      auto absorb = [&](const uint4* kr, const uint4* vr, const bool* valid, auto count, auto all) {
        constexpr int NR = decltype(count)::value;
        constexpr bool ALL = decltype(all)::value;
        float sc[NR], p[NR];
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          float2 kf[EPL / 2];
          Elem<T>::unpack(kf, kr[u]);
          float2 dot = fmul2(qf[0], kf[0]);
#pragma unroll
          for (int e = 1; e < EPL / 2; ++e) dot = ffma2(qf[e], kf[e], dot);
          sc[u] = dot.x + dot.y;
        }
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < NR; ++u) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
        float m_new = m;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          sc[u] = ALL || valid[u] ? sc[u] * scale_unit : -FLT_MAX;
          m_new = fmaxf(m_new, sc[u]);
        }
        // (while m_new is still -FLT_MAX the state is all zeros: corr = 1 leaves it so)
        const float corr = Elem<T>::exp_of(m - m_new);
        float sum = 0.f;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          p[u] = Elem<T>::exp_of(sc[u] - m_new);
          if (!ALL && !valid[u]) p[u] = 0.f;
          sum += p[u];
        }
        l = fmaf(l, corr, sum);
#pragma unroll
        for (int e = 0; e < EPL / 2; ++e) acc[e] = fmul2(acc[e], make_float2(corr, corr));
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          float2 vf[EPL / 2];
          Elem<T>::unpack(vf, vr[u]);
#pragma unroll
          for (int e = 0; e < EPL / 2; ++e) acc[e] = ffma2(make_float2(p[u], p[u]), vf[e], acc[e]);
        }
        m = m_new;
      };

      // the token being appended: its vectors are used and stored by the CTA whose share ends there
      if (warp == 0 && s.row0 < s.row1 && s.row1 == s.len + 1) {
        const bool mine = slot == 0;
        if (mine) {
          const size_t at = (bh * max_len + s.len) * D + part * EPL;
          *reinterpret_cast<uint4*>(k_cache + at) = kn_raw;
          *reinterpret_cast<uint4*>(v_cache + at) = vn_raw;
        }
        absorb(&kn_raw, &vn_raw, &mine, std::integral_constant<int, 1>{}, std::false_type{});
      }
      const int end = min(s.row1, s.len);
      for (int r = s.row0; r < end; r += Tile::kRows) {
        if (!ok || !(ok = mbar_wait(&sh.full[st], phase, abort_flag))) break;
        const uint4* kt = reinterpret_cast<const uint4*>(smem + st * 2 * kTileBytes) + warp * kGroups * 32 + lane;
        const uint4* vt = kt + kTileBytes / 16;
        uint4 kr[kGroups], vr[kGroups];
#pragma unroll
        for (int u = 0; u < kGroups; ++u) kr[u] = kt[u * 32];
#pragma unroll
        for (int u = 0; u < kGroups; ++u) vr[u] = vt[u * 32];
        if (r + Tile::kRows <= end) {
          absorb(kr, vr, nullptr, std::integral_constant<int, kGroups>{}, std::true_type{});
        } else {   // an item's last tile: what lies beyond the rows loaded is left over from earlier tiles
          bool valid[kGroups];
#pragma unroll
          for (int u = 0; u < kGroups; ++u) {
            valid[u] = r + (warp * kGroups + u) * KPI + slot < end;
            if (!valid[u]) kr[u] = vr[u] = make_uint4(0, 0, 0, 0);
          }
          absorb(kr, vr, valid, std::integral_constant<int, kGroups>{}, std::false_type{});
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[st]);
        if (++st == stages) st = 0, phase ^= 1;
      }

      // the next item; its token vectors arrive while this one is merged
      have = false;
      if (kPersistent) {
        const int slot_i = n % kItemRing;
        if (ok && (ok = mbar_wait(&sh.item_ready[slot_i], (n / kItemRing) & 1, abort_flag))) {
          const int e = *reinterpret_cast<volatile int*>(&sh.item[slot_i]);
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.item_free[slot_i]);
          if ((have = e < n_items)) {
            nxt = item(e);
            fetch_token(nxt);
          }
        }
      }

      // Merge the KPI row slots of the warp (lanes with equal `part`), then the warps.
#pragma unroll
      for (int o = LPK; o < 32; o <<= 1) {
        const float m_o = __shfl_xor_sync(0xffffffffu, m, o);
        const float l_o = __shfl_xor_sync(0xffffffffu, l, o);
        const float m_new = fmaxf(m, m_o);
        const float ca = m > -FLT_MAX ? Elem<T>::exp_of(m - m_new) : 0.f;
        const float cb = m_o > -FLT_MAX ? Elem<T>::exp_of(m_o - m_new) : 0.f;
        l = l * ca + l_o * cb;
#pragma unroll
        for (int e = 0; e < EPL / 2; ++e) {
          acc[e].x = acc[e].x * ca + __shfl_xor_sync(0xffffffffu, acc[e].x, o) * cb;
          acc[e].y = acc[e].y * ca + __shfl_xor_sync(0xffffffffu, acc[e].y, o) * cb;
        }
        m = m_new;
      }
      if (slot == 0) {
#pragma unroll
        for (int e = 0; e < EPL / 2; ++e) {
          sh.acc[warp][part * EPL + 2 * e] = acc[e].x;
          sh.acc[warp][part * EPL + 2 * e + 1] = acc[e].y;
        }
        if (part == 0) {
          sh.m[warp] = m;
          sh.l[warp] = l;
        }
      }
      consumers_sync();
      const int d = threadIdx.x;
      if (d < D) {
        float mm = -FLT_MAX;
#pragma unroll
        for (int w = 0; w < kDecodeWarps; ++w) mm = fmaxf(mm, sh.m[w]);
        float ll = 0.f, aa = 0.f;
#pragma unroll
        for (int w = 0; w < kDecodeWarps; ++w) {
          const float c = sh.m[w] > -FLT_MAX ? Elem<T>::exp_of(sh.m[w] - mm) : 0.f;
          ll += sh.l[w] * c;
          aa += sh.acc[w][d] * c;
        }
        if (kPersistent) {
          if (s.row1 > 0) out[bh * D + d] = Elem<T>::from_float(aa / ll);
        } else {
          // hand the share to the CTA that merges it, which is known to run once the cluster's first barrier is through
          cluster_wait();
          const uint32_t rec = cluster_address(&sh.record[rank][0], second ? 1 : 0);
          st_cluster(rec + d * 4, aa);
          if (d == 0) {
            st_cluster(rec + D * 4, mm);
            st_cluster(rec + D * 4 + 4, ll);
          }
        }
      }
      if (kPersistent) {
        if (s.row1 == 0 && s.h == 0 && threadIdx.x == 0) atomicExch(status, DADATTN_E_ARG);
        // sh.acc / sh.m are read: the next item may write them. The warps go on together or not at all: one whose
        // wait ran out would be missing at the named barriers of the next item.
        if (consumers_any(!ok)) have = false;
      }
    }
  }

  if (!kPersistent) {
    // Threads without a share to hand over join the first barrier here; after the second the shares are merged.
    const int d = threadIdx.x;
    if (d >= D) cluster_wait();
    cluster_arrive();
    cluster_wait();
    if (merges >= 0) {
      const int b = kPairs ? sh.member[merges].x : first.b, len = kPairs ? sh.member[merges].y : first.len;
      if (len >= 0 && len < max_len) {
        if (d < D) {
          float mm = -FLT_MAX;
          for (int j = part0; j < part1; ++j) mm = fmaxf(mm, sh.record[j][D]);
          float ll = 0.f, aa = 0.f;
          for (int j = part0; j < part1; ++j) {
            const float c = Elem<T>::exp_of(sh.record[j][D] - mm);   // a share without rows has m = -FLT_MAX: 0
            ll += sh.record[j][D + 1] * c;
            aa += sh.record[j][d] * c;
          }
          out[(static_cast<size_t>(b) * H + first.h) * D + d] = Elem<T>::from_float(aa / ll);
        }
      } else if (first.h == 0 && d == 0) {
        atomicExch(status, DADATTN_E_ARG);
      }
    }
  }

  if (lengths != nullptr && !snapshot) {   // the lengths were read all along: tickets only now
    __shared__ int sh_advance;
    __syncthreads();
    if (threadIdx.x == 0) sh_advance = is_last(draw_ticket());
    __syncthreads();
    if (sh_advance)
      for (int i = threadIdx.x; i < B; i += kDecodeThreads) {
        const int len = lengths[i];
        if (len >= 0 && len < max_len) lengths[i] = len + 1;
      }
  }
  if (threadIdx.x == 0 && sh.abort_flag) report_timeout(status, sh.abort_flag);
}

constexpr size_t decode_smem(int stages) { return static_cast<size_t>(stages) * 2 * kTileBytes + sizeof(DecodeShared); }
static_assert((decode_smem(kFewStages) + 1024) * kFewPerSm <= 228 * 1024 && kFewStages <= kMaxStages &&
              (decode_smem(kManyStages) + 1024) * kManyPerSm <= 228 * 1024 && kManyStages <= kMaxStages,
              "shared memory of an SM exceeded");

template <typename T, int DH>
int launch_decode(T* out, const T* q, const T* k_new, const T* v_new, T* k_cache, T* v_cache, int32_t* lengths,
                  int fixed_len, int B, int H, int max_len, float scale, unsigned* tickets, int* status, int early,
                  cudaStream_t st) {
  // the workspace's tickets: one per (sequence, head), the first of which counts the items; then those
  // of the lengths
  unsigned* item_counter = tickets;
  unsigned* seq_tickets = tickets ? tickets + static_cast<size_t>(B) * H : nullptr;
  int dev = 0, sms = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  DAD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const long long pairs = static_cast<long long>(B) * H;
  // CTAs per (sequence, head): as many as the longest sequence there can be has 64 KB of K and V
  // for, while all of the call's CTAs still fit on the GPU at once. Beyond that, waiting clusters
  // cost more than the finer cut gives (4 sequences x 24 heads of up to 8000 rows: 131 us with 4 CTAs
  // each, 145 with 8). us a call in a CUDA graph, 12 heads x 64, by KB of K and V per CTA:
  //                                  32      64     128     256
  //   fp32, 150 rows               3.54    3.88    4.01    4.01
  //   fp32, 300 rows               4.10    4.31    4.95    6.10
  //   fp32, 700 rows               4.78    4.78    5.55    7.08
  //   bf16, 700 rows               4.69    4.91    5.97    6.95
  //   bf16, 4 x 50-200 rows        4.53    4.27    4.27    4.23
  //   bf16, 10 x 80-800 rows       8.19    8.36    8.36    8.71
  // (fp32, 16 heads x 16, 400 rows: 4.22, 3.80 from 64 on.)
  const long long bytes = static_cast<long long>(lengths ? max_len : fixed_len + 1) * 2 * DH * sizeof(T);
  const int resident = kManyPerSm * sms;
  int ranks = 1;
  while (ranks < kMaxCluster && ranks * kBytesPerRank < bytes && pairs * ranks * 2 <= resident) ranks *= 2;
  // Two or four CTAs for each: a cluster of four or eight for two sequences, where the lengths are on the device. It is
  // for lengths that differ; equal ones are 0-7 % slower with it. Not where clusters are the last to fit: they wait for
  // each other, and the next call's have no room to set themselves up in. Clusters of eight take up to 84 % of the GPU's
  // places for CTAs, of four up to 92 %. Nor beyond kMaxPaired sequences, all of whose lengths every CTA ranks. us a call
  // in a CUDA graph, bf16, head size 128, a cluster for each / for two, by the longest of evenly spread lengths and (")
  // of one long sequence, the others an eighth of it:
  //   clusters of eight         1000           2000           6000           2000 "         6000 "
  //   4 x 20 heads, 320 CTAs                   12.8 / 12.2    27.2 / 25.1    12.4 / 10.5    26.9 / 20.7
  //   4 x 31, 496            11.9 / 11.9       15.9 / 16.3    36.2 / 34.6    16.1 / 13.2    36.8 / 26.7
  //   8 x 16, 512            11.4 / 12.4       16.5 / 16.7    37.8 / 36.5    13.8 / 12.1    32.4 / 25.1
  //   4 x 33, 528            11.2 / 12.6       16.1 / 18.4    35.2 / 37.8    16.4 / 13.7    37.6 / 27.6
  //   of four: 8 x 34, 544   18.2 / 17.4       28.5 / 27.3    68.4 / 65.8    26.3 / 21.4    66.5 / 52.6
  //   4 x 70, 560            16.2 / 18.1       27.8 / 30.1    74.4 / 76.8    28.1 / 22.6    71.0 / 55.1
  //   64 x 4, 512            18.0 / 18.6       28.1 / 27.1    69.2 / 65.6    20.6 / 17.5    50.7 / 40.3
  //   96 x 2, 384            14.6 / 15.4       128 x 2, 512   17.1 / 19.0    96 x 1, clusters of eight  9.3 / 10.9
  Deal deal = ranks > 1 ? Deal::kCluster : Deal::kPersistent;
  // (without a workspace there is no counter to deal items from: one CTA each)
  long long grid = ranks > 1 || !item_counter ? pairs * ranks : min(pairs, static_cast<long long>(resident));
  const long long paired = static_cast<long long>((B + 1) / 2) * H * ranks * 2;
  if (lengths && ranks > 1 && ranks < kMaxCluster && B >= 2 && B <= kMaxPaired &&
      paired * 100 <= resident * (ranks * 2 == kMaxCluster ? 84LL : 92LL))
    deal = Deal::kPairCluster, ranks *= 2, grid = paired;
  // The deeper ring for clusters of eight as long as some more would fit (48 do on 148 SMs; 4, 8 or 2 sequences, spread
  // up to 2000 rows, deeper / not: 320 CTAs 12.2 / 12.4, 368 13.4 / 13.9, 384 13.9 / 14.0 and, one long, 9.8 / 9.3, 400
  // 18.0 / 14.1).
  const long long few = deal == Deal::kPairCluster && ranks == kMaxCluster ? sms * 5LL / 2 : kFewPerSm * sms;
  const int stages = grid <= few ? kFewStages : kManyStages;
  // Longest first pays once a CTA takes more than one item; the in-kernel ranking handles 32..256 sequences.
  const int reorder = B >= 32 && B <= kMaxRanked && pairs > grid;
  auto kern = deal == Deal::kPersistent ? decode_kernel<T, DH, Deal::kPersistent>
              : deal == Deal::kCluster ? decode_kernel<T, DH, Deal::kCluster> : decode_kernel<T, DH, Deal::kPairCluster>;
  // (a cheap host call, 0.06 us)
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(decode_smem(kMaxStages))));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(kDecodeThreads);
  cfg.dynamicSmemBytes = decode_smem(stages);
  cfg.stream = st;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim = {static_cast<unsigned>(ranks), 1, 1};
  cfg.attrs = attrs;
  cfg.numAttrs = ranks > 1 ? 2 : 1;
  DAD_CUDA(cudaLaunchKernelEx(&cfg, kern, out, item_counter, seq_tickets, q, k_new, v_new, k_cache, v_cache, lengths, fixed_len, B,
                              H, max_len, ranks, stages, reorder, early, scale, status));
  return DADATTN_OK;
}

int launch_decode_bf16(uint16_t* out, const uint16_t* q, const uint16_t* k_new, const uint16_t* v_new,
                       uint16_t* k_cache, uint16_t* v_cache, int32_t* lengths, int B, int H, int D, int max_len,
                       float scale, unsigned* tickets, int* status, int early, cudaStream_t st) {
  using BF = __nv_bfloat16;
  auto* launch = D == 64 ? launch_decode<BF, 64> : launch_decode<BF, 128>;
  return launch(reinterpret_cast<BF*>(out), reinterpret_cast<const BF*>(q), reinterpret_cast<const BF*>(k_new),
                reinterpret_cast<const BF*>(v_new), reinterpret_cast<BF*>(k_cache), reinterpret_cast<BF*>(v_cache),
                lengths, 0, B, H, max_len, scale, tickets, status, early, st);
}

int launch_decode_f32(float* out, const float* q, const float* k_new, const float* v_new, float* k_cache,
                      float* v_cache, int32_t* lengths, int fixed_len, int B, int H, int D, int max_len, float scale,
                      unsigned* tickets, int* status, cudaStream_t st) {
  auto* launch = D == 16 ? launch_decode<float, 16> : D == 32 ? launch_decode<float, 32>
                 : D == 64 ? launch_decode<float, 64> : launch_decode<float, 128>;
  return launch(out, q, k_new, v_new, k_cache, v_cache, lengths, fixed_len, B, H, max_len, scale,
                tickets, status, 0, st);
}

// Rows 0..n-1 of sequence b's cache from the K / V heads a prefill leaves behind: k_heads,
// v_heads [H, n, D] fp32 (the reference's q_heads / k_heads / v_heads layout for batch 1,
// src/model.cpp:385-387) -> k_cache, v_cache [B, H, max_len, D] in T; sets lengths[b] = n. One
// launch for both tensors; the reference does two cudaMemcpy2D per layer (src/model.cpp:835-843).
template <typename T>
__global__ void kv_cache_fill_kernel(T* __restrict__ k_cache, T* __restrict__ v_cache,
                                     int32_t* __restrict__ lengths, const float* __restrict__ k_heads,
                                     const float* __restrict__ v_heads, int b, int H, int n, int max_len,
                                     int D) {
  const int64_t per = static_cast<int64_t>(H) * n * D / 4;   // float4 groups per tensor
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t == 0 && lengths) lengths[b] = n;
  if (t >= 2 * per) return;
  const bool is_v = t >= per;
  const int64_t i = (is_v ? t - per : t) * 4;         // element index in [H, n, D]
  const int64_t h = i / (static_cast<int64_t>(n) * D), rem = i - h * n * D;
  const float4 x = *reinterpret_cast<const float4*>((is_v ? v_heads : k_heads) + i);
  T* dst = (is_v ? v_cache : k_cache) + ((static_cast<int64_t>(b) * H + h) * max_len) * D + rem;
  dst[0] = Elem<T>::from_float(x.x);
  dst[1] = Elem<T>::from_float(x.y);
  dst[2] = Elem<T>::from_float(x.z);
  dst[3] = Elem<T>::from_float(x.w);
}

int check_decode_bf16(const void* out, const void* q, const void* k_new, const void* v_new,
                      const void* k_cache, const void* v_cache, const void* lengths, int B, int H,
                      int D, int max_len) {
  if (!out || !q || !k_new || !v_new || !k_cache || !v_cache || !lengths)
    return fail(DADATTN_E_ARG, "decode: null pointer");
  if (B <= 0 || H <= 0 || max_len <= 0 || H > 65535 ||
      static_cast<long long>(B) * H > 0x7fffffffLL)
    return fail(DADATTN_E_ARG, "decode: bad sizes B=%d H=%d max_len=%d", B, H, max_len);
  if (D != 64 && D != 128) return fail(DADATTN_E_UNSUPPORTED, "decode bf16: unsupported D %d", D);
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k_new, 16) || !aligned(v_new, 16) ||
      !aligned(k_cache, 16) || !aligned(v_cache, 16))
    return fail(DADATTN_E_ARG, "decode: pointers must be 16-byte aligned");
  return DADATTN_OK;
}

thread_local int g_decode_early = 0;

}  // namespace
}  // namespace dadattn

using namespace dadattn;

extern "C" size_t dadattn_decode_workspace_bytes(int B, int H, int D, int max_len) {
  if (B <= 0 || H <= 0 || D <= 0 || max_len <= 0) return 0;
  return workspace_bytes(B, H, D, max_len);
}

extern "C" int dadattn_decode_bf16(uint16_t* out, const uint16_t* q, const uint16_t* k_new,
                                   const uint16_t* v_new, uint16_t* k_cache, uint16_t* v_cache,
                                   int32_t* lengths, int B, int H, int D, int max_len,
                                   float scale, void* workspace, size_t workspace_bytes_given,
                                   dadattn_stream_t stream) {
  if (int rc = check_decode_bf16(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, D, max_len))
    return rc;
  if (!workspace || !aligned(workspace, 16))
    return fail(DADATTN_E_ARG, "decode: workspace must be a 16-byte aligned device pointer");
  if (workspace_bytes_given < workspace_bytes(B, H, D, max_len))
    return fail(DADATTN_E_WORKSPACE, "decode: workspace %zu < %zu bytes", workspace_bytes_given,
                workspace_bytes(B, H, D, max_len));
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned* tickets = static_cast<unsigned*>(workspace);
  return launch_decode_bf16(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, D, max_len, scale, tickets, status,
                            g_decode_early, st);
}

extern "C" int dadattn_set_decode_early_start(int on) {
  g_decode_early = on ? 1 : 0;
  return DADATTN_OK;
}

extern "C" int dadattn_decode_f32(float* out, const float* q, const float* k_new,
                                  const float* v_new, float* k_cache, float* v_cache, int H,
                                  int max_len, int D, int pos, float scale,
                                  dadattn_stream_t stream) {
  if (!out || !q || !k_new || !v_new || !k_cache || !v_cache)
    return fail(DADATTN_E_ARG, "decode: null pointer");
  if (H <= 0 || max_len <= 0 || H > 65535) return fail(DADATTN_E_ARG, "decode: bad sizes");
  if (pos < 0 || pos >= max_len)
    return fail(DADATTN_E_ARG, "decode: pos %d outside context length %d", pos, max_len);
  if (D != 16 && D != 32 && D != 64 && D != 128)
    return fail(DADATTN_E_UNSUPPORTED, "decode f32: unsupported D %d", D);
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k_new, 16) || !aligned(v_new, 16) ||
      !aligned(k_cache, 16) || !aligned(v_cache, 16))
    return fail(DADATTN_E_ARG, "decode: pointers must be 16-byte aligned");
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return launch_decode_f32(out, q, k_new, v_new, k_cache, v_cache, nullptr, pos, 1, H, D, max_len, scale, nullptr,
                           status, st);
}

// ---------------------------------------------------------------------------------------------
// Decode without any allocation.
//
// Some hosts of this library must not allocate device memory once they are running: a serving
// process that hands every free byte of HBM to its own cache pool at start-up has nothing left
// for a later cudaMalloc; a latency-critical decode loop cannot afford the device-wide
// synchronisation an allocation implies; and DadGPT itself sizes all of its buffers once, in
// model_alloc / kv_cache_alloc, and never allocates inside generate_tokens. For such callers the
// counters live in the fixed array below instead of a caller-provided workspace, and the bad-length
// report goes to a word of its own beside the array.
//
// The array is part of the library image: every GPU that loads libdadattn.so holds these 64 KiB until
// the process exits, whether or not this entry point is ever called. The counters are at a fixed place
// whatever the shape of a call: they are zero when the module is loaded and every call returns them to
// zero, which is the only state a call needs from its predecessors.
// A sequence that is already at max_len is skipped and noted in g_decode_noalloc_status, which
// dadattn_decode_noalloc_status() reads and clears (a symbol copy: no allocation either).
// ---------------------------------------------------------------------------------------------
namespace dadattn {
namespace {

constexpr size_t kNoAllocTicketBytes = size_t(64) << 10;
constexpr size_t kNoAllocLimitBytes = size_t(8) << 20;   // largest workspace of a shape that is taken
static __device__ __align__(256) unsigned g_decode_tickets[kNoAllocTicketBytes / sizeof(unsigned)];
static __device__ int g_decode_noalloc_status[2];   // status and its detail, as in device_status_word()

constexpr int kNoAllocMaxDevices = 64;
std::atomic<unsigned*> g_tickets_ptr[kNoAllocMaxDevices] = {};
std::atomic<int*> g_noalloc_status_ptr[kNoAllocMaxDevices] = {};

// In host code the names g_decode_tickets / g_decode_noalloc_status are only handles; the
// device addresses a kernel can use come from cudaGetSymbolAddress, per device, with that
// device current. Looked up on the first call on each device and cached.
int noalloc_setup(unsigned** tickets, int** status) {
  int dev = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return fail(DADATTN_E_UNSUPPORTED, "device ordinal %d not supported", dev);
  if (!(*tickets = g_tickets_ptr[dev]) || !(*status = g_noalloc_status_ptr[dev])) {
    DAD_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(tickets), g_decode_tickets));
    DAD_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(status), g_decode_noalloc_status));
    g_tickets_ptr[dev] = *tickets;
    g_noalloc_status_ptr[dev] = *status;
  }
  return DADATTN_OK;
}

}  // namespace
}  // namespace dadattn

extern "C" int dadattn_decode_bf16_noalloc(uint16_t* out, const uint16_t* q,
                                           const uint16_t* k_new, const uint16_t* v_new,
                                           uint16_t* k_cache, uint16_t* v_cache, int32_t* lengths,
                                           int B, int H, int D, int max_len, float scale,
                                           dadattn_stream_t stream) {
  if (int rc = check_decode_bf16(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, D, max_len))
    return rc;
  const size_t need_tickets = ticket_bytes(B, H), need_records = record_bytes(B, H, D, max_len);
  if (need_tickets > kNoAllocTicketBytes || need_records > kNoAllocLimitBytes - kNoAllocTicketBytes)
    return fail(DADATTN_E_WORKSPACE,
                "decode (no-alloc): B=%d H=%d D=%d max_len=%d counts as %zu bytes of tickets and %zu "
                "bytes of split-K records; of %zu bytes in all, %zu and %zu are taken; use "
                "dadattn_decode_bf16 with your own workspace",
                B, H, D, max_len, need_tickets, need_records, kNoAllocLimitBytes, kNoAllocTicketBytes,
                kNoAllocLimitBytes - kNoAllocTicketBytes);
  unsigned* tickets = nullptr;
  int* status = nullptr;
  if (int rc = noalloc_setup(&tickets, &status)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // never with early start: every call shares the one array with the call before it
  return launch_decode_bf16(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, D, max_len, scale, tickets, status,
                            0, st);
}

extern "C" int dadattn_decode_noalloc_status(dadattn_stream_t stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int words[2] = {0, 0};
  const int zero[2] = {0, 0};
  DAD_CUDA(cudaMemcpyFromSymbolAsync(words, g_decode_noalloc_status, sizeof(words), 0,
                                     cudaMemcpyDeviceToHost, st));
  DAD_CUDA(cudaMemcpyToSymbolAsync(g_decode_noalloc_status, zero, sizeof(zero), 0,
                                   cudaMemcpyHostToDevice, st));
  DAD_CUDA(cudaStreamSynchronize(st));
  const int host = words[0];
  if (host == DADATTN_E_TIMEOUT)
    fail(host, "decode (no-alloc): a bounded device-side wait ran out (source line %d)", words[1]);
  else if (host == DADATTN_E_ARG)
    fail(host, "decode (no-alloc): a sequence was skipped, its length is outside [0, max_len)");
  else if (host != 0)
    fail(host, "decode (no-alloc): device status %d", host);
  return host;
}

// Batched decode on fp32 caches: the arithmetic of dadattn_decode_f32 for many sequences at once.
extern "C" int dadattn_decode_f32_batched(float* out, const float* q, const float* k_new, const float* v_new,
                                          float* k_cache, float* v_cache, int32_t* lengths, int B, int H,
                                          int D, int max_len, float scale, void* workspace,
                                          size_t workspace_bytes_given, dadattn_stream_t stream) {
  if (!out || !q || !k_new || !v_new || !k_cache || !v_cache || !lengths)
    return fail(DADATTN_E_ARG, "decode: null pointer");
  if (B <= 0 || H <= 0 || max_len <= 0 || H > 65535 || static_cast<long long>(B) * H > 0x7fffffffLL)
    return fail(DADATTN_E_ARG, "decode: bad sizes B=%d H=%d max_len=%d", B, H, max_len);
  if (D != 16 && D != 32 && D != 64 && D != 128)
    return fail(DADATTN_E_UNSUPPORTED, "decode f32: unsupported D %d", D);
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k_new, 16) || !aligned(v_new, 16) ||
      !aligned(k_cache, 16) || !aligned(v_cache, 16))
    return fail(DADATTN_E_ARG, "decode: pointers must be 16-byte aligned");
  if (!workspace || !aligned(workspace, 16))
    return fail(DADATTN_E_ARG, "decode: workspace must be a 16-byte aligned device pointer");
  if (workspace_bytes_given < workspace_bytes(B, H, D, max_len))
    return fail(DADATTN_E_WORKSPACE, "decode: workspace %zu < %zu bytes", workspace_bytes_given,
                workspace_bytes(B, H, D, max_len));
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned* tickets = static_cast<unsigned*>(workspace);
  return launch_decode_f32(out, q, k_new, v_new, k_cache, v_cache, lengths, 0, B, H, D, max_len, scale, tickets,
                           status, st);
}

extern "C" int dadattn_kv_cache_fill(void* k_cache, void* v_cache, int32_t* lengths, const float* k_heads,
                                     const float* v_heads, int b, int B, int H, int n, int max_len, int D,
                                     int cache_is_bf16, dadattn_stream_t stream) {
  if (!k_cache || !v_cache || !k_heads || !v_heads) return fail(DADATTN_E_ARG, "cache fill: null pointer");
  if (B <= 0 || H <= 0 || D <= 0 || D % 4 != 0 || b < 0 || b >= B || n < 1 || n > max_len)
    return fail(DADATTN_E_ARG, "cache fill: bad sizes b=%d B=%d H=%d n=%d max_len=%d D=%d", b, B, H, n, max_len, D);
  if (!aligned(k_heads, 16) || !aligned(v_heads, 16))
    return fail(DADATTN_E_ARG, "cache fill: k_heads / v_heads must be 16-byte aligned");
  const int64_t groups = 2 * (static_cast<int64_t>(H) * n * D / 4);
  const unsigned blocks = static_cast<unsigned>((groups + 255) / 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cache_is_bf16)
    kv_cache_fill_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(static_cast<__nv_bfloat16*>(k_cache),
                                                                static_cast<__nv_bfloat16*>(v_cache), lengths,
                                                                k_heads, v_heads, b, H, n, max_len, D);
  else
    kv_cache_fill_kernel<float><<<blocks, 256, 0, st>>>(static_cast<float*>(k_cache), static_cast<float*>(v_cache),
                                                        lengths, k_heads, v_heads, b, H, n, max_len, D);
  DAD_LAUNCH_CHECK("kv_cache_fill_kernel");
  return DADATTN_OK;
}
