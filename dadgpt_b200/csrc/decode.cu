// KV-cache decode attention: one new query token per sequence against that sequence's cache.
//
// The reference runs this as 61 tiny launches per layer (per-head M=1 cuBLAS products, 256-byte
// device-to-device appends, one softmax; src/model.cpp:745-790). Here it is ONE split-K kernel
// per layer call, for any number of concurrent sequences:
//   * grid = (sequences x heads, splits); a CTA of 8 warps owns `chunk` consecutive cache rows
//     of one (sequence, head): the whole sequence when there are enough pairs to fill the GPU,
//     a slice otherwise. Splits are the slow grid dimension, so CTAs whose chunk lies
//     beyond the sequence's length (they exit at once) are scheduled last, not in between;
//   * a cache row (D elements) is read by D*sizeof(T)/16 adjacent lanes with one 128-bit load
//     each, so a warp instruction covers 512 contiguous bytes of the cache; a lane issues the K
//     and V loads of 4 row groups (128 bytes) before it consumes any, and 16-24 such warps per
//     SM keep ~100 KB in flight: memory-level parallelism is what a bandwidth-bound kernel
//     lives on;
//   * q.k partial sums are reduced over those lanes with warp shuffles; each lane keeps an
//     online-softmax state (max, sum, D/lanes accumulators) for the rows it has seen;
//   * the append is fused: the lanes that own row `len` take k_new/v_new from the token's
//     vectors, use them, and store them into the cache;
//   * split-K merge without a second kernel and without waiting: a CTA writes (unnormalised
//     out[D], max, sum) to the workspace, fences, and takes a ticket; whoever draws the last
//     ticket of its (sequence, head) merges the records and writes `out`. A second ticket per
//     sequence, taken by every CTA after it has read the length, lets the very last CTA of a
//     sequence store length + 1. Tickets are returned to zero by their last holder, so a
//     workspace zeroed once stays usable forever;
//   * launched with programmatic stream serialization: the next decode call's CTAs are already
//     resident (parked in griddepcontrol.wait) when this grid drains.
// In direct mode (one split; the fp32 single-sequence path) the CTA normalises and writes the
// output itself and no workspace is used.
#include <cfloat>
#include <climits>
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace {

constexpr int kDecodeWarps = 4;                         // consumer warps
constexpr int kDecodeThreads = (kDecodeWarps + 1) * 32;  // and one producer warp
constexpr int kTileBytes = 8192;                        // K (and V) bytes of one ring stage
constexpr int kDecodeStages = 4;
constexpr int kDecodeCtasPerSm = 3;
constexpr unsigned kTicketGroups = 32;  // first-level counters of the "all lengths read" tickets
constexpr int kMinChunk = 128;      // smallest number of cache rows worth a CTA's start and a record
constexpr int kMinRecordChunk = 256;  // what the workspace is sized for
constexpr int kTargetCtas = 592;    // 4 per SM: below that the cache is split across CTAs
constexpr int kMaxChunkSeqs = 592;  // split calls have fewer (sequence, head) pairs than kTargetCtas
constexpr int kMaxCluster = 8;      // CTAs that share a head of one sequence (portable cluster size)
constexpr int kRowsPerRank = 64;    // and the cache rows that are worth one of them

// Rows per CTA. With enough (sequence, head) pairs to fill the GPU a CTA walks a whole
// sequence (measured fastest: no records, no tickets); with few pairs the rows are split so
// that about kTargetCtas CTAs exist. Depends only on (B, H, max_len), so the workspace size and
// the kernel agree.
inline int chunk_rows(int B, int H, int max_len) {
  const long long pairs = static_cast<long long>(B) * H;
  long long want_splits = (kTargetCtas + pairs - 1) / pairs;
  if (want_splits < 1) want_splits = 1;
  long long rows = (max_len + want_splits - 1) / want_splits;
  if (rows < kMinRecordChunk) rows = kMinRecordChunk;
  rows = (rows + 127) / 128 * 128;
  return static_cast<int>(rows);
}
inline int split_count(int B, int H, int max_len) {
  const int c = chunk_rows(B, H, max_len);
  return (max_len + c - 1) / c;
}

template <typename T>
struct Elem;
template <>
struct Elem<float> {
  static constexpr int kPerLane = 4;
  __device__ static void unpack(float (&f)[4], const uint4& raw) {
    f[0] = __uint_as_float(raw.x); f[1] = __uint_as_float(raw.y);
    f[2] = __uint_as_float(raw.z); f[3] = __uint_as_float(raw.w);
  }
  __device__ static float from_float(float x) { return x; }
};
template <>
struct Elem<__nv_bfloat16> {
  static constexpr int kPerLane = 8;
  __device__ static void unpack(float (&f)[8], const uint4& raw) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  __device__ static __nv_bfloat16 from_float(float x) { return __float2bfloat16_rn(x); }
};

// Workspace: one ticket per (sequence, head), then the 1 + kTicketGroups counters of the "all
// lengths read" tickets (uint32, zero between calls), padded to 256 bytes, then the records [B*H][splits][D + 2] fp32 (unnormalised output, max, sum).
__host__ __device__ inline size_t partial_stride(int D) { return static_cast<size_t>(D) + 2; }
inline size_t record_bytes(int B, int H, int D, int max_len) {
  const int splits = split_count(B, H, max_len);
  if (splits == 1) return 0;  // every CTA finishes its (sequence, head) itself: no records
  return static_cast<size_t>(B) * H * splits * partial_stride(D) * sizeof(float);
}
inline size_t ticket_bytes(int B, int H) {
  return (sizeof(uint32_t) * (static_cast<size_t>(B) * H + 1 + kTicketGroups) + 255) / 256 * 256;
}
inline size_t workspace_bytes(int B, int H, int D, int max_len) {
  return ticket_bytes(B, H) + (record_bytes(B, H, D, max_len) + 255) / 256 * 256;
}

// ---- the kernel --------------------------------------------------------------------------------
// How a call's work is dealt out (launch_decode_batched, dadattn_decode_f32 choose):
//   kWhole    CTA = one (sequence, head), all of its rows; hardware schedules the CTAs, the longest
//             sequences first (rank by counting) when `reorder` is set
//   kChunks   few (sequence, head) pairs: the rows of all of them are cut into chunks of one length
//             that the kernel derives from the sequence lengths, CTA c takes chunks c, c + grid, ...
//   kCluster  one sequence, no workspace: the CTAs of a thread-block cluster share a head's rows and
//             merge through distributed shared memory
enum DecodeMode { kWhole = 0, kChunks = 1, kCluster = 2 };

template <typename T, int D>
struct DecodeTile {
  static constexpr int kRowBytes = D * static_cast<int>(sizeof(T));
  static constexpr int kRows = kTileBytes / kRowBytes;   // cache rows of one ring stage
  static_assert(kRows >= 1 && kTileBytes % kRowBytes == 0, "a tile is a whole number of rows");
};

struct DecodeShared {
  uint64_t full[kDecodeStages], empty[kDecodeStages];
  int abort_flag;
  int b, len, last, advance, chunk;
  float m[kDecodeWarps], l[kDecodeWarps];
  float acc[kDecodeWarps][128];
  union {
    struct {
      __align__(16) int lens[kMaxChunkSeqs];   // sequence lengths, resp. rows
      int first[kMaxChunkSeqs + 1];            // ranks (kWhole), first chunk of a sequence (kChunks)
    } seq;
    float record[kMaxCluster][130];            // kCluster: every CTA's partial result, in CTA 0
  } u;
};

// How the rows are cut: kChunks: aim at `target` chunks, never more than `capacity` records, never
// longer than `longest` rows. kCluster: `target` CTAs per head.
struct DecodeSplit {
  int target, capacity, longest;
};

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   ptx::smem_u32(smem_dst)),
               "l"(src), "r"(bytes), "r"(ptx::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// stores to the same shared-memory variable of the cluster's CTA 0
__device__ __forceinline__ uint32_t cluster_rank0_address(const void* own) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(ptx::smem_u32(own)));
  return a;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void consumers_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kDecodeWarps * 32) : "memory");
}

template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kDecodeThreads, kDecodeCtasPerSm)
decode_kernel(T* __restrict__ out, float* __restrict__ partial, unsigned* __restrict__ tickets,
              unsigned* __restrict__ seq_tickets, const T* __restrict__ q, const T* __restrict__ k_new,
              const T* __restrict__ v_new, T* __restrict__ k_cache, T* __restrict__ v_cache,
              int32_t* __restrict__ lengths, int fixed_len, int B, int H, int max_len, DecodeSplit split,
              int reorder, int early, float scale, int* __restrict__ status) {
  using namespace ptx;
  using Tile = DecodeTile<T, D>;
  constexpr int EPL = Elem<T>::kPerLane;  // elements per lane (16 bytes)
  constexpr int LPK = D / EPL;            // lanes per cache row
  constexpr int KPI = 32 / LPK;           // cache rows per warp instruction
  constexpr int kGroups = Tile::kRows / (kDecodeWarps * KPI);   // row groups of a tile per warp
  static_assert(LPK >= 1 && LPK <= 32 && (LPK & (LPK - 1)) == 0, "row must split over a warp");
  static_assert(kGroups * kDecodeWarps * KPI == Tile::kRows && D <= kDecodeWarps * 32, "tile split");

  extern __shared__ __align__(128) uint8_t smem[];
  DecodeShared& sh = *reinterpret_cast<DecodeShared*>(smem + kDecodeStages * 2 * kTileBytes);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0);
  const int lane = threadIdx.x % 32;
  const bool producer = warp == kDecodeWarps;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kDecodeStages; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], kDecodeWarps);
    }
    sh.abort_flag = 0;
    fence_mbar_init();
  }
  if (MODE == kCluster) cluster_arrive();   // (every CTA of the cluster has started: waited for below)
  // Everything this grid reads may have been written by the grid before it — unless the caller
  // has promised (dadattn_set_decode_early_start) that the grid before it does not write this
  // call's caches, lengths and workspace: then the lengths are read, and the ring is filled with
  // the first cache rows, while that grid drains, and only the token vectors wait for it.
  if (!early) pdl_wait();
  pdl_launch_dependents();

  // ---- which rows this CTA works on ----
  if (MODE == kWhole) {
    const int slot_seq = static_cast<int>(blockIdx.x) / H;
    if (reorder) {
      // CTAs are handed to the SMs in blockIdx order, and a CTA lasts as long as its sequence is
      // long: with the sequences taken longest first, the short ones fill the gaps at the end
      // instead of a long one starting last. rank(s) = number of sequences that come before s
      // (longer, or as long with a smaller index); with the count padded to a power of two n_pad
      // (32..256; padding is INT_MIN and comes last), threads share out the n_pad^2 comparisons.
      const int t = threadIdx.x;
      for (int i = t; i < 256; i += kDecodeThreads) {
        sh.u.seq.lens[i] = i < B ? lengths[i] : INT_MIN;
        sh.u.seq.first[i] = 0;
      }
      __syncthreads();
      if (t < 128) {
        const int lg = 32 - __clz(B - 1);   // n_pad = 1 << lg, 5 <= lg <= 8
        const int n_pad = 1 << lg;
        const int groups = lg < 7 ? 128 >> lg : 1;
        const int per = n_pad / groups, g = (t >> lg) & (groups - 1);
        for (int si = t & (n_pad - 1); si < n_pad; si += 128) {
          const int mine = sh.u.seq.lens[si];
          int count = 0;
#pragma unroll 4
          for (int j = g * per; j < (g + 1) * per; j += 4) {
            const int4 o = *reinterpret_cast<const int4*>(sh.u.seq.lens + j);   // broadcast reads
            count += static_cast<int>(o.x > mine) | (static_cast<int>(o.x == mine) & static_cast<int>(j + 0 < si));
            count += static_cast<int>(o.y > mine) | (static_cast<int>(o.y == mine) & static_cast<int>(j + 1 < si));
            count += static_cast<int>(o.z > mine) | (static_cast<int>(o.z == mine) & static_cast<int>(j + 2 < si));
            count += static_cast<int>(o.w > mine) | (static_cast<int>(o.w == mine) & static_cast<int>(j + 3 < si));
          }
          if (count) atomicAdd(&sh.u.seq.first[si], count);
        }
      }
      __syncthreads();
      for (int i = t; i < B; i += kDecodeThreads)
        if (sh.u.seq.first[i] == slot_seq) {
          sh.b = i;
          sh.len = sh.u.seq.lens[i];
        }
    } else if (threadIdx.x == 0) {
      sh.b = slot_seq;
      sh.len = lengths[slot_seq];
    }
  } else if (MODE == kChunks) {
    // rows of every sequence (0 where its length is invalid), the chunk length that spreads their
    // sum over split.target chunks, and each sequence's first chunk
    if (threadIdx.x == 0) sh.len = 0;
    __syncthreads();
    int rows = 0;
    for (int i = threadIdx.x; i < B; i += kDecodeThreads) {
      const int l = lengths[i];
      const bool valid = l >= 0 && l < max_len;
      sh.u.seq.lens[i] = valid ? l + 1 : 0;
      rows += valid ? l + 1 : 0;
      if (!valid && blockIdx.x == 0) atomicExch(status, DADATTN_E_ARG);
    }
    if (rows) atomicAdd(&sh.len, rows);
    __syncthreads();
    if (warp == 0) {
      const long long all = static_cast<long long>(sh.len) * H;
      const int spare = split.capacity - B * H;   // chunks beyond one per (sequence, head)
      int chunk = split.longest;
      if (spare > 0) {
        const long long even = (all + split.target - 1) / split.target, fit = (all + spare - 1) / spare;
        const long long want = max(max(even, fit), static_cast<long long>(kMinChunk));
        chunk = static_cast<int>(min(want, static_cast<long long>(chunk)));
        chunk = (chunk + Tile::kRows - 1) / Tile::kRows * Tile::kRows;
      }
      int at = 0;
      for (int i = 0; i < B; i += 32) {
        const int own = i + lane < B ? (sh.u.seq.lens[i + lane] + chunk - 1) / chunk : 0;
        int sum = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += up;
        }
        if (i + lane < B) sh.u.seq.first[i + lane] = at + sum - own;
        at += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) {
        sh.u.seq.first[B] = at;
        sh.chunk = chunk;
      }
    }
  }
  __syncthreads();  // the CTA's ticket below is taken strictly after the reads of the lengths
  // Every CTA of the call draws a ticket once it has read the lengths; whoever holds the last one
  // knows that nobody will read them again and advances them. Two levels keep the atomics off one
  // address: the CTAs are dealt into kTicketGroups groups, a CTA draws its group's ticket here, at
  // the start, and looks at it only at the very end (the round trip through L2 costs it nothing);
  // the last of each group then draws from a second counter, and the last of those advances.
  unsigned my_ticket = 0;
  if (MODE != kCluster && threadIdx.x == 0)
    my_ticket = atomicAdd(&seq_tickets[1 + blockIdx.x % kTicketGroups], 1u);

  // Segment i of this CTA: rows [row0, row1) of (b, h); false when there is none. All roles walk
  // the same list.
  struct Segment {
    int b, h, len, row0, row1, parts, record;   // parts: segments the (b, h) is cut into
  };
  auto segment = [&](int i, Segment& s) -> bool {
    if (MODE == kChunks) {
      const int per_head = sh.u.seq.first[B];
      const long long c = static_cast<long long>(blockIdx.x) + static_cast<long long>(i) * gridDim.x;
      if (c >= static_cast<long long>(per_head) * H) return false;
      s.record = static_cast<int>(c);
      s.h = s.record / per_head;
      const int r = s.record - s.h * per_head;
      int lo = 0, hi = B;                       // the last sequence whose first chunk is <= r
      while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (sh.u.seq.first[mid] <= r) lo = mid; else hi = mid;
      }
      s.b = lo;
      const int rows = sh.u.seq.lens[lo], j = r - sh.u.seq.first[lo];
      s.len = rows - 1;
      s.parts = sh.u.seq.first[lo + 1] - sh.u.seq.first[lo];
      s.record -= j;                            // records of the pair start here
      s.row0 = j * sh.chunk;
      s.row1 = min(s.row0 + sh.chunk, rows);
      return true;
    }
    if (i > 0) return false;
    s.record = 0;
    if (MODE == kCluster) {
      const int ranks = split.target, rank = static_cast<int>(blockIdx.x) % ranks;
      const int rows = fixed_len + 1, chunk = (rows + ranks - 1) / ranks;
      s.b = 0, s.h = static_cast<int>(blockIdx.x) / ranks, s.len = fixed_len, s.parts = ranks;
      s.row0 = min(rank * chunk, rows), s.row1 = min(s.row0 + chunk, rows);
      return true;
    }
    s.b = sh.b, s.h = static_cast<int>(blockIdx.x) % H, s.len = sh.len, s.parts = 1;
    s.row0 = 0, s.row1 = sh.len + 1;
    if (sh.len >= 0 && sh.len < max_len) return true;
    if (threadIdx.x == 0 && s.h == 0) atomicExch(status, DADATTN_E_ARG);
    return false;
  };

  volatile int* abort_flag = &sh.abort_flag;
  float part_acc = 0.f, part_m = -FLT_MAX, part_l = 0.f;   // kCluster: this CTA's share, one d per thread
  if (producer) {
    if (elect_one()) {
      int it = 0;
      Segment s;
      bool ok = true;
      for (int i = 0; ok && segment(i, s); ++i) {
        const size_t base = (static_cast<size_t>(s.b) * H + s.h) * max_len * D;
        const int end = min(s.row1, s.len);   // the row being appended comes from k_new / v_new
        for (int r = s.row0; r < end; r += Tile::kRows, ++it) {
          const int st = it % kDecodeStages;
          if (it >= kDecodeStages && !(ok = mbar_wait(&sh.empty[st], (it / kDecodeStages - 1) & 1, abort_flag))) break;
          const uint32_t bytes = static_cast<uint32_t>(min(Tile::kRows, end - r)) * Tile::kRowBytes;
          mbar_arrive_expect_tx(&sh.full[st], 2 * bytes);
          bulk_load(smem + st * 2 * kTileBytes, k_cache + base + static_cast<size_t>(r) * D, bytes, &sh.full[st]);
          bulk_load(smem + (st * 2 + 1) * kTileBytes, v_cache + base + static_cast<size_t>(r) * D, bytes, &sh.full[st]);
        }
      }
    }
  } else {
    if (early) pdl_wait();
    const int slot = lane / LPK, part = lane % LPK;
    int it = 0;
    bool ok = true;
    Segment s;
    for (int i = 0; segment(i, s); ++i) {
      const size_t bh = static_cast<size_t>(s.b) * H + s.h;
      const size_t vec_off = bh * D + part * EPL;
      float m = -FLT_MAX, l = 0.f, acc[EPL], qf[EPL];
      Elem<T>::unpack(qf, *reinterpret_cast<const uint4*>(q + vec_off));
#pragma unroll
      for (int e = 0; e < EPL; ++e) acc[e] = 0.f;

      // NR row groups' worth of K / V registers into the lane's online-softmax state
      auto absorb = [&](const uint4* kr, const uint4* vr, const bool* valid, auto count) {
        constexpr int NR = decltype(count)::value;
        float sc[NR];
        float m_new = m;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          float kf[EPL];
          Elem<T>::unpack(kf, kr[u]);
          float dot = 0.f;
#pragma unroll
          for (int e = 0; e < EPL; ++e) dot = fmaf(qf[e], kf[e], dot);
#pragma unroll
          for (int o = LPK / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
          sc[u] = valid[u] ? dot * scale : -FLT_MAX;
          m_new = fmaxf(m_new, sc[u]);
        }
        if (m_new > -FLT_MAX) {  // at least one row seen by this lane group so far
          const float corr = expf(m - m_new);
          l *= corr;
#pragma unroll
          for (int e = 0; e < EPL; ++e) acc[e] *= corr;
#pragma unroll
          for (int u = 0; u < NR; ++u) {
            if (!valid[u]) continue;
            const float p = expf(sc[u] - m_new);
            l += p;
            float vf[EPL];
            Elem<T>::unpack(vf, vr[u]);
#pragma unroll
            for (int e = 0; e < EPL; ++e) acc[e] = fmaf(p, vf[e], acc[e]);
          }
          m = m_new;
        }
      };

      if (warp == 0 && s.row0 <= s.len && s.row1 == s.len + 1) {   // the token being appended: use its vectors and store them
        uint4 kr = make_uint4(0, 0, 0, 0), vr = kr;
        const bool mine = slot == 0;
        if (mine) {
          kr = *reinterpret_cast<const uint4*>(k_new + vec_off);
          vr = *reinterpret_cast<const uint4*>(v_new + vec_off);
          const size_t at = (bh * max_len + s.len) * D + part * EPL;
          *reinterpret_cast<uint4*>(k_cache + at) = kr;
          *reinterpret_cast<uint4*>(v_cache + at) = vr;
        }
        absorb(&kr, &vr, &mine, std::integral_constant<int, 1>{});
      }
      const int end = min(s.row1, s.len);
      for (int r = s.row0; r < end; r += Tile::kRows, ++it) {
        const int st = it % kDecodeStages;
        if (!ok || !(ok = mbar_wait(&sh.full[st], (it / kDecodeStages) & 1, abort_flag))) break;
        const uint4* kt = reinterpret_cast<const uint4*>(smem + st * 2 * kTileBytes) + warp * kGroups * 32 + lane;
        const uint4* vt = kt + kTileBytes / 16;
        uint4 kr[kGroups], vr[kGroups];
        bool valid[kGroups];
#pragma unroll
        for (int u = 0; u < kGroups; ++u) {
          kr[u] = kt[u * 32];
          vr[u] = vt[u * 32];
          valid[u] = r + (warp * kGroups + u) * KPI + slot < end;
        }
        absorb(kr, vr, valid, std::integral_constant<int, kGroups>{});
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[st]);
      }

      // Merge the KPI row slots of the warp (lanes with equal `part`), then the warps.
#pragma unroll
      for (int o = LPK; o < 32; o <<= 1) {
        const float m_o = __shfl_xor_sync(0xffffffffu, m, o);
        const float l_o = __shfl_xor_sync(0xffffffffu, l, o);
        const float m_new = fmaxf(m, m_o);
        const float ca = m > -FLT_MAX ? expf(m - m_new) : 0.f;
        const float cb = m_o > -FLT_MAX ? expf(m_o - m_new) : 0.f;
        l = l * ca + l_o * cb;
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          const float a_o = __shfl_xor_sync(0xffffffffu, acc[e], o);
          acc[e] = acc[e] * ca + a_o * cb;
        }
        m = m_new;
      }
      if (slot == 0) {
#pragma unroll
        for (int e = 0; e < EPL; ++e) sh.acc[warp][part * EPL + e] = acc[e];
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
          const float c = sh.m[w] > -FLT_MAX ? expf(sh.m[w] - mm) : 0.f;
          ll += sh.l[w] * c;
          aa += sh.acc[w][d] * c;
        }
        if (s.parts == 1) {  // the only part of this (sequence, head): finish here
          out[bh * D + d] = Elem<T>::from_float(aa / ll);
        } else if (MODE == kCluster) {
          part_acc = aa, part_m = mm, part_l = ll;   // handed to CTA 0 below
        } else {
          float* rec = partial + (static_cast<size_t>(s.record) + s.row0 / sh.chunk) * partial_stride(D);
          rec[d] = aa;
          if (d == 0) {
            rec[D] = mm;
            rec[D + 1] = ll;
          }
        }
      }
      if (MODE == kChunks && s.parts > 1) {
        // Publish the record, then draw a ticket; the holder of the last one merges.
        __threadfence();
        consumers_sync();
        if (threadIdx.x == 0) sh.last = atomicAdd(&tickets[bh], 1u) == static_cast<unsigned>(s.parts - 1);
        consumers_sync();
        if (sh.last) {
          __threadfence();
          if (d < D) {
            const float* rec = partial + static_cast<size_t>(s.record) * partial_stride(D);
            float mm = -FLT_MAX;
            for (int j = 0; j < s.parts; ++j) mm = fmaxf(mm, __ldcg(rec + j * partial_stride(D) + D));
            float ll = 0.f, aa = 0.f;
            for (int j = 0; j < s.parts; ++j) {
              const float* rj = rec + j * partial_stride(D);
              const float c = expf(__ldcg(rj + D) - mm);
              ll += __ldcg(rj + D + 1) * c;
              aa += __ldcg(rj + d) * c;
            }
            out[bh * D + d] = Elem<T>::from_float(aa / ll);
          }
          if (threadIdx.x == 0) tickets[bh] = 0;  // ready for the next call
        }
      }
      if (MODE == kChunks) consumers_sync();   // sh.acc / sh.m are read: the next segment may write them
    }
  }

  if (MODE == kCluster && split.target > 1) {
    // The CTAs of the cluster hand their shares to CTA 0 through distributed shared memory. All
    // threads take part in both barriers; the first (arrived at on entry) says that CTA 0 runs.
    const int ranks = split.target, rank = static_cast<int>(blockIdx.x) % ranks, d = threadIdx.x;
    cluster_wait();
    if (d < D) {
      const uint32_t rec = cluster_rank0_address(&sh.u.record[rank][0]);
      st_cluster(rec + d * 4, part_acc);
      if (d == 0) {
        st_cluster(rec + D * 4, part_m);
        st_cluster(rec + D * 4 + 4, part_l);
      }
    }
    cluster_arrive();
    cluster_wait();
    if (rank == 0 && d < D) {
      float mm = -FLT_MAX;
      for (int j = 0; j < ranks; ++j) mm = fmaxf(mm, sh.u.record[j][D]);
      float ll = 0.f, aa = 0.f;
      for (int j = 0; j < ranks; ++j) {
        const float c = expf(sh.u.record[j][D] - mm);   // a share without rows has m = -FLT_MAX: 0
        ll += sh.u.record[j][D + 1] * c;
        aa += sh.u.record[j][d] * c;
      }
      out[static_cast<size_t>(blockIdx.x / ranks) * D + d] = Elem<T>::from_float(aa / ll);
    }
  } else if (MODE == kCluster) {
    cluster_wait();
  }

  if (MODE != kCluster) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned all_ctas = gridDim.x, group = blockIdx.x % kTicketGroups;
      const unsigned group_size = (all_ctas - group + kTicketGroups - 1) / kTicketGroups;
      int last = 0;
      if (my_ticket == group_size - 1) {
        seq_tickets[1 + group] = 0;   // ready for the next call
        const unsigned groups = all_ctas < kTicketGroups ? all_ctas : kTicketGroups;
        last = atomicAdd(&seq_tickets[0], 1u) == groups - 1;
        if (last) seq_tickets[0] = 0;
      }
      sh.advance = last;
    }
    __syncthreads();
    if (sh.advance) {
      for (int i = threadIdx.x; i < B; i += kDecodeThreads) {
        const int l = lengths[i];
        if (l >= 0 && l < max_len) lengths[i] = l + 1;   // a full or invalid sequence is left alone
      }
    }
  }
  if (threadIdx.x == 0 && sh.abort_flag) report_timeout(status, sh.abort_flag);
}

constexpr size_t kDecodeSmem = kDecodeStages * 2 * kTileBytes + sizeof(DecodeShared);
static_assert((kDecodeSmem + 1024) * kDecodeCtasPerSm <= 228 * 1024, "shared memory of an SM exceeded");

// The kernel's opt-in to its dynamic shared memory (a cheap host call: 0.06 us measured).
template <typename Kernel>
int allow_decode_smem(Kernel kern) {
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDecodeSmem)));
  return DADATTN_OK;
}

template <typename T, typename Raw, int DH>
int launch_decode_batched(Raw* out, const Raw* q, const Raw* k_new, const Raw* v_new, Raw* k_cache,
                          Raw* v_cache, int32_t* lengths, int B, int H, int max_len, float scale,
                          unsigned* tickets, float* partial, int* status, int early, cudaStream_t st) {
  const int splits = split_count(B, H, max_len);
  unsigned* seq_tickets = tickets + static_cast<size_t>(B) * H;
  int dev = 0, sms = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  DAD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int pairs = B * H, resident = kDecodeCtasPerSm * sms;
  DecodeSplit split = {0, 0, 0};
  int grid = pairs, reorder = 0;
  auto kern = decode_kernel<T, DH, kWhole>;
  if (splits > 1) {
    kern = decode_kernel<T, DH, kChunks>;
    split.capacity = pairs * splits;
    split.longest = chunk_rows(B, H, max_len);
    // Every (sequence, head) ends in a chunk that is half empty on average. With few pairs the
    // chunks are to fill the GPU once, remainders included; with many, about half of it.
    split.target = max(resident - pairs, resident / 2);
    grid = min(split.capacity, resident);
  } else {
    // Longest-first order pays once the CTAs no longer all fit on the GPU at the same time; the
    // in-kernel ranking handles 32..256 sequences.
    reorder = B >= 32 && B <= 256 && pairs > resident;
  }
  if (int rc = allow_decode_smem(kern)) return rc;
  DAD_CUDA(launch_pdl(kern, dim3(grid), dim3(kDecodeThreads), kDecodeSmem, st, reinterpret_cast<T*>(out), partial,
                      tickets, seq_tickets, reinterpret_cast<const T*>(q), reinterpret_cast<const T*>(k_new),
                      reinterpret_cast<const T*>(v_new), reinterpret_cast<T*>(k_cache),
                      reinterpret_cast<T*>(v_cache), lengths, 0, B, H, max_len, split, reorder, early, scale,
                      status));
  return DADATTN_OK;
}

// One fp32 sequence without a workspace: a cluster of CTAs per head.
template <int DH>
int launch_decode_one(float* out, const float* q, const float* k_new, const float* v_new, float* k_cache,
                      float* v_cache, int H, int max_len, int pos, float scale, int* status, cudaStream_t st) {
  auto kern = decode_kernel<float, DH, kCluster>;
  if (int rc = allow_decode_smem(kern)) return rc;
  int ranks = 1;
  while (ranks < kMaxCluster && ranks * kRowsPerRank < pos + 1 && H * ranks < kTargetCtas) ranks *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(H) * ranks);
  cfg.blockDim = dim3(kDecodeThreads);
  cfg.dynamicSmemBytes = kDecodeSmem;
  cfg.stream = st;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim = {static_cast<unsigned>(ranks), 1, 1};
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  const DecodeSplit split = {ranks, 0, 0};
  DAD_CUDA(cudaLaunchKernelEx(&cfg, kern, out, static_cast<float*>(nullptr), static_cast<unsigned*>(nullptr),
                              static_cast<unsigned*>(nullptr), q, k_new, v_new, k_cache, v_cache,
                              static_cast<int32_t*>(nullptr), pos, 1, H, max_len, split, 0, 0, scale, status));
  return DADATTN_OK;
}

template <int DH>
int launch_decode_bf16(uint16_t* out, const uint16_t* q, const uint16_t* k_new,
                       const uint16_t* v_new, uint16_t* k_cache, uint16_t* v_cache,
                       int32_t* lengths, int B, int H, int max_len, float scale,
                       unsigned* tickets, float* partial, int* status, int early, cudaStream_t st) {
  return launch_decode_batched<__nv_bfloat16, uint16_t, DH>(out, q, k_new, v_new, k_cache, v_cache, lengths, B,
                                                            H, max_len, scale, tickets, partial, status,
                                                            early, st);
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
  float* partial = reinterpret_cast<float*>(static_cast<char*>(workspace) + ticket_bytes(B, H));
  return D == 64 ? launch_decode_bf16<64>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H,
                                          max_len, scale, tickets, partial, status, g_decode_early, st)
                 : launch_decode_bf16<128>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H,
                                           max_len, scale, tickets, partial, status, g_decode_early, st);
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
  switch (D) {
    case 16: return launch_decode_one<16>(out, q, k_new, v_new, k_cache, v_cache, H, max_len, pos, scale, status, st);
    case 32: return launch_decode_one<32>(out, q, k_new, v_new, k_cache, v_cache, H, max_len, pos, scale, status, st);
    case 64: return launch_decode_one<64>(out, q, k_new, v_new, k_cache, v_cache, H, max_len, pos, scale, status, st);
    default: return launch_decode_one<128>(out, q, k_new, v_new, k_cache, v_cache, H, max_len, pos, scale, status, st);
  }
}

// ---------------------------------------------------------------------------------------------
// Decode without any allocation.
//
// Some hosts of this library must not allocate device memory once they are running: a serving
// process that hands every free byte of HBM to its own cache pool at start-up has nothing left
// for a later cudaMalloc; a latency-critical decode loop cannot afford the device-wide
// synchronisation an allocation implies; and DadGPT itself sizes all of its buffers once, in
// model_alloc / kv_cache_alloc, and never allocates inside generate_tokens. For such callers the
// split-K tickets and records live in the fixed array below instead of a caller-provided
// workspace, and the bad-length report goes to a fixed word instead of the lazily allocated
// status word.
//
// The array is part of the library image: every GPU that loads libdadattn.so holds these
// 8 MiB until the process exits, whether or not this entry point is ever called. Its first
// 64 KiB are the tickets, at a fixed place whatever the shape of a call: they are zero when the
// module is loaded and every call returns them to zero, which is the only state a call needs
// from its predecessors. The records behind them are written before they are read.
// A sequence that is already at max_len is skipped and noted in g_decode_noalloc_status, which
// dadattn_decode_noalloc_status() reads and clears (a symbol copy: no allocation either).
// ---------------------------------------------------------------------------------------------
namespace dadattn {
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(8) << 20;
constexpr size_t kNoAllocTicketBytes = size_t(64) << 10;
static __device__ __align__(256) unsigned char g_decode_scratch[kNoAllocScratchBytes];
static __device__ int g_decode_noalloc_status[2];   // status and its detail, as in device_status_word()

constexpr int kNoAllocMaxDevices = 64;
float* g_scratch_ptr[kNoAllocMaxDevices] = {};
int* g_noalloc_status_ptr[kNoAllocMaxDevices] = {};

// In host code the names g_decode_scratch / g_decode_noalloc_status are only handles; the
// device addresses a kernel can use come from cudaGetSymbolAddress, per device, with that
// device current. Looked up on the first call on each device and cached.
int noalloc_setup(float** scratch, int** status) {
  int dev = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return fail(DADATTN_E_UNSUPPORTED, "device ordinal %d not supported", dev);
  if (!g_scratch_ptr[dev] || !g_noalloc_status_ptr[dev]) {
    float* s = nullptr;
    int* w = nullptr;
    DAD_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&s), g_decode_scratch));
    DAD_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&w), g_decode_noalloc_status));
    g_noalloc_status_ptr[dev] = w;
    g_scratch_ptr[dev] = s;
  }
  *scratch = g_scratch_ptr[dev];
  *status = g_noalloc_status_ptr[dev];
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
  if (need_tickets > kNoAllocTicketBytes || need_records > kNoAllocScratchBytes - kNoAllocTicketBytes)
    return fail(DADATTN_E_WORKSPACE,
                "decode (no-alloc): B=%d H=%d D=%d max_len=%d needs %zu bytes of tickets and %zu "
                "bytes of split-K records; the built-in array of %zu bytes holds %zu and %zu; use "
                "dadattn_decode_bf16 with your own workspace",
                B, H, D, max_len, need_tickets, need_records,
                static_cast<size_t>(kNoAllocScratchBytes), static_cast<size_t>(kNoAllocTicketBytes),
                static_cast<size_t>(kNoAllocScratchBytes - kNoAllocTicketBytes));
  float* scratch = nullptr;
  int* status = nullptr;
  if (int rc = noalloc_setup(&scratch, &status)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned* tickets = reinterpret_cast<unsigned*>(scratch);
  float* partial = reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + kNoAllocTicketBytes);
  // never with early start: every call shares the one scratch array with the call before it
  return D == 64 ? launch_decode_bf16<64>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H,
                                          max_len, scale, tickets, partial, status, 0, st)
                 : launch_decode_bf16<128>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H,
                                           max_len, scale, tickets, partial, status, 0, st);
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
  float* partial = reinterpret_cast<float*>(static_cast<char*>(workspace) + ticket_bytes(B, H));
  switch (D) {
    case 16: return launch_decode_batched<float, float, 16>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, max_len, scale, tickets, partial, status, 0, st);
    case 32: return launch_decode_batched<float, float, 32>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, max_len, scale, tickets, partial, status, 0, st);
    case 64: return launch_decode_batched<float, float, 64>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, max_len, scale, tickets, partial, status, 0, st);
    default: return launch_decode_batched<float, float, 128>(out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, max_len, scale, tickets, partial, status, 0, st);
  }
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
