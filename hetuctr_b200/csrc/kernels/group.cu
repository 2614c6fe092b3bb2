// Preprocess, the grouping of a batch: unique keys in (owner, key) order, position lists, batch->unique map - by a
// stable radix sort of (sort key, position) pairs, sort key = owner << key_bits | key in 32 bits.
//
// A stable sort gives everything the next step's reduction wants in one go: equal keys stand together, their positions
// ascending, so no run has to be put in order afterwards, whatever its length.  All accesses are streams or scatters
// inside arrays of the batch's size (L2-resident); the only thing that grows with the table is the number of key bits:
// three passes of nine bits serve 2^27 (owner, key) pairs.  (The bitmap ranking of dedupe.cu touches table-sized
// arrays at random - bitmap, word ranks, owners, rows - which on tables of 1e8 keys is bound by address translation:
// 851,968 keys cost 158 us there, 87 here; 212,992 keys of a table of
// 3.4e7 59 and 54, the former without putting long runs in order.)
//
// A tile is 1024 * ITEMS consecutive pairs held by one block of 1024 threads, ITEMS (1..8) pairs per thread, in the
// order (warp, item, lane).  Per pass a tile ranks its pairs by digit (rank_tile), learns how many pairs of each digit stand
// in front of it, and scatters.  What is in front comes from the tiles' digit counts:
//   group_cluster   up to 65,536 pairs: ONE launch for the whole job, a cluster of one block per tile; counts are read
//                   through distributed shared memory, passes are separated by cluster barriers.
//   group_pass ...  more tiles: histogram of all digits, one launch per pass (a tile publishes its counts and waits,
//                   bounded, for those of the tiles before it - blocks are dispatched in index order, so these are
//                   running or done), group_finish.  Chained launches: 212,992 keys of a table of 3.4e7 61 us alone, 52 so.
#include <cooperative_groups.h>

#include "common.cuh"

namespace hctr {

namespace cg = cooperative_groups;

constexpr int kTileThreads = 1024;
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kMaxItems = 8;
constexpr int kMaxDigits = 512;
constexpr int kMaxPasses = 4;
constexpr u32 kMaxTiles = HCTR_GROUP_MAX_TILES;
constexpr u32 kMaxCluster = 16;  // (more than 8 blocks is not portable: see cluster_blocks)
// Tiles of the multi-launch form before a thread takes more pairs: a tile adds up the counts of all tiles in front of
// it, and ranking and scattering a tile cost what they cost per SM, so the batch is spread over about as many SMs as
// there are (212,992 keys as 26 tiles of 8192: 16 us per pass, as 104 tiles of 2048: 9).
constexpr u32 kSpreadTiles = 112;

struct TileSmem {
  uint16_t cnt[kTileWarps][kMaxDigits];  // pairs of a digit in a warp, then in the warps before it
  u32 total[kMaxDigits];                 // pairs of a digit in the tile (read by the other blocks of a cluster)
  u32 start[kMaxDigits];                 // where the tile's first pair of a digit goes
  u32 warp_sum[kTileWarps];
  u32 heads;                             // heads in the tile (cluster)
};

struct GroupPlan {
  int passes, digit_bits, key_bits;
  u32 sentinel;  // sort key of an invalid key: behind all others
};

__device__ __forceinline__ u32 digit_of(u32 sk, const GroupPlan &g, int pass) {
  return (sk >> (pass * g.digit_bits)) & ((1u << g.digit_bits) - 1u);
}

__device__ __forceinline__ u32 sort_key(const hctr_group_args &a, const GroupPlan &g, size_t i) {
  const long long key = a.keys[i];
  u32 owner = 0;
  bool ok = key >= 0 && (size_t)key < a.length;
  if (ok && a.nrank > 1) {
    owner = a.owner_of[key];
    ok = owner < (u32)a.nrank;
  }
  if (ok) return (owner << g.key_bits) | (u32)key;  // (key_bits < 32 whenever owner can be non-zero)
  atomicOr(&a.meta[HCTR_META_ERR], HCTR_ERR_KEY_RANGE);
  return g.sentinel;
}

// index in the batch of a thread's j-th pair
template <int ITEMS>
__device__ __forceinline__ u32 pair_index(u32 tile, int j) {
  return tile * (kTileThreads * ITEMS) + (threadIdx.x >> 5) * (32 * ITEMS) + j * 32 + (threadIdx.x & 31);
}

// Barrier over the cluster's threads, global and shared memory included; the warps are brought together first (divergent
// code stands in front of every use).
__device__ __forceinline__ void sync_cluster() {
  __syncwarp();
  cg::this_cluster().sync();
}

// Exclusive prefix of v over the block's threads, in thread order; *total = sum.  Two barriers.
__device__ __forceinline__ u32 block_prefix(u32 v, u32 *warp_sum, u32 *total) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32 incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (unsigned)d) incl += t;
  }
  __syncthreads();  // warp_sum may still be read by an earlier call
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  u32 w = warp_sum[lane], wi = w;  // every warp scans the 32 sums for itself
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, wi, d);
    if (lane >= (unsigned)d) wi += t;
  }
  *total = __shfl_sync(0xffffffffu, wi, 31);
  return incl - v + __shfl_sync(0xffffffffu, wi - w, warp);
}

// Stable rank of every pair among the tile's pairs of the same digit; s.total = pairs per digit.  A warp counts in its
// own row of s.cnt: equal digits among its lanes find each other with one ballot per digit bit, the lowest lane moves
// the counter.  (__match_any_sync instead of the ballots: 1650 cycles per item with 32 warps on the SM, 1000 with them.)
template <int ITEMS>
__device__ __forceinline__ void rank_tile(TileSmem &s, const u32 (&digit)[ITEMS], const bool (&act)[ITEMS],
                                          int digit_bits, u32 (&rank)[ITEMS]) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint16_t *mine = s.cnt[warp];
#pragma unroll
  for (int k = 0; k < kMaxDigits / 64; k++) reinterpret_cast<u32 *>(mine)[k * 32 + lane] = 0;
  unsigned peers[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; j++) peers[j] = __ballot_sync(0xffffffffu, act[j]);
  for (int b = 0; b < digit_bits; b++) {
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const bool one = (digit[j] >> b) & 1u;
      const unsigned m = __ballot_sync(0xffffffffu, one);
      peers[j] &= one ? m : ~m;
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const unsigned leader = act[j] ? (unsigned)(__ffs(peers[j]) - 1) : lane;
    u32 old = 0;
    if (act[j] && lane == leader) {
      old = mine[digit[j]];
      mine[digit[j]] = (uint16_t)(old + __popc(peers[j]));
    }
    old = __shfl_sync(0xffffffffu, old, leader);
    rank[j] = old + __popc(peers[j] & ((1u << lane) - 1u));
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < kMaxDigits) {
    u32 sum = 0;
#pragma unroll
    for (int w0 = 0; w0 < kTileWarps; w0 += 16) {
      u32 c[16];
#pragma unroll
      for (int w = 0; w < 16; w++) c[w] = s.cnt[w0 + w][threadIdx.x];
#pragma unroll
      for (int w = 0; w < 16; w++) {
        s.cnt[w0 + w][threadIdx.x] = (uint16_t)sum;
        sum += c[w];
      }
    }
    s.total[threadIdx.x] = sum;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (act[j]) rank[j] += s.cnt[warp][digit[j]];
}

// The sorted pairs of one tile -> unique keys, runs, positions.  before(heads) returns the number of heads (first pairs
// of a key) in the tiles in front, given the tile's own; every thread calls it.
// broken: a pass gave up its wait, so pairs may be missing and old ones in their place - none of them is looked at, and
// the batch comes out with no keys.
template <int ITEMS, class F>
__device__ __forceinline__ void finish_tile(TileSmem &s, const hctr_group_args &a, const GroupPlan &g,
                                            const u64 *pairs, u32 tile, bool broken, F before) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32 n = (u32)a.batch;
  u32 sk[ITEMS], pos[ITEMS], prev[ITEMS], next[ITEMS], heads[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const u32 q = pair_index<ITEMS>(tile, j);
    const u64 w = q < n && !broken ? __ldcg(pairs + q) : ((u64)g.sentinel << 32 | q);
    sk[j] = (u32)(w >> 32);
    pos[j] = (u32)w;
    // neighbours across the warp's edges (the others come by shuffle)
    prev[j] = next[j] = g.sentinel;
    if (lane == 0 && q > 0 && q < n) prev[j] = (u32)(__ldcg(pairs + q - 1) >> 32);
    if (lane == 31 && q + 1 < n) next[j] = (u32)(__ldcg(pairs + q + 1) >> 32);
  }
  u32 in_warp = 0;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const u32 up = __shfl_up_sync(0xffffffffu, sk[j], 1), down = __shfl_down_sync(0xffffffffu, sk[j], 1);
    if (lane != 0) prev[j] = up;
    if (lane != 31) next[j] = down;
    const u32 q = pair_index<ITEMS>(tile, j);
    heads[j] = __ballot_sync(0xffffffffu, sk[j] != g.sentinel && (q == 0 || prev[j] != sk[j]));
    in_warp += __popc(heads[j]);
  }
  // what the heads need from elsewhere, all of it in flight while the tiles add up their counts
  int32_t row[ITEMS];
  bool heavy[ITEMS], very[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const u32 q = pair_index<ITEMS>(tile, j);
    const bool head = (heads[j] >> lane) & 1u;
    row[j] = head ? a.pos_row[pos[j]] : 0;
    const bool run = head && next[j] == sk[j];
    heavy[j] = run && q + HCTR_LIGHT_RUN < n && (u32)(__ldcg(pairs + q + HCTR_LIGHT_RUN) >> 32) == sk[j];
    very[j] = run && q + HCTR_LONG_RUN < n && (u32)(__ldcg(pairs + q + HCTR_LONG_RUN) >> 32) == sk[j];
  }
  __syncthreads();
  if (lane == 0) s.warp_sum[warp] = in_warp;
  __syncthreads();
  const u32 w = s.warp_sum[lane];
  const u32 all = __reduce_add_sync(0xffffffffu, w);
  const u32 first = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
  u32 base = before(all) + first;  // heads in front of this warp's next item
  const u32 key_mask = g.key_bits >= 32 ? 0xffffffffu : (1u << g.key_bits) - 1u;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const u32 q = pair_index<ITEMS>(tile, j);
    const bool valid = sk[j] != g.sentinel;
    const bool head = (heads[j] >> lane) & 1u;
    const u32 upto = base + __popc(heads[j] & ((1u << lane) - 1u));  // heads at positions before q
    const u32 u = upto + (head ? 1u : 0u) - 1u;                      // this pair's unique index (if valid)
    base += __popc(heads[j]);
    if (q < n) {
      if (q % HCTR_CHUNK_POS == 0) a.chunk_key[q / HCTR_CHUNK_POS] = upto;
      a.sorted_pos[q] = pos[j];
      if (a.idx_map) a.idx_map[pos[j]] = valid ? (int32_t)u : -1;
      const u32 owner = a.nrank > 1 ? sk[j] >> g.key_bits : 0u;
      if (head) {
        a.run_start[u] = q;
        a.uniq[u] = sk[j] & key_mask;
        a.uniq_row[u] = row[j];
        if (a.nrank > 1) {
          a.uniq_owner[u] = (uint8_t)owner;
          // segments of the owners between the key before and this one start here
          const u32 from = q == 0 ? 0u : (prev[j] >> g.key_bits) + 1u;
          for (u32 p = from; p <= owner; p++) a.meta[HCTR_META_SEG + p] = u;
        }
        // long runs are listed from the front, very long ones from the back as well (both fit: a very long run is one
        // entry of each and takes the place of several long ones)
        if (heavy[j]) a.heavy_list[atomicAdd(&a.meta[HCTR_META_NHEAVY], 1u)] = u;
        if (very[j]) a.heavy_list[n / 32 + 1 - atomicAdd(&a.meta[HCTR_META_NLONG], 1u)] = u;
      }
      if (valid && (q + 1 == n || next[j] == g.sentinel)) {  // the last key of the batch
        const u32 U = u + 1;
        a.meta[HCTR_META_UNIQUE] = U;
        a.run_start[U] = q + 1;
        a.chunk_key[(q + HCTR_CHUNK_POS) / HCTR_CHUNK_POS] = U;
        for (u32 p = owner + 1; p <= (u32)a.nrank; p++) a.meta[HCTR_META_SEG + p] = U;
      }
      if (q == 0 && !valid) a.run_start[0] = a.chunk_key[0] = 0;  // nothing but invalid keys
    }
  }
  if (n == 0 && tile == 0 && threadIdx.x == 0) a.run_start[0] = a.chunk_key[0] = 0;
}

// One launch, a cluster of up to 16 tiles.  Bound: a chain of short phases (per pass ~2 us of ranking and two cluster barriers).
template <int ITEMS>
__global__ void __launch_bounds__(kTileThreads) group_cluster(hctr_group_args a, GroupPlan g) {
  extern __shared__ __align__(16) unsigned char group_smem[];
  TileSmem &s = *reinterpret_cast<TileSmem *>(group_smem);
  cg::cluster_group cluster = cg::this_cluster();
  const u32 tile = blockIdx.x, tiles = gridDim.x;
  const unsigned tid = threadIdx.x;
  const u32 n = (u32)a.batch;
  const u64 *in = nullptr;
  u64 *out = reinterpret_cast<u64 *>(a.pairs0);
  for (int pass = 0; pass < g.passes; pass++) {
    u64 pair[ITEMS];
    u32 digit[ITEMS], rank[ITEMS];
    bool act[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const u32 q = pair_index<ITEMS>(tile, j);
      act[j] = q < n;
      pair[j] = 0;
      if (act[j]) pair[j] = pass == 0 ? ((u64)sort_key(a, g, q) << 32) | q : __ldcg(in + q);
      digit[j] = digit_of((u32)(pair[j] >> 32), g, pass);
    }
    rank_tile<ITEMS>(s, digit, act, g.digit_bits, rank);
    sync_cluster();
    u32 all = 0, before = 0;
    if (tid < kMaxDigits) {
#pragma unroll
      for (u32 t = 0; t < kMaxCluster; t++) {
        const u32 v = t < tiles ? *cluster.map_shared_rank(&s.total[tid], t < tiles ? t : tile) : 0u;
        if (t < tile) before += v;
        all += v;
      }
    }
    u32 sum;
    const u32 base = block_prefix(all, s.warp_sum, &sum);
    if (tid < kMaxDigits) s.start[tid] = base + before;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++)
      if (act[j]) out[s.start[digit[j]] + rank[j]] = pair[j];
    sync_cluster();  // pairs in place for everybody; nobody reads s.total any more
    in = out;
    out = reinterpret_cast<u64 *>(in == reinterpret_cast<u64 *>(a.pairs0) ? a.pairs1 : a.pairs0);
  }
  finish_tile<ITEMS>(s, a, g, in, tile, false, [&](u32 heads) -> u32 {
    if (tiles == 1) return 0u;
    if (tid == 0) s.heads = heads;
    sync_cluster();
    u32 before = 0;
    for (u32 t = 0; t < tile; t++) before += *cluster.map_shared_rank(&s.heads, t);
    return before;
  });
  sync_cluster();  // the blocks behind have read this block's count
}

// Sort keys of the batch and, for every pass, how many have each digit (hist: all-zero on entry).
__global__ void __launch_bounds__(512) group_histogram(hctr_group_args a, GroupPlan g) {
  __shared__ u32 h[kMaxPasses][kMaxDigits];
  for (int i = threadIdx.x; i < g.passes * kMaxDigits; i += 512) (&h[0][0])[i] = 0;
  __syncthreads();
  for (size_t i = (size_t)blockIdx.x * 512 + threadIdx.x; i < a.batch; i += (size_t)gridDim.x * 512) {
    const u32 sk = sort_key(a, g, i);
    a.sort_keys[i] = sk;
    for (int p = 0; p < g.passes; p++) atomicAdd(&h[p][digit_of(sk, g, p)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < g.passes * kMaxDigits; i += 512) {
    const u32 v = (&h[0][0])[i];
    if (v) atomicAdd(&a.hist[i], v);
  }
}

template <int ITEMS>
__global__ void __launch_bounds__(kTileThreads) group_pass(hctr_group_args a, GroupPlan g, int pass) {
  extern __shared__ __align__(16) unsigned char group_smem[];
  TileSmem &s = *reinterpret_cast<TileSmem *>(group_smem);
  const u32 tile = blockIdx.x;
  const unsigned tid = threadIdx.x;
  const u32 n = (u32)a.batch;
  const u64 *in = reinterpret_cast<const u64 *>(pass & 1 ? a.pairs0 : a.pairs1);
  u64 *out = reinterpret_cast<u64 *>(pass & 1 ? a.pairs1 : a.pairs0);
  u64 pair[ITEMS];
  u32 digit[ITEMS], rank[ITEMS];
  bool act[ITEMS];
  wait_predecessor();
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const u32 q = pair_index<ITEMS>(tile, j);
    act[j] = q < n;
    pair[j] = 0;
    if (act[j]) pair[j] = pass == 0 ? ((u64)__ldcg(a.sort_keys + q) << 32) | q : __ldcg(in + q);
    digit[j] = digit_of((u32)(pair[j] >> 32), g, pass);
  }
  rank_tile<ITEMS>(s, digit, act, g.digit_bits, rank);
  u32 *flags = a.tile_flags + pass * kMaxTiles;
  if (tid < kMaxDigits) a.tile_counts[tile * kMaxDigits + tid] = s.total[tid];
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flags + tile), "r"(a.epoch) : "memory");
  }
  u32 sum;
  const u32 base = block_prefix(tid < kMaxDigits ? a.hist[pass * kMaxDigits + tid] : 0u, s.warp_sum, &sum);
  if (tid < kMaxDigits) s.start[tid] = base;
  for (u32 t = tid; t < tile; t += kTileThreads) {
    u32 v, spins = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + t) : "memory");
      if (v == a.epoch) break;
      if (++spins > 4000000u) {  // ~ a second: a predecessor never published
        atomicOr(&a.meta[HCTR_META_ERR], HCTR_ERR_TIMEOUT);
        break;
      }
      __nanosleep(40);
    }
  }
  __syncthreads();
  u32 before = 0;
#pragma unroll 16
  for (u32 t = tid / kMaxDigits; t < tile; t += kTileThreads / kMaxDigits)
    before += __ldcg(a.tile_counts + t * kMaxDigits + tid % kMaxDigits);
  atomicAdd(&s.start[tid % kMaxDigits], before);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (act[j]) {
      const u32 to = s.start[digit[j]] + rank[j];
      if (to < n) out[to] = pair[j];  // (always, unless a wait ran out)
    }
}

template <int ITEMS>
__global__ void __launch_bounds__(kTileThreads) group_finish(hctr_group_args a, GroupPlan g) {
  __shared__ TileSmem s;
  const u64 *in = reinterpret_cast<const u64 *>(g.passes & 1 ? a.pairs0 : a.pairs1);
  wait_predecessor();
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < g.passes * kMaxDigits; i += kTileThreads) a.hist[i] = 0;  // at rest again
  // (the passes are over; a bit that a tile of this launch sets while others start changes nothing that they index)
  finish_tile<ITEMS>(s, a, g, in, blockIdx.x, grouping_broke_off(a.meta), [&](u32 heads) {
    return chained_cta_prefix(reinterpret_cast<u64 *>(a.chain_scratch), a.epoch, blockIdx.x, heads,
                              &a.meta[HCTR_META_ERR]);
  });
}

// idx_map[position] = unique index, from the finished grouping (for callers that did not ask for it there)
__global__ void __launch_bounds__(256) group_index_map(const u32 *__restrict__ meta, const u32 *__restrict__ run_start,
                                                       const u32 *__restrict__ sorted_pos, int32_t *__restrict__ idx_map) {
  const u32 U = unique_of(meta);
  const u32 lane = threadIdx.x & 31, n_warps = gridDim.x * 8;
  for (u32 u = blockIdx.x * 8 + (threadIdx.x >> 5); u < U; u += n_warps)
    for (u32 q = run_start[u] + lane; q < run_start[u + 1]; q += 32) idx_map[sorted_pos[q]] = (int32_t)u;
}

// What hctr_group_keys leaves for the reduction, from runs that were made otherwise.
__global__ void __launch_bounds__(256) run_chunks(u32 n, const u32 *__restrict__ run_start, u32 *__restrict__ chunk_key,
                                                  u32 *__restrict__ heavy_list, u32 *meta) {
  if (grouping_broke_off(meta)) return;
  const u32 U = meta[HCTR_META_UNIQUE];
  for (u32 u = blockIdx.x * 256 + threadIdx.x; u <= U; u += gridDim.x * 256) {
    // chunks that begin behind the start of the key before and not behind this one's
    const u32 here = u < U ? run_start[u] : run_start[U] + HCTR_CHUNK_POS - 1;
    const u32 from = u == 0 ? 0u : run_start[u - 1] / HCTR_CHUNK_POS + 1;
    for (u32 c = from; c <= here / HCTR_CHUNK_POS; c++) chunk_key[c] = u;
    if (u < U && run_start[u + 1] - here > HCTR_LONG_RUN) heavy_list[n / 32 + 1 - atomicAdd(&meta[HCTR_META_NLONG], 1u)] = u;
  }
}

}  // namespace hctr

using namespace hctr;

static bool group_plan(size_t length, int nrank, GroupPlan *g) {
  if (length == 0) length = 1;
  int key_bits = 0;
  while (key_bits < 40 && ((size_t)1 << key_bits) < length) key_bits++;
  // every sort key is below the sentinel, the all-ones pattern of `bits` bits
  const unsigned long long last = ((unsigned long long)(nrank - 1) << key_bits) + (length - 1);
  int bits = 1;
  while (bits < 63 && ((1ull << bits) - 1) <= last) bits++;
  if (bits > 32) return false;
  g->key_bits = key_bits;
  g->passes = (bits + 8) / 9;
  g->digit_bits = (bits + g->passes - 1) / g->passes;
  g->sentinel = bits == 32 ? 0xffffffffu : (1u << bits) - 1u;
  return true;
}

template <int ITEMS>
static cudaLaunchConfig_t cluster_config(u32 tiles, cudaStream_t s, cudaLaunchAttribute *at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles);
  cfg.blockDim = dim3(kTileThreads);
  cfg.dynamicSmemBytes = sizeof(TileSmem);
  cfg.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = tiles;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Blocks a cluster of this kernel may have here: 16 where the device places such a cluster, else the portable 8.
static u32 cluster_blocks() {
  static PerDevice most;
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) return 8u;
  return (u32)most.get(device, [] {
    bool big = true;
    for (const void *k : {(const void *)group_cluster<1>, (const void *)group_cluster<2>, (const void *)group_cluster<4>})
      big = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess && big;
    int clusters = 0;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config<4>(kMaxCluster, nullptr, &at);
    big = big && cudaOccupancyMaxActiveClusters(&clusters, group_cluster<4>, &cfg) == cudaSuccess && clusters > 0;
    cudaGetLastError();
    return big ? (int)kMaxCluster : 8;
  });
}

template <int ITEMS>
static int launch_cluster(const hctr_group_args &a, const GroupPlan &g, cudaStream_t s) {
  const u32 tiles = a.batch ? (u32)((a.batch + kTileThreads * ITEMS - 1) / (kTileThreads * ITEMS)) : 1u;
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = cluster_config<ITEMS>(tiles, s, &at);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, group_cluster<ITEMS>, a, g);
  count_launches(1);
  return launch_status(e);
}

template <int ITEMS>
static int launch_passes(const hctr_group_args &a, const GroupPlan &g, cudaStream_t s) {
  const u32 tiles = (u32)((a.batch + kTileThreads * ITEMS - 1) / (kTileThreads * ITEMS));
  group_histogram<<<kSMs, 512, 0, s>>>(a, g);
  for (int p = 0; p < g.passes; p++)
    if (const int e = launch_chained(group_pass<ITEMS>, tiles, kTileThreads, sizeof(TileSmem), s, a, g, p)) return e;
  if (const int e = launch_chained(group_finish<ITEMS>, tiles, kTileThreads, 0, s, a, g)) return e;
  count_launches(g.passes + 2);
  return launch_status();
}

extern "C" int hctr_group_fits(size_t batch, size_t length, int nrank) {
  GroupPlan g;
  return batch <= (size_t)kTileThreads * kMaxItems * kMaxTiles && group_plan(length, nrank, &g) ? 1 : 0;
}

extern "C" int hctr_group_is_small(size_t batch) { return batch <= (size_t)kTileThreads * 4 * cluster_blocks() ? 1 : 0; }

extern "C" int hctr_group_keys(const hctr_group_args *ap, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const hctr_group_args a = *ap;
  GroupPlan g;
  if (a.epoch == 0 || a.batch > (size_t)kTileThreads * kMaxItems * kMaxTiles || !group_plan(a.length, a.nrank, &g))
    return (int)cudaErrorInvalidValue;
  // One launch while a cluster's blocks take at most four pairs per thread: beyond, the few SMs of a cluster take longer
  // (53,248 keys with eight pairs per thread on eight SMs: 61 us) than the launches of the other form cost.
  const size_t one = (size_t)kTileThreads * cluster_blocks();
  if (a.batch <= one) return launch_cluster<1>(a, g, s);
  if (a.batch <= one * 2) return launch_cluster<2>(a, g, s);
  if (a.batch <= one * 4) return launch_cluster<4>(a, g, s);
  const size_t per = (size_t)kTileThreads * kSpreadTiles;
  return a.batch <= per       ? launch_passes<1>(a, g, s)
         : a.batch <= per * 2 ? launch_passes<2>(a, g, s)
         : a.batch <= per * 4 ? launch_passes<4>(a, g, s)
                              : launch_passes<8>(a, g, s);
}

extern "C" int hctr_group_index_map(const uint32_t *meta, const uint32_t *run_start, const uint32_t *sorted_pos,
                                    int32_t *idx_map, void *stream) {
  group_index_map<<<kSMs * 4, 256, 0, (cudaStream_t)stream>>>(meta, run_start, sorted_pos, idx_map);
  count_launches(1);
  return launch_status();
}

extern "C" int hctr_run_chunks(size_t batch, const uint32_t *run_start, uint32_t *chunk_key, uint32_t *heavy_list,
                               uint32_t *meta, void *stream) {
  run_chunks<<<kSMs * 4, 256, 0, (cudaStream_t)stream>>>((u32)batch, run_start, chunk_key, heavy_list, meta);
  count_launches(1);
  return launch_status();
}
