// Gradient side of a step on a single-rank table: for every unique key of the previous batch, s = (sum of its gradient
// rows, in ascending batch position) * (-lr), then row += s and version += count.  The sum order and the single multiply
// are the reference's (csrc/core/generate_query.cu:34-40), so results are bit-identical to a sequential evaluation.
// (Tables with peers also push and hold rows: update.cu.)
//
// ONE launch, one resident round of blocks.  Bound: HBM (every gradient row once, every touched table row read and
// written).  What stands in the way is that a key's rows must be added one after the other, and that CTR batches mix
// keys seen once with keys seen thousands of times.  Three kinds of work, longest first:
//   very long runs (> HCTR_LONG_RUN rows)   a block takes 32 columns of one key: all warps copy rows into a ring of shared
//                         memory stages (cp.async), one warp adds them - one addition per lane and row, four cycles
//                         apart.  Slicing the columns puts W/32 blocks on one key and keeps 48 KB of one slice in flight.
//   long runs (> HCTR_LIGHT_RUN rows)       a warp takes 32 columns of one key, with a ring of its own: 56 rows in flight.
//                         (One warp per key with eight whole rows in registers: 26 us per run on average, 84 for 256 rows.)
//   everything else       a warp takes the keys whose runs start in 32 positions of sorted_pos (chunk_key), so all warps
//                         get about the same number of rows however the runs are distributed.  LANES lanes move one
//                         row; the lane groups share the chunk's keys by position.  Gradient rows and the keys' table
//                         rows come through shared memory (cp.async; a lane reads back what it copied itself, so
//                         nothing is waited for but the copy): two rounds of four positions are in flight without a
//                         register held for them, and the next chunk's indices arrive meanwhile.
// The pieces are dealt out, not drawn: a counter for 7,372 pieces of work cost more than the unevenness it removes (107 us
// against 51).  They are dealt in the order of their lists: the very long runs of 638,976 x 64 put 36 tiles on the worst block
// and 9.5 on the average one, those of 212,992 x 128 8 and 2.5.  Rounds of two or eight positions and four blocks per SM were slower.
// Measured alone: 212,992 x 128 (66,251 keys, 177 MB) 40 us, 106,496 x 256 39, 638,976 x 64 (220 MB) 64, 851,968 x 32
// (839,991 keys, 324 MB) 103; the two kernels these took the place of 60 side by side, 50, 110 and 146.
#include <algorithm>

#include "rowops.cuh"

namespace hctr {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kResident = 3;        // blocks per SM
constexpr u32 kSliceFloats = 32;    // columns of a slice (long and very long runs)
constexpr int kStages = 4;          // very long runs: ring of kStages tiles
constexpr u32 kStageRows = 128;     // rows of a tile
constexpr u32 kWarpStages = 8;      // long runs: ring of kWarpStages tiles per warp
constexpr u32 kWarpStageRows = 8;   // rows of a tile
constexpr u32 kRound = 4;           // short runs: positions of a round, two rounds in flight
constexpr u32 kChunkMax = 64;       // positions of one chunk's short runs: 31 before its end + 32 of the last one
constexpr u32 kRingBytes = 2 * kRound * 2 * 32 * 16;  // per warp: a gradient and a table row for each position in flight
constexpr u32 kWarpBytes = kRingBytes + kChunkMax * sizeof(uint2);
constexpr u32 kBlockBytes = kWarps * kWarpBytes;
constexpr u32 kNoPosition = 0xffffffffu;
static_assert(kStages * kStageRows * kSliceFloats * sizeof(float) <= kBlockBytes &&
                  kWarpStages * kWarpStageRows * kSliceFloats * sizeof(float) <= kRingBytes, "the rings share one area");

// Gradients that arrive over the host link come in pieces of ascending batch positions, and a key can be summed as soon as
// its last one is there: a launch with WINDOW takes the keys whose last position lies in [lo, hi).
struct Window {
  u32 lo, hi;
  __device__ __forceinline__ bool has(u32 last) const { return last - lo < hi - lo; }
};

// More batch positions for the row's version.  Nobody else writes it: the atomic only saves waiting for the old value.
__device__ __forceinline__ void count_updates(const hctr_local_reduce_args &a, int32_t row, u32 count) {
  atomicAdd(reinterpret_cast<u64 *>(a.version) + row, (u64)count);
}

// Gradient rows are read exactly once: their copies carry an evict-first L2 policy so that 100+ MB of them per step do
// not push the table rows out of the cache.
__device__ __forceinline__ u64 l2_evict_first_policy() {
  u64 p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
template <int V>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, u64 policy) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if (V == 4)
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "l"(policy) : "memory");
  else
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], %3, %2;" ::"r"(s), "l"(gmem), "l"(policy), "n"(V * 4)
                 : "memory");
}
template <int V>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if (V == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(V * 4) : "memory");
}

// ---- very long runs ----------------------------------------------------------------------------
template <int V, bool WINDOW>
__device__ __forceinline__ void sum_very_long(const hctr_local_reduce_args &a, Window win, float *ring) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32 W = (u32)a.width, slices = (W + kSliceFloats - 1) / kSliceFloats;
  const u32 n_tasks = a.meta[HCTR_META_NLONG] * slices;
  constexpr u32 kRowsPerWarp = kStageRows / kWarps, kLanesPerRow = kSliceFloats / V;
  const unsigned sub = lane / kLanesPerRow, col = lane % kLanesPerRow * V;
  const u64 once = l2_evict_first_policy();
  for (u32 task = blockIdx.x; task < n_tasks; task += gridDim.x) {
    const u32 u = a.heavy_list[a.batch / 32 + 1 - task / slices];
    const u32 col0 = task % slices * kSliceFloats, cols = min(kSliceFloats, W - col0);
    const u32 l = a.run_start[u], len = a.run_start[u + 1] - l;
    if (WINDOW && !win.has(a.sorted_pos[l + len - 1])) continue;  // (the same for the whole block)
    const u32 n_tiles = (len + kStageRows - 1) / kStageRows;
    // positions come two tiles at a time, one per lane: lane i has tile i / 16 of the two, row i % 16 of the warp's
    constexpr u32 kAtOnce = 32 / kRowsPerWarp;
    auto positions = [&](u32 group) {
      const u32 r = (group * kAtOnce + lane / kRowsPerWarp) * kStageRows + warp * kRowsPerWarp + lane % kRowsPerWarp;
      return r < len ? a.sorted_pos[l + r] : 0u;
    };
    u32 here = positions(0), ahead = positions(1), issued = 0;
    auto issue = [&]() {
      if (issued < n_tiles) {
        if (issued != 0 && issued % kAtOnce == 0) {
          here = ahead;
          ahead = positions(issued / kAtOnce + 1);
        }
        float *stage = ring + (size_t)(issued % kStages) * kStageRows * kSliceFloats;
#pragma unroll
        for (u32 i = 0; i < kRowsPerWarp / V; i++) {
          const u32 r = i * V + sub, rr = warp * kRowsPerWarp + r;
          const u32 p = __shfl_sync(0xffffffffu, here, issued % kAtOnce * kRowsPerWarp + r);
          if (issued * kStageRows + rr < len && col < cols)
            cp_async<V>(stage + rr * kSliceFloats + col, a.grad + (size_t)p * W + col0 + col, once);
        }
        issued++;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // one group per tile, even an empty one
    };
#pragma unroll
    for (int t = 0; t < kStages - 1; t++) issue();
    float sum = 0.f;
    for (u32 tile = 0; tile < n_tiles; tile++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      // everybody's copies of this tile have landed, and its predecessor, whose stage is filled next, has been added
      __syncthreads();
      issue();
      if (warp == 0) {
        const float *src = ring + (size_t)(tile % kStages) * kStageRows * kSliceFloats + lane;
        const u32 nr = min(kStageRows, len - tile * kStageRows);
        u32 r = 0;
        for (; r + 32 <= nr; r += 32) {
          float v[32];
#pragma unroll
          for (int k = 0; k < 32; k++) v[k] = src[(r + k) * kSliceFloats];
#pragma unroll
          for (int k = 0; k < 32; k++) sum = __fadd_rn(sum, v[k]);
        }
        for (; r < nr; r++) sum = __fadd_rn(sum, src[r * kSliceFloats]);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (warp == 0 && lane < cols) {
      const int32_t row = a.uniq_row[u];
      if (col0 == 0 && lane == 0) count_updates(a, row, len);
      float *e = a.embedding + (size_t)row * W + col0 + lane;
      *e = __fadd_rn(*e, __fmul_rn(sum, a.neg_lr));
    }
    __syncthreads();  // the ring is free for the next key
  }
}

// ---- long runs: one warp, 32 columns of one key -----------------------------------------------------
template <int V, bool WINDOW>
__device__ __forceinline__ void sum_long(const hctr_local_reduce_args &a, Window win, u32 u, u32 slice, float *ring) {
  const unsigned lane = threadIdx.x & 31;
  const u32 l = a.run_start[u], len = a.run_start[u + 1] - l;
  const int32_t row = a.uniq_row[u];
  if (len > HCTR_LONG_RUN) return;  // a block's work
  if (WINDOW && !win.has(a.sorted_pos[l + len - 1])) return;
  const u32 W = (u32)a.width, col0 = slice * kSliceFloats, cols = min(kSliceFloats, W - col0);
  constexpr u32 kLanesPerRow = kSliceFloats / V, kRowsPerCopy = V;
  const unsigned sub = lane / kLanesPerRow, col = lane % kLanesPerRow * V;
  const u64 once = l2_evict_first_policy();
  const u32 n_tiles = (len + kWarpStageRows - 1) / kWarpStageRows;
  // positions come 32 at a time, one per lane; `here` serves the tiles being issued, `ahead` the next 32
  u32 here = a.sorted_pos[l + lane];  // (len > 32)
  u32 ahead = 32 + lane < len ? a.sorted_pos[l + 32 + lane] : 0u;
  if (slice == 0 && lane == 0) count_updates(a, row, len);
  float *e = a.embedding + (size_t)row * W + col0 + lane;
  float e_old = 0.f;
  if (lane < cols) e_old = *e;
  u32 issued = 0;
  auto issue = [&]() {
    if (issued < n_tiles) {
      const u32 r0 = issued * kWarpStageRows;
      if (issued != 0 && r0 % 32 == 0) {
        here = ahead;
        ahead = r0 + 32 + lane < len ? a.sorted_pos[l + r0 + 32 + lane] : 0u;
      }
      float *stage = ring + (issued % kWarpStages) * kWarpStageRows * kSliceFloats;
#pragma unroll
      for (u32 i = 0; i < kWarpStageRows / kRowsPerCopy; i++) {
        const u32 r = i * kRowsPerCopy + sub;
        const u32 p = __shfl_sync(0xffffffffu, here, (r0 + r) & 31);
        if (r0 + r < len && col < cols)
          cp_async<V>(stage + r * kSliceFloats + col, a.grad + (size_t)p * W + col0 + col, once);
      }
      issued++;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (u32 t = 0; t < kWarpStages - 1; t++) issue();
  float sum = 0.f;
  for (u32 tile = 0; tile < n_tiles; tile++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kWarpStages - 2) : "memory");
    __syncwarp();  // every lane's copies of this tile have landed, and the tile before it has been added by all
    issue();
    const float *src = ring + (tile % kWarpStages) * kWarpStageRows * kSliceFloats + lane;
    const u32 nr = min(kWarpStageRows, len - tile * kWarpStageRows);
    if (nr == kWarpStageRows) {
      float v[kWarpStageRows];
#pragma unroll
      for (u32 k = 0; k < kWarpStageRows; k++) v[k] = src[k * kSliceFloats];
#pragma unroll
      for (u32 k = 0; k < kWarpStageRows; k++) sum = __fadd_rn(sum, v[k]);
    } else {
      for (u32 k = 0; k < nr; k++) sum = __fadd_rn(sum, src[k * kSliceFloats]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (lane < cols) *e = __fadd_rn(e_old, __fmul_rn(sum, a.neg_lr));
  __syncwarp();
}

// ---- short runs: the keys of one chunk ------------------------------------------------------------
// What a warp must know of a chunk, one key and up to two positions per lane.
static_assert(HCTR_CHUNK_POS - 1 + HCTR_LIGHT_RUN < 64, "the short runs of a chunk end within 64 positions of its start");
struct ChunkMeta {
  u32 m;                   // number of keys
  u32 l, next;             // start of the lane's run and of the one behind it
  int32_t row;
  u32 sp[2];               // sorted_pos[32 chunk + lane + 32 i]
};

__device__ __forceinline__ void load_chunk(const hctr_local_reduce_args &a, u32 chunk, u32 k0, u32 k1, ChunkMeta &c) {
  const unsigned lane = threadIdx.x & 31;
  c.m = k1 - k0;
  c.l = c.next = 0;
  c.row = 0;
  if (c.m == 0) return;
#pragma unroll
  for (u32 i = 0; i < 2; i++) c.sp[i] = a.sorted_pos[min(chunk * HCTR_CHUNK_POS + i * 32 + lane, (u32)a.batch - 1)];
  if (lane < c.m) {
    c.l = a.run_start[k0 + lane];
    c.next = a.run_start[k0 + lane + 1];
    c.row = a.uniq_row[k0 + lane];
  }
}

template <int V, int LANES, bool WINDOW>
__device__ __forceinline__ void sum_chunk(const hctr_local_reduce_args &a, Window win, u32 chunk, u32 slab,
                                          const ChunkMeta &ck, unsigned char *smem, u64 once) {
  typedef RowV<V> R;
  typedef typename R::T T;
  constexpr u32 kGroups = 32 / LANES;
  const unsigned lane = threadIdx.x & 31, gl = lane % LANES, grp = lane / LANES;
  u32 m = ck.m;
  const u32 len = ck.next - ck.l;
  // a chunk's last run may be a long one (any other ends inside the chunk)
  if (__any_sync(0xffffffffu, len > HCTR_LIGHT_RUN)) m--;
  if (m == 0) return;
  u32 wanted = 0xffffffffu;  // bit k: key k of the chunk is summed now
  if (WINDOW) {
    wanted = __ballot_sync(0xffffffffu, lane < m && win.has(a.sorted_pos[lane < m ? ck.next - 1 : 0u]));
    if (wanted == 0) return;
  }
  if (slab == 0 && lane < m && (wanted >> lane & 1)) count_updates(a, ck.row, len);
  uint2 *s_row = reinterpret_cast<uint2 *>(smem + kRingBytes);
  const u32 base = __shfl_sync(0xffffffffu, ck.l, 0), P = __shfl_sync(0xffffffffu, ck.next, m - 1) - base;
  // bit p of `firsts`: a key's run starts at position p (of the P <= 63 positions of the chunk's short runs)
  const u32 at = ck.l - base;
  const u32 lo = __reduce_or_sync(0xffffffffu, lane < m && at < 32 ? 1u << at : 0u);
  const u32 hi = __reduce_or_sync(0xffffffffu, lane < m && at >= 32 ? 1u << (at - 32) : 0u);
  const u64 firsts = (u64)lo | (u64)hi << 32, lasts = firsts >> 1 | 1ull << (P - 1);
  __syncwarp();
#pragma unroll
  for (u32 i = 0; i < 2; i++) {
    const u32 p = chunk * HCTR_CHUNK_POS + i * 32 + lane - base;  // (wraps to a large number in front of the base)
    const u32 key = p < P ? (u32)__popcll(firsts & ((2ull << p) - 1ull)) - 1u : 0u;
    const int32_t row = __shfl_sync(0xffffffffu, ck.row, key);
    // {batch position, table row | last row of its key}; a key that is not wanted now: no position, no last row
    const bool now = !WINDOW || (wanted >> key & 1);
    if (p < P) s_row[p] = now ? make_uint2(ck.sp[i], (u32)row | ((u32)(lasts >> p) << 31)) : make_uint2(kNoPosition, 0);
  }
  __syncwarp();
  // the lane groups take shares of the positions that begin and end with a key
  auto share = [&](u32 g) {
    const u32 from = g * P / kGroups;
    const u64 rest = firsts >> from;
    return rest ? from + (u32)__ffsll(rest) - 1u : P;
  };
  const u32 p_lo = kGroups == 1 ? 0u : share(grp), p_hi = kGroups == 1 || grp == kGroups - 1 ? P : share(grp + 1);
  const u32 row_bytes = (u32)a.width * 4, c = slab * 32 + gl;
  if (c < (u32)a.width / V) {
    const char *grad = reinterpret_cast<const char *>(a.grad) + c * sizeof(T);
    char *emb = reinterpret_cast<char *>(a.embedding) + c * sizeof(T);
    T *mine = reinterpret_cast<T *>(smem) + lane;  // this lane's piece of every row slot
    const u32 rounds = (p_hi - p_lo + kRound - 1) / kRound;
    auto issue = [&](u32 r) {
#pragma unroll
      for (u32 i = 0; i < kRound; i++) {
        const u32 p = p_lo + r * kRound + i;
        if (p < p_hi) {
          const uint2 w = s_row[p];
          if (WINDOW && w.x == kNoPosition) continue;
          T *slot = mine + ((r & 1) * kRound + i) * 64;
          cp_async<V>(slot, grad + (u64)w.x * row_bytes, once);
          if ((int32_t)w.y < 0) cp_async<V>(slot + 32, emb + (u64)(w.y & 0x7fffffffu) * row_bytes);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    issue(1);
    T sum = R::zero();
    for (u32 r = 0; r < rounds; r++) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
      for (u32 i = 0; i < kRound; i++) {
        const u32 p = p_lo + r * kRound + i;
        if (p < p_hi) {
          const T *slot = mine + ((r & 1) * kRound + i) * 64;
          if (WINDOW && s_row[p].x == kNoPosition) continue;
          sum = R::add(sum, slot[0]);
          const u32 row = s_row[p].y;
          if ((int32_t)row < 0) {
            *reinterpret_cast<T *>(emb + (u64)(row & 0x7fffffffu) * row_bytes) = R::add(slot[32], R::scale(sum, a.neg_lr));
            sum = R::zero();
          }
        }
      }
      issue(r + 2);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncwarp();
}

template <int V, int LANES, bool WINDOW>
__global__ void __launch_bounds__(kThreads, kResident) grad_reduce_local(hctr_local_reduce_args a, Window win) {
  extern __shared__ __align__(16) unsigned char reduce_smem[];
  const unsigned warp = threadIdx.x >> 5;
  if (grouping_broke_off(a.meta)) {  // no runs to go by: nothing is updated, and the host hears of it
    if (a.err && blockIdx.x == 0 && threadIdx.x == 0) *a.err = HCTR_ERR_TIMEOUT;
    return;
  }
  sum_very_long<V, WINDOW>(a, win, reinterpret_cast<float *>(reduce_smem));
  __syncthreads();
  unsigned char *smem = reduce_smem + warp * kWarpBytes;
  // Long runs go to the warps of blocks that had no very long one, chunks first to warps with neither, then to those with a
  // long run, then to the rest.
  const u32 n_warps = gridDim.x * kWarps, place = (gridDim.x - 1 - blockIdx.x) * kWarps + warp;
  const u32 slices = ((u32)a.width + kSliceFloats - 1) / kSliceFloats;
  const u32 n_long = a.meta[HCTR_META_NHEAVY] * slices;
  // pieces of short runs: (chunk, 32 elements of the row)
  const u32 slabs = ((u32)a.width / V + 31) / 32;
  const u32 n_chunks = (a.run_start[a.meta[HCTR_META_UNIQUE]] + HCTR_CHUNK_POS - 1) / HCTR_CHUNK_POS, n_pieces = n_chunks * slabs;
  const u64 once = l2_evict_first_policy();
  for (u32 t = place; t < n_long; t += n_warps)
    sum_long<V, WINDOW>(a, win, a.heavy_list[t / slices], t % slices, reinterpret_cast<float *>(smem));
  const u32 n_very = min(a.meta[HCTR_META_NLONG] * slices, gridDim.x) * kWarps;
  const u32 n_free = n_warps - n_very > n_long ? n_warps - n_very - n_long : 0u;
  u32 piece = n_free == 0 || place >= n_warps - n_very ? place : place < n_long ? n_free + place : place - n_long;
  ChunkMeta now, then;
  u32 k0 = 0, k1 = 0;
  auto keys_of = [&](u32 at) {
    if (at < n_pieces) k0 = a.chunk_key[at / slabs], k1 = a.chunk_key[at / slabs + 1];
  };
  keys_of(piece);
  if (piece < n_pieces) load_chunk(a, piece / slabs, k0, k1, now);
  keys_of(piece + n_warps);
  for (; piece < n_pieces; piece += n_warps) {
    const u32 next = piece + n_warps;
    if (next < n_pieces) load_chunk(a, next / slabs, k0, k1, then);
    keys_of(next + n_warps);
    sum_chunk<V, LANES, WINDOW>(a, win, piece / slabs, piece % slabs, now, smem, once);
    now = then;
  }
}

}  // namespace hctr

using namespace hctr;

template <bool WINDOW>
static int launch_local(const hctr_local_reduce_args &a, Window win, cudaStream_t st) {
  if (a.batch == 0) return 0;
  // (32-bit piece and row-byte arithmetic: 2^31 positions, rows of up to 2^28 floats)
  if (a.batch >= ((size_t)1 << 31) || a.width >= ((size_t)1 << 28)) return (int)cudaErrorInvalidValue;
  const uintptr_t addr = (uintptr_t)a.grad | (uintptr_t)a.embedding;
  // one resident round, fewer blocks where the pieces of work are fewer
  const size_t pieces = (a.batch / HCTR_CHUNK_POS + 1) * ((a.width + 127) / 128) + a.batch / (HCTR_LIGHT_RUN + 1);
  const unsigned blocks = (unsigned)std::min((pieces + kWarps - 1) / kWarps, (size_t)kSMs * kResident);
#define CALL(V, L)                                                                                                     \
  do {                                                                                                                 \
    static PerDevice allowed;                                                                                          \
    if (const int e = allow_shared(allowed, grad_reduce_local<V, L, WINDOW>, kBlockBytes)) return e;                   \
    grad_reduce_local<V, L, WINDOW><<<blocks, kThreads, kBlockBytes, st>>>(a, win);                                    \
  } while (0)
  HCTR_DISPATCH_ELEMS(a.width, addr, CALL);
#undef CALL
  count_launches(1);
  return launch_status();
}

extern "C" int hctr_grad_reduce_local(const hctr_local_reduce_args *a, void *stream) {
  return launch_local<false>(*a, Window{}, (cudaStream_t)stream);
}

extern "C" int hctr_grad_reduce_window(const hctr_local_reduce_args *a, uint32_t last_lo, uint32_t last_hi, void *stream) {
  if (last_lo > last_hi) return (int)cudaErrorInvalidValue;
  return launch_local<true>(*a, Window{last_lo, last_hi}, (cudaStream_t)stream);
}
