// Pull side of the peer-to-peer exchange: the owner answers the queries in its mailbox, the requester takes the
// answers in.  Nothing is compacted: the row returned for the j-th query of requester s goes to row
// (owner * cap + j) of s's mailbox, the place s can compute for each of its unique keys without knowing what the
// owner decided.  So neither side needs a prefix sum over flags (the reference compacts on the owner,
// csrc/core/handle_query.cu:24-73, and scans again on the requester, csrc/core/writeback.cu:43-50), and the
// owner's staleness test and row gather are one launch, the requester's flag collection and cache refresh another.
#include "p2p.cuh"
#include "rowops.cuh"

namespace hctr {

constexpr int kPullThreads = 1024;  // fat blocks, at most a few per SM: every block polls or fences at system scope
constexpr long long kInvalidVersion = INT64_MIN;
constexpr int kCopyUnroll = 4;

// dst = src + add (the cache refresh) for `cnt` rows (cnt <= 32; lane i holds the pointers of row i): their elements as ONE
// flat range for the warp, kCopyUnroll independent loads in flight per lane.  All 32 lanes must call it.
template <class R>
__device__ __forceinline__ void warp_refresh_rows(u32 cnt, u32 E, const typename R::T *src_row,
                                                  const typename R::T *add_row, typename R::T *dst_row) {
  typedef typename R::T T;
  const unsigned lane = threadIdx.x & 31;
  const u32 total = cnt * E;
  for (u32 t0 = 0; t0 < total; t0 += 32 * kCopyUnroll) {
    T v[kCopyUnroll], w[kCopyUnroll];
    T *d[kCopyUnroll];
    u32 ee[kCopyUnroll];
#pragma unroll
    for (int k = 0; k < kCopyUnroll; k++) {
      const u32 t = t0 + 32u * k + lane;
      const u32 j = t / E, e = t - j * E;
      ee[k] = e;
      const bool act = t < total;
      // (shuffles are executed by all lanes; slots beyond the range read lane 0's pointers and are not used)
      const T *sp = reinterpret_cast<const T *>(__shfl_sync(0xffffffffu, (unsigned long long)src_row, act ? j : 0));
      const T *ap = reinterpret_cast<const T *>(__shfl_sync(0xffffffffu, (unsigned long long)add_row, act ? j : 0));
      d[k] = reinterpret_cast<T *>(__shfl_sync(0xffffffffu, (unsigned long long)dst_row, act ? j : 0));
      if (act) {
        v[k] = sp[e];
        w[k] = ap[e];
      } else {
        d[k] = nullptr;
      }
    }
#pragma unroll
    for (int k = 0; k < kCopyUnroll; k++)
      if (d[k]) d[k][ee[k]] = R::add(v[k], w[k]);
  }
}

// Lane i of the warp receives the value that the i-th lane with its bit set in `mask` holds.
template <class V>
__device__ __forceinline__ V warp_compact(unsigned mask, V value) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned from = __fns(mask, 0, (int)lane + 1);  // 0xffffffff when there is no such lane
  return __shfl_sync(0xffffffffu, value, from < 32 ? (int)from : 0);
}

// Owner.  For every query received from another rank (flat index q over the sources' sub-regions; counts and starts were
// recorded in c.cnt_in by the kernel that waited for them): stale = (requester's version is INT64_MIN or version +
// pull_bound < owner's version) (csrc/core/handle_query.cu:7-22; a rank's queries to itself are never stale, and nobody reads
// a flag for them).  The flag byte goes to the requester's mailbox; a stale key's row and version follow, to row rank * cap + j
// of that mailbox (write_return_value_kernel, csrc/core/handle_query.cu:24-40).  A warp takes up to 32 queries, one per lane
// for the decision, then moves the rows of the stale ones together; so many that all warps of the grid have some: with 32
// each, 26,500 queries kept 26 SMs busy.  Their addresses go through shared memory, and a power of two of lanes moves a row.
// (Two ranks on one GPU, 53,248 x 128: 21.5 -> 18 us a launch, half of the queries a rank's own before; what is left is four
// dependent accesses and the fences.)  The block that finishes last releases `seq`
// (phase 1) to every peer, all2allReturnOutdated / all2allReturnValue in one, csrc/core/all2all.cu:89-130.
template <bool VEC>
__global__ void __launch_bounds__(kPullThreads) p2p_stale_gather(hctr_p2p_ctx c, u32 seq,
                                                                 const int32_t *__restrict__ row_of, size_t length,
                                                                 size_t n_cached, const float *embedding,
                                                                 const long long *version, long long pull_bound) {
  typedef RowT<VEC> R;
  typedef typename R::T T;
  __shared__ u32 qstart[kMaxRanks + 1];
  __shared__ u32 s_served;
  __shared__ const T *s_src[kPullThreads / 32][32];  // rows to move, per warp
  __shared__ T *s_dst[kPullThreads / 32][32];
  wait_predecessor();
  for (int i = threadIdx.x; i <= c.nrank; i += kPullThreads) qstart[i] = c.cnt_in[3 * c.nrank + i];
  if (threadIdx.x == 0) s_served = 0;
  __syncthreads();
  // (the queries of the others: those of this rank stand between own_at and own_at + own)
  const u32 own_at = qstart[c.rank], own = qstart[c.rank + 1] - own_at, Q = qstart[c.nrank] - own;
  const unsigned lane = threadIdx.x & 31;
  const u32 warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, n_warps = gridDim.x * (kPullThreads / 32);
  const u32 per = min(32u, max(4u, (Q + n_warps - 1) / n_warps));
  const u32 E = (u32)R::elems(c.width);
  // a row is moved by the smallest power of two of lanes that covers it, at most a warp
  const int lane_bits = E > 16 ? 5 : E > 8 ? 4 : E > 4 ? 3 : E > 2 ? 2 : E > 1 ? 1 : 0;
  const u32 lanes = 1u << lane_bits, at_once = 32u >> lane_bits, sub = lane >> lane_bits, col0 = lane & (lanes - 1);
  const T **src_of = s_src[threadIdx.x >> 5];
  T **dst_of = s_dst[threadIdx.x >> 5];
  const hctr_p2p_box me = c.box[c.rank];
  u32 served = 0;
  for (size_t q0 = (size_t)warp * per; q0 < Q; q0 += (size_t)n_warps * per) {
    size_t q = q0 + lane;
    bool stale = false;
    const T *src_row = nullptr;
    T *dst_row = nullptr;
    if (lane < per && q < Q) {
      if (q >= own_at) q += own;
      const unsigned s = segment_of(qstart, c.nrank, (u32)q);
      const u32 j = (u32)q - qstart[s];
      const size_t slot = (size_t)s * c.cap + j;
      const long long key = me.qkey[slot], lv = me.qver[slot];
      int32_t row = -1;
      if (key >= 0 && (size_t)key < length) row = row_of[key];
      const size_t out = (size_t)c.rank * c.cap + j;
      const hctr_p2p_box b = c.box[s];
      if (row < 0 || (size_t)row < n_cached) {
        atomicOr(c.err, HCTR_ERR_NOT_OWNER);
      } else {
        const long long gv = version[row];
        stale = lv == kInvalidVersion || (long long)((u64)lv + (u64)pull_bound) < gv;
        if (stale) {
          b.rver[out] = gv;
          src_row = reinterpret_cast<const T *>(embedding) + (size_t)row * E;
          dst_row = reinterpret_cast<T *>(b.rval) + out * E;
        }
      }
      b.flag[out] = stale ? 1 : 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, stale);
    if (m == 0) continue;
    const u32 cnt = __popc(m);
    served += cnt;
    if (stale) {
      const u32 place = __popc(m & ((1u << lane) - 1u));
      src_of[place] = src_row;
      dst_of[place] = dst_row;
    }
    __syncwarp();
    for (u32 r0 = sub; r0 < cnt; r0 += kCopyUnroll * at_once) {
      for (u32 col = col0; col < E; col += lanes) {
        T v[kCopyUnroll];
#pragma unroll
        for (int k = 0; k < kCopyUnroll; k++)
          if (r0 + k * at_once < cnt) v[k] = src_of[r0 + k * at_once][col];
#pragma unroll
        for (int k = 0; k < kCopyUnroll; k++)
          if (r0 + k * at_once < cnt) dst_of[r0 + k * at_once][col] = v[k];
      }
    }
    __syncwarp();
  }
  if (lane == 0 && served) atomicAdd(&s_served, served);
  __syncthreads();
  if (threadIdx.x == 0 && s_served) atomicAdd(c.cnt_in + HCTR_P2P_SERVED(c.nrank), s_served);
  if (!last_block_of_launch(c.cnt_in + HCTR_P2P_TICKET1(c.nrank))) return;
  for (int p = threadIdx.x; p < c.nrank; p += kPullThreads) {
    u32 *hdr = c.box[p].hdr + (size_t)c.rank * kHdrWords;
    hdr[9] = 0;
    st_release_sys(hdr + 8, seq);
  }
}

// Requester.  Waits (bounded) for every owner's phase-1 release of `seq`, then for each unique key u of the batch:
// recv_index[u] = owner * cap + j, the row of this rank's mailbox the owner of u would have written (j = u's place
// among the keys sent to that owner); flags[u] = what the owner decided; and, for a flagged key that is cached
// here, the cache refresh embedding[row] = returned row + pending[row], version[row] = returned version
// (csrc/core/writeback.cu:8-27).  A warp takes 32 unique keys and moves the rows of those to refresh together.
// The number of flagged keys of the step is added to c.cnt_in[2 * nrank] (statistics).
template <bool VEC>
__global__ void __launch_bounds__(kPullThreads) p2p_refresh_index(hctr_p2p_ctx c, u32 seq,
                                                                  const u32 *__restrict__ meta,
                                                                  const uint8_t *__restrict__ uniq_owner,
                                                                  const int32_t *__restrict__ uniq_row,
                                                                  size_t n_cached, const float *__restrict__ pending,
                                                                  float *__restrict__ embedding,
                                                                  long long *__restrict__ version,
                                                                  uint8_t *__restrict__ flags,
                                                                  u32 *__restrict__ recv_index) {
  typedef RowT<VEC> R;
  typedef typename R::T T;
  __shared__ u32 ret_base[kMaxRanks + 1];
  __shared__ u32 s_flagged;
  if (threadIdx.x == 0) s_flagged = 0;
  wait_returns(c, seq, ret_base, false, blockIdx.x == 0);  // (ends with a block barrier)
  const size_t U = unique_of(meta);
  const u32 *seg = meta + HCTR_META_SEG;
  const unsigned lane = threadIdx.x & 31;
  const size_t warp = ((size_t)blockIdx.x * kPullThreads + threadIdx.x) >> 5;
  const size_t n_warps = ((size_t)gridDim.x * kPullThreads) >> 5;
  const u32 E = (u32)R::elems(c.width);
  const hctr_p2p_box me = c.box[c.rank];
  u32 flagged = 0;
  for (size_t u0 = warp * 32; u0 < U; u0 += n_warps * 32) {
    const size_t u = u0 + lane;
    bool refresh = false, f = false;
    const T *src_row = nullptr, *add_row = nullptr;
    T *dst_row = nullptr;
    if (u < U) {
      const unsigned p = uniq_owner[u];
      const u32 j = (u32)u - seg[p];
      u32 idx = 0;
      if (j < c.cap) {  // (a larger j was reported when the query was sent)
        idx = p * c.cap + j;
        f = p != (unsigned)c.rank && me.flag[idx] != 0;
      }
      flags[u] = f ? 1 : 0;
      recv_index[u] = idx;
      const int32_t row = uniq_row[u];
      refresh = f && row >= 0 && (size_t)row < n_cached;
      if (refresh) {
        version[row] = reinterpret_cast<const long long *>(me.rver)[idx];
        src_row = reinterpret_cast<const T *>(me.rval) + (size_t)idx * E;
        add_row = reinterpret_cast<const T *>(pending) + (size_t)row * E;
        dst_row = reinterpret_cast<T *>(embedding) + (size_t)row * E;
      }
    }
    flagged += __popc(__ballot_sync(0xffffffffu, f));
    const unsigned m = __ballot_sync(0xffffffffu, refresh);
    if (m == 0) continue;
    const T *sp = reinterpret_cast<const T *>(warp_compact(m, (unsigned long long)src_row));
    const T *ap = reinterpret_cast<const T *>(warp_compact(m, (unsigned long long)add_row));
    T *dp = reinterpret_cast<T *>(warp_compact(m, (unsigned long long)dst_row));
    warp_refresh_rows<R>(__popc(m), E, sp, ap, dp);
  }
  if (lane == 0 && flagged) atomicAdd(&s_flagged, flagged);
  __syncthreads();
  if (threadIdx.x == 0 && s_flagged) atomicAdd(c.cnt_in + 2 * c.nrank, s_flagged);
}

// Requester, everything after the owners' answers in ONE launch: the cache refresh of p2p_refresh_index and the row
// expansion (writeBack, csrc/core/writeback.cu:8-71) without the per-key flag / row-index arrays between them.
// Every block waits (bounded) for the owners' phase-1 release, then takes a share of the unique keys (refresh of the
// flagged cached rows, as above) and a share of the batch positions.  A position's row comes from
//   the table            when the key is owned here, or cached and not flagged,
//   the mailbox          when the key is not stored here (row owner * cap + j, j = its place among the keys sent there),
//   mailbox + pending    when the key is cached and flagged - the same sum the refresh stores into the cache row,
//                        computed again here so that no block has to wait for the block that refreshes that row.
// The refresh writes only flagged cached rows, which the expansion never reads: the two parts are independent.
constexpr int kFusedRows = 4;  // rows per lane group and iteration, as in the plain expansion
constexpr int kFusedThreads = 256;  // >= kMaxRanks: thread s of every block polls owner s
// Blocks an SM holds and the grid counts on: one resident round, since every block polls the headers.  From four lanes per row
// on 64 registers do; with one or two the column loop is unrolled into more (80, three blocks).
constexpr int fused_blocks(int lanes) { return lanes >= 4 ? 4 : 3; }

template <int LANES, bool VEC>
__global__ void __launch_bounds__(kFusedThreads, fused_blocks(LANES))
    p2p_refresh_expand(hctr_p2p_ctx c, u32 seq, const u32 *meta, const int32_t *uniq_row, size_t n_cached,
                       const float *pending, float *embedding, long long *version, size_t batch, const int32_t *pos_row,
                       const int32_t *idx_map, float *dst) {
  typedef RowT<VEC> R;
  typedef typename R::T T;
  __shared__ u32 ret_base[kMaxRanks + 1];
  __shared__ u32 seg[kMaxRanks + 1];
  __shared__ u32 s_flagged, s_n;
  __shared__ u32 s_idx[kFusedThreads], s_row[kFusedThreads];
  wait_predecessor();
  if (threadIdx.x == 0) s_flagged = s_n = 0;
  for (int i = threadIdx.x; i <= c.nrank; i += kFusedThreads) seg[i] = meta[HCTR_META_SEG + i];
  // (the expansion's first indices, on their way while the block waits)
  const u32 stride = (u32)((size_t)gridDim.x * kFusedThreads / LANES * kFusedRows), n_pos = (u32)batch;
  const unsigned gl = threadIdx.x % LANES;
  static_assert(kFusedRows == 4, "indices come four at a time");
  const bool fours = aligned16(pos_row) && aligned16(idx_map);  // (a table's own arrays are)
  auto four_at = [&](const int32_t *p, u32 i) {
    if (fours && i + 3 < n_pos) return *reinterpret_cast<const int4 *>(p + i);
    int4 r = make_int4(HCTR_INVALID_ROW, HCTR_INVALID_ROW, HCTR_INVALID_ROW, HCTR_INVALID_ROW);
    if (i < n_pos) r.x = p[i];
    if (i + 1 < n_pos) r.y = p[i + 1];
    if (i + 2 < n_pos) r.z = p[i + 2];
    if (i + 3 < n_pos) r.w = p[i + 3];
    return r;
  };
  u32 i0 = (u32)(((size_t)blockIdx.x * kFusedThreads + threadIdx.x) / LANES) * kFusedRows;
  int4 next_row = four_at(pos_row, i0), next_u = four_at(idx_map, i0);
  wait_returns(c, seq, ret_base, false, blockIdx.x == 0);  // (ends with a block barrier)
  const size_t U = unique_of(meta);
  const unsigned lane = threadIdx.x & 31;
  const u32 E = (u32)R::elems(c.width);
  const hctr_p2p_box me = c.box[c.rank];
  const T *rval = reinterpret_cast<const T *>(me.rval);

  // refresh of the flagged cached rows: the block looks at kFusedThreads unique keys at a time, one per thread, lists
  // the rows to refresh in shared memory and then shares them out evenly among its lane groups (a few rows per
  // block: spread over the whole block they cost one round of loads, left to the warp that found them, several)
  {
    const unsigned n_groups = kFusedThreads / LANES, group = threadIdx.x / LANES, gl = threadIdx.x % LANES;
    u32 flagged = 0;
    for (size_t base = (size_t)blockIdx.x * kFusedThreads; base < U; base += (size_t)gridDim.x * kFusedThreads) {
      const size_t u = base + threadIdx.x;
      bool f = false;
      if (u < U) {
        const unsigned p = segment_of(seg, c.nrank, (u32)u);
        const u32 j = (u32)u - seg[p];
        if (p != (unsigned)c.rank && j < c.cap) {  // (a larger j was reported when the query was sent)
          const u32 idx = p * c.cap + j;
          f = me.flag[idx] != 0;
          const int32_t row = uniq_row[u];
          if (f && row >= 0 && (size_t)row < n_cached) {
            version[row] = reinterpret_cast<const long long *>(me.rver)[idx];
            const u32 e = atomicAdd(&s_n, 1u);
            s_idx[e] = idx;
            s_row[e] = (u32)row;
          }
        }
      }
      flagged += f ? 1u : 0u;
      __syncthreads();
      const u32 n = s_n;
      for (u32 e0 = group * kFusedRows; e0 < n; e0 += n_groups * kFusedRows) {
        for (u32 col = gl; col < E; col += LANES) {
          T v[kFusedRows], w[kFusedRows];
#pragma unroll
          for (int k = 0; k < kFusedRows; k++)
            if (e0 + k < n) {
              v[k] = rval[(size_t)s_idx[e0 + k] * E + col];
              w[k] = reinterpret_cast<const T *>(pending)[(size_t)s_row[e0 + k] * E + col];
            }
#pragma unroll
          for (int k = 0; k < kFusedRows; k++)
            if (e0 + k < n) reinterpret_cast<T *>(embedding)[(size_t)s_row[e0 + k] * E + col] = R::add(v[k], w[k]);
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) s_n = 0;
      // (the next round's first barrier orders this store before the next list is read; its appends come after the
      // barrier below)
      __syncthreads();
    }
    flagged = __reduce_add_sync(0xffffffffu, flagged);
    if (lane == 0 && flagged) atomicAdd(&s_flagged, flagged);
  }

  // Expansion: a group of LANES lanes takes kFusedRows positions per iteration; the next iteration's row and unique indices
  // arrive meanwhile, and a key's owner is the segment its unique index falls into (no access to wait for: two ranks on one
  // GPU, 212,992 x 32 20.5 -> 16.6 us a launch, 53,248 x 128 21.4 -> 20.3).
  for (; i0 < n_pos; i0 += stride) {
    const int32_t row4[kFusedRows] = {next_row.x, next_row.y, next_row.z, next_row.w};
    const int32_t u4[kFusedRows] = {next_u.x, next_u.y, next_u.z, next_u.w};
    next_row = four_at(pos_row, i0 + stride);
    next_u = four_at(idx_map, i0 + stride);
    const T *src[kFusedRows], *add[kFusedRows];
#pragma unroll
    for (int k = 0; k < kFusedRows; k++) {
      src[k] = nullptr;
      add[k] = nullptr;
      if (i0 + k < n_pos) {
        const int32_t row = row4[k];
        if (row >= 0 && (size_t)row >= n_cached) {
          src[k] = reinterpret_cast<const T *>(embedding) + (size_t)row * E;
        } else {
          // < 0: key was out of range, or the grouping broke off (the host reports either); write zeros
          const int32_t u = U > 0 ? u4[k] : -1;
          if (u >= 0) {
            const unsigned p = segment_of(seg, c.nrank, (u32)u);
            const u32 j = (u32)u - seg[p];
            const u32 idx = j < c.cap ? p * c.cap + j : 0u;
            if (row < 0) {
              src[k] = rval + (size_t)idx * E;
            } else if (j < c.cap && me.flag[idx] != 0) {
              src[k] = rval + (size_t)idx * E;
              add[k] = reinterpret_cast<const T *>(pending) + (size_t)row * E;
            } else {
              src[k] = reinterpret_cast<const T *>(embedding) + (size_t)row * E;
            }
          }
        }
      }
    }
    for (size_t col = gl; col < E; col += LANES) {
      T v[kFusedRows];
#pragma unroll
      for (int k = 0; k < kFusedRows; k++) {
        v[k] = src[k] ? src[k][col] : R::zero();
        if (add[k]) v[k] = R::add(v[k], add[k][col]);
      }
#pragma unroll
      for (int k = 0; k < kFusedRows; k++)
        if (i0 + k < n_pos) R::st_once(reinterpret_cast<T *>(dst) + (size_t)(i0 + k) * E + col, v[k]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_flagged) atomicAdd(c.cnt_in + 2 * c.nrank, s_flagged);
}

}  // namespace hctr

using namespace hctr;

extern "C" int hctr_p2p_stale_gather(const hctr_p2p_ctx *c, uint32_t seq, const int32_t *row_of, size_t length,
                                     size_t n_cached, const float *embedding, const int64_t *version,
                                     int64_t pull_bound, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (c->nrank > kMaxRanks) return (int)cudaErrorInvalidValue;
  // a warp per four queries; a publishing kernel runs one block per SM at most
  size_t g = ((size_t)c->nrank * c->cap / 4 + 1 + kPullThreads / 32 - 1) / (kPullThreads / 32);
  if (g > (size_t)kSMs) g = kSMs;
  if (g == 0) g = 1;
  const bool vec = host_aligned16(embedding) && c->width % 4 == 0;
  const auto kernel = vec ? p2p_stale_gather<true> : p2p_stale_gather<false>;
  if (const int e = launch_chained(kernel, (unsigned)g, kPullThreads, 0, st, *c, seq, row_of, length, n_cached, embedding,
                                           (const long long *)version, pull_bound))
    return e;
  count_launches(1);
  return launch_status();
}

extern "C" int hctr_p2p_refresh_index(const hctr_p2p_ctx *c, uint32_t seq, const uint32_t *meta, size_t u_max,
                                      const uint8_t *uniq_owner, const int32_t *uniq_row, size_t n_cached,
                                      const float *pending, float *embedding, int64_t *version, uint8_t *flags,
                                      uint32_t *recv_index, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (c->nrank > kMaxRanks) return (int)cudaErrorInvalidValue;
  size_t g = (u_max / 32 + 1 + kPullThreads / 32 - 1) / (kPullThreads / 32);
  if (g > (size_t)kSMs) g = kSMs;  // every block starts by polling the mailbox headers
  if (g == 0) g = 1;               // (an empty batch still waits for the peers: the step's protocol)
  const bool vec = host_aligned16(embedding) && host_aligned16(pending) && c->width % 4 == 0;
  if (vec)
    p2p_refresh_index<true><<<(unsigned)g, kPullThreads, 0, st>>>(*c, seq, meta, uniq_owner, uniq_row, n_cached,
                                                                  pending, embedding, (long long *)version, flags,
                                                                  recv_index);
  else
    p2p_refresh_index<false><<<(unsigned)g, kPullThreads, 0, st>>>(*c, seq, meta, uniq_owner, uniq_row, n_cached,
                                                                   pending, embedding, (long long *)version, flags,
                                                                   recv_index);
  count_launches(1);
  return launch_status();
}

extern "C" int hctr_p2p_refresh_expand(const hctr_p2p_ctx *c, uint32_t seq, const uint32_t *meta,
                                       const uint8_t * /*uniq_owner: the segments in meta say it*/, const int32_t *uniq_row, size_t n_cached,
                                       const float *pending, float *embedding, int64_t *version, size_t batch,
                                       const int32_t *pos_row, const int32_t *idx_map, float *dst, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  // (positions are 32-bit, up to one round of the grid beyond the last)
  if (c->nrank > kMaxRanks || batch > 0xfff00000u) return (int)cudaErrorInvalidValue;
  const size_t width = c->width;
  // (the mailbox arrays are device allocations of their own: aligned; c->box is a device array)
  const bool al = host_aligned16(embedding) && host_aligned16(pending) && host_aligned16(dst);
#define CALL(L, V)                                                                                         \
  do {                                                                                                     \
    size_t g_ = (((size_t)batch + kFusedRows - 1) / kFusedRows * L + kFusedThreads - 1) / kFusedThreads;              \
    const size_t cap_ = (size_t)kSMs * fused_blocks(L);                                                    \
    if (g_ > cap_) g_ = cap_;                                                                              \
    if (g_ == 0) g_ = 1; /* an empty batch still waits for the peers: the step's protocol */               \
    if (const int e_ = launch_chained(p2p_refresh_expand<L, V>, (unsigned)g_, kFusedThreads, 0, st, *c, seq, meta, \
                                              uniq_row, n_cached, pending, embedding, (long long *)version, batch, pos_row, \
                                              idx_map, dst))                                               \
      return e_;                                                                                      \
  } while (0)
  HCTR_DISPATCH_ROWS(width, al, CALL);
#undef CALL
  count_launches(1);
  return launch_status();
}
