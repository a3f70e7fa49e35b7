// qm_part.cu — partitioned aggregation for group tables larger than a
// block's shared memory (many groups, many selected rows).
//
// The fused scan updates the group table with one atomic per accumulator
// word per selected row; when the table lives in L2 or DRAM those atomics,
// not the column reads, set the pace.  Here the work is split instead:
//   1. counting pass: the scan's filter and compaction, then per survivor
//      its key's partition, counted per (partition, block) in shared memory;
//   2. offsets: each (partition, block)'s first record, partitions back to
//      back (a prefix over blocks per partition, then over partitions);
//   3. scatter pass: the same scan over the same rows (same grid, so every
//      block sees the same rows), each survivor written as a record at its
//      (partition, block)'s next place;
//   4. aggregation: blocks take chunks of the record array (contiguous,
//      coalesced reads) and aggregate each partition's records in a
//      shared-memory table — a window of the direct table or a hash table
//      of the partition's keys — with shared-memory updates, then merge
//      that table into the group table once per chunk.
// Every record of a group lands in one partition; a partition held whole by
// one chunk is written to its slots by plain stores.  First-seen order,
// exact integer sums and compensated float sums follow from the same
// accumulator code as the scan.  The partitions are kept few (at most 512)
// so that the scatter's open write lines, one per (partition, block), stay
// in L2 and reach DRAM as whole lines.
#include "qm_kernels.cuh"
#include "qm_device_once.h"
#include "qm_launch.h"
#include "qm_scan.cuh"

#define QM_PART_WQ (QM_TILE_ROWS + 32)  // per-warp queue: a tile's survivors + < 32 left over

#include <algorithm>
#include <mutex>

namespace qm {

__device__ __forceinline__ int part_of(const qm_scan_args &a, const qm_part_spec &ps, uint64_t key, int special) {
  if (special) return ps.parts;
  if (ps.direct) {
    const uint64_t d = key - (uint64_t)a.key.base;
    return d < (uint64_t)a.n_slots ? (int)(d >> ps.shift) : ps.parts;
  }
  return ps.bits > 0 ? (int)(fmix64(key ^ 0x5851f42d4c957f2dULL) >> (64 - ps.bits)) : 0;
}

// One survivor per lane: its partition counted (pass 0) or its record
// written (pass 1).  Lanes of a warp bound for one partition take
// consecutive places with one shared-memory atomic.
template <int PASS, int NV, int KK>
__device__ __forceinline__ void part_round(const qm_scan_args &a, const qm_part_spec &ps, uint32_t *cnt, int lane,
                                           bool active, int64_t row) {
  int special = 0;
  uint64_t key = 0;
  int p = 0;
  if (active) {
    key = row_key<KK>(a.key, row, special);
    p = part_of(a, ps, key, special);
  }
  const unsigned act = __ballot_sync(QM_FULL, active);
  if (!active) return;
  const unsigned peers = __match_any_sync(act, p);
  const int leader = __ffs(peers) - 1;
  uint32_t at = 0;
  if (lane == leader) at = atomicAdd(&cnt[p], (uint32_t)__popc(peers));
  at = __shfl_sync(peers, at, leader) + __popc(peers & ((1u << lane) - 1));
  if (PASS == 0) return;
  uint64_t vb[QM_MAX_VCOLS];
  uint32_t vnull;
  gather_values<NV>(a.agg, row, vb, vnull);
  const uint64_t pos = ps.bases[p] + ps.offsets[(int64_t)p * ps.blocks + blockIdx.x] + at;
  if (pos >= (uint64_t)ps.rec_cap) {  // more survivors than planned: regrow and run again
    set_error(a.status, QM_DEV_OVERFLOW);
    return;
  }
  // a record is a whole number of 32-byte sectors, written as 16-byte
  // stores: full sectors reach L2, so no partial sector goes back to DRAM
  ulonglong2 *rec = reinterpret_cast<ulonglong2 *>(ps.records + pos * ps.rec_words);
  const int nv = NV > QM_MAX_VCOLS ? a.agg.n_vcols : NV;
  uint64_t w[QM_MAX_VCOLS + 2];
  w[0] = key;
  w[1] = (uint64_t)(uint32_t)row | ((uint64_t)(uint32_t)special << 32) | ((uint64_t)vnull << 40);
#pragma unroll
  for (int c = 0; c < QM_MAX_VCOLS; ++c) w[2 + c] = c < QM_NV_BOUND(NV) && c < nv ? vget<NV>(vb, c) : 0;
#pragma unroll
  for (int k = 0; k < (QM_MAX_VCOLS + 2) / 2; ++k)
    if (2 * k < ps.rec_words) rec[k] = make_ulonglong2(w[2 * k], w[2 * k + 1]);
}

// Passes 0 and 1: the scan's tile walk and filter (every warp takes tiles
// round robin, so a block sees the same rows in both passes).
template <int PASS, int NV, int KK>
__global__ void __launch_bounds__(QM_SCAN_THREADS)
    qm_part_scan(const __grid_constant__ qm_scan_args a, const __grid_constant__ qm_part_spec ps) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  uint32_t *queue = reinterpret_cast<uint32_t *>(smem) + warp * QM_PART_WQ;
  uint32_t *cnt = reinterpret_cast<uint32_t *>(smem) + warps * QM_PART_WQ;  // parts + 1 counters
  __shared__ unsigned long long blk_selected;
  const int P1 = ps.parts + 1;
  for (int p = threadIdx.x; p < P1; p += blockDim.x) cnt[p] = 0;
  if (threadIdx.x == 0) blk_selected = 0;
  __syncthreads();
  const int64_t n_tiles = (a.n + QM_TILE_ROWS - 1) / QM_TILE_ROWS;
  const int64_t gwarps = (int64_t)gridDim.x * warps;
  const int64_t first = (int64_t)blockIdx.x * warps + warp;
  const int64_t n_virtual = a.zones ? a.n_zone_tiles : n_tiles;
  auto tile_of = [&](int64_t v) -> int64_t {
    return a.zones ? ((int64_t)a.zones[v / QM_ZONE_TILES] * QM_ZONE_TILES + v % QM_ZONE_TILES) : v;
  };
  int qn = 0;
  unsigned long long selected = 0;
  const char *pf_base;
  int pf_elem;
  prefetch_column(a.pred, lane, pf_base, pf_elem);
  uint32_t pf_want = ~0u;
  for (int64_t v = first; v < n_virtual; v += gwarps) {
    const int64_t tile = tile_of(v);
    if (tile >= n_tiles) continue;
    const int64_t e0 = tile * QM_TILE_ROWS;
    const int64_t r0 = e0 + (int64_t)lane * QM_R;
    uint32_t m;
    if (a.vec_ok && e0 + QM_TILE_ROWS <= a.n) {
      const int64_t nxt = v + gwarps < n_virtual ? tile_of(v + gwarps) * QM_TILE_ROWS : a.n;
      if (nxt + QM_TILE_ROWS <= a.n) prefetch_tile_l2(pf_base, pf_elem, pf_want, nxt, QM_TILE_ROWS, lane);
      m = eval_pred_contig<1>(a.pred, r0, (1u << QM_R) - 1, pf_want);
    } else {
      int64_t rowv[QM_R];
      m = 0;
#pragma unroll
      for (int j = 0; j < QM_R; ++j) {
        m |= (uint32_t)(r0 + j < a.n) << j;
        rowv[j] = r0 + j;
      }
      auto rowf = [&](int j) { return rowv[j]; };
      m = eval_pred(a.pred, rowf, m);
    }
    const uint32_t c = __popc(m);
    uint32_t off = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(QM_FULL, off, o);
      if (lane >= o) off += x;
    }
    const uint32_t tot = __shfl_sync(QM_FULL, off, 31);
    uint32_t q = qn + off - c;
    for (uint32_t mm = m; mm; mm &= mm - 1) queue[q++] = (uint32_t)r0 + (uint32_t)(__ffs(mm) - 1);
    qn += (int)tot;
    selected += tot;
    __syncwarp();
    while (qn >= 32) {
      const int64_t row = queue[qn - 32 + lane];
      __syncwarp();
      qn -= 32;
      part_round<PASS, NV, KK>(a, ps, cnt, lane, true, row);
    }
  }
  if (qn > 0) {
    const bool active = lane < qn;
    const int64_t row = active ? (int64_t)queue[lane] : 0;
    __syncwarp();
    part_round<PASS, NV, KK>(a, ps, cnt, lane, active, row);
  }
  if (PASS == 0) {
    if (lane == 0 && selected) atomicAdd(&blk_selected, selected);
    __syncthreads();
    if (threadIdx.x == 0 && blk_selected) atomicAdd(&a.status->rows_selected, blk_selected);
    for (int p = threadIdx.x; p < P1; p += blockDim.x) ps.counts[(int64_t)p * ps.blocks + blockIdx.x] = cnt[p];
  }
}

// Pass 2a: one warp per partition: each block's first record relative to
// the partition's start (an exclusive prefix over blocks, 32 at a time), and
// the partition's total into bases[p].
__global__ void qm_part_prefix(const __grid_constant__ qm_part_spec ps) {
  const int lane = threadIdx.x & 31;
  const int P1 = ps.parts + 1;
  const int B = ps.blocks;
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t p = wid; p < P1; p += nw) {
    uint64_t carry = 0;
    for (int b0 = 0; b0 < B; b0 += 32) {
      const int b = b0 + lane;
      const uint64_t c = b < B ? ps.counts[p * B + b] : 0;
      uint64_t x = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(QM_FULL, x, o);
        if (lane >= o) x += y;
      }
      if (b < B) ps.offsets[p * B + b] = carry + x - c;
      carry += __shfl_sync(QM_FULL, x, 31);
    }
    if (lane == 0) ps.bases[p] = carry;
  }
}

// Pass 2b, one block of 1024 threads: the partitions' totals into their
// first records (an exclusive prefix), then the total of all records.
__global__ void qm_part_bases(const __grid_constant__ qm_part_spec ps) {
  __shared__ uint64_t sums[1024];
  const int P1 = ps.parts + 1;
  const int per = (P1 + blockDim.x - 1) / blockDim.x;
  const int b0 = threadIdx.x * per;
  uint64_t t = 0;
  for (int i = 0; i < per; ++i)
    if (b0 + i < P1) t += ps.bases[b0 + i];
  sums[threadIdx.x] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t acc = 0;
    for (int i = 0; i < (int)blockDim.x; ++i) {
      const uint64_t x = sums[i];
      sums[i] = acc;
      acc += x;
    }
    ps.bases[P1] = acc;
  }
  __syncthreads();
  uint64_t acc = sums[threadIdx.x];
  for (int i = 0; i < per; ++i)
    if (b0 + i < P1) {
      const uint64_t x = ps.bases[b0 + i];
      ps.bases[b0 + i] = acc;
      acc += x;
    }
}

// A partition's shared-memory table written into the group table by plain
// stores: the block holding every record of the partition owns its slots.
__device__ __forceinline__ void store_local(const qm_aggspec &A, uint64_t *lw, int L, int s, uint64_t *gp, bool raw,
                                            int64_t row_offset) {
  for (int i = 0; i < A.n_accs; i++) {
    const qm_acc ac = A.acc[i];
    uint64_t v0, v1;
    if (raw) {
      v0 = lw[(int64_t)ac.word * L + s];
      v1 = ac.kind == QA_FSUM || (ac.kind == QA_ISUM && ac.wide) ? lw[(int64_t)(ac.word + 1) * L + s] : 0;
    } else {
      local_load(A, ac, lw, L, s, v0, v1);
    }
    uint64_t *g0 = gp + ac.word;
    if (ac.kind == QA_ISUM) {
      if (ac.wide) {
        g0[0] = v0;
        g0[1] = v1;
      } else if (ac.narrow) {
        g0[0] = v0;
      } else {  // a 64-bit block-local sum into the 128-bit table word pair
        g0[0] = v0;
        g0[1] = (int64_t)v0 < 0 ? ~0ULL : 0ULL;
      }
    } else if (ac.kind == QA_FSUM) {
      const qm_vcol &vc = A.vcol[ac.vcol];
      if (!raw && !(vc.flags & VF_FIXED) && vc.lim != 0.0) {
        // added, not stored: rare parts of the sum went to these words already
        double h, l;
        split_words(vc, (int64_t)v0, (int64_t)v1, h, l);
        if (h != 0.0) atomicAdd(reinterpret_cast<double *>(g0), h);
        if (l != 0.0) atomicAdd(reinterpret_cast<double *>(g0 + 1), l);
      } else {
        g0[0] = v0;
        g0[1] = v1;
      }
    } else if (ac.kind == QA_FIRST && !raw) {
      g0[0] = (uint64_t)row_offset + v0;
    } else {
      g0[0] = v0;
    }
  }
}

// Pass 4: blocks claim chunks of `chunk` records of the record array (a
// large partition is shared by several blocks, a small one shares a chunk
// with its neighbours) and walk a chunk partition by partition: each
// partition's records go through a shared-memory table — the partition's
// window of a direct table, or a hash table of its keys (keys it does not
// admit go to the group table directly) — which is then merged into the
// group table: by plain stores when the chunk holds the whole partition of a
// direct table, else with atomics.  The last partition (special keys, direct
// keys outside the table) goes to the group table directly, where the scan's
// range check reports them.
template <int DD, int NV>
__global__ void __launch_bounds__(QM_SCAN_THREADS)
    qm_part_agg(const __grid_constant__ qm_scan_args a, const __grid_constant__ qm_part_spec ps, int64_t chunk) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ qm_scan_args P;
  __shared__ int s_chunk;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  const qm_aggspec &A = a.agg;
  const int Lmax = ps.local_slots;
  const int hashed = ps.direct ? 0 : 1;
  uint64_t *lkeys = reinterpret_cast<uint64_t *>(smem);
  uint64_t *lw = lkeys + (hashed ? Lmax : 0);
  const int nv = NV > QM_MAX_VCOLS ? A.n_vcols : NV;
  const int P1 = ps.parts + 1;
  const uint64_t total = ps.bases[P1];
  for (;;) {
    if (threadIdx.x == 0) s_chunk = atomicAdd(ps.counter, 1);
    __syncthreads();
    const uint64_t c0 = (uint64_t)s_chunk * (uint64_t)chunk;
    if (c0 >= total) break;
    const uint64_t c1 = min(total, c0 + (uint64_t)chunk);
    // the partition holding record c0: the last p with bases[p] <= c0
    int lo = 0, hi = P1 - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (ps.bases[mid] <= c0) lo = mid;
      else hi = mid - 1;
    }
    for (int p = lo; p < P1; ++p) {
      const uint64_t pb = ps.bases[p], pe = ps.bases[p + 1];
      const uint64_t r0 = max(pb, c0), r1 = min(pe, c1);
      if (r0 >= c1) break;
      if (r0 >= r1) continue;
      const bool whole = pb >= c0 && pe <= c1;
      // this partition's plan: a window of the direct table, or the hash
      // table with a shared-memory front
      {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(&a);
        uint32_t *dst = reinterpret_cast<uint32_t *>(&P);
        for (int i = threadIdx.x; i < (int)(sizeof(qm_scan_args) / 4); i += blockDim.x) dst[i] = src[i];
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        P.priv = 0;
        P.local_rep = 0;
        if (p == ps.parts) {
          P.local_slots = 0;
        } else if (ps.direct) {
          const int64_t base = (int64_t)p << ps.shift;
          P.key.base = a.key.base + base;
          P.n_slots = min((int64_t)Lmax, a.n_slots - base);
          P.table = a.table + base * a.stride;
          P.local_slots = (int)P.n_slots;
          P.local_hash = 0;
        } else {
          P.local_slots = Lmax;
          P.local_hash = 1;
        }
      }
      __syncthreads();
      const int L = P.local_slots;
      if (L > 0) {
        if (hashed)
          for (int s2 = threadIdx.x; s2 < L; s2 += blockDim.x) lkeys[s2] = QM_EMPTY_KEY;
        for (int i = threadIdx.x; i < L * A.n_words; i += blockDim.x) lw[i] = A.init[i / L];
      }
      __syncthreads();
      for (uint64_t base = r0 + (uint64_t)warp * 32; base < r1; base += (uint64_t)warps * 32) {
        const uint64_t i = base + lane;
        const bool active = i < r1;
        uint64_t w[QM_MAX_VCOLS + 2];
        if (active) {
          const ulonglong2 *rec = reinterpret_cast<const ulonglong2 *>(ps.records + i * ps.rec_words);
#pragma unroll
          for (int k = 0; k < (QM_MAX_VCOLS + 2) / 2; ++k) {
            if (2 * k < 2 + QM_NV_BOUND(NV) && 2 * k < ps.rec_words) {
              const ulonglong2 v = __ldcs(rec + k);
              w[2 * k] = v.x;
              w[2 * k + 1] = v.y;
            } else {
              w[2 * k] = w[2 * k + 1] = 0;
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < QM_MAX_VCOLS + 2; ++k) w[k] = 0;
        }
        uint64_t vb[QM_MAX_VCOLS];
#pragma unroll
        for (int c = 0; c < QM_MAX_VCOLS; ++c) vb[c] = c < QM_NV_BOUND(NV) && c < nv ? w[2 + c] : 0;
        const int special = (int)((w[1] >> 32) & 0xff);
        const uint32_t vnull = (uint32_t)((w[1] >> 40) & 0xff);
        drain_apply<DD, NV, (NV > QM_MAX_VCOLS ? QM_FT_FULL : QM_FT_DBL)>(P, lkeys, lw, L, lane, active, w[0], special, (uint32_t)w[1],
                                                vb, vnull);
      }
      __syncthreads();
      if (L > 0) {
        const bool raw = P.dedupe != 0;
        for (int s2 = threadIdx.x; s2 < L; s2 += blockDim.x) {
          if (raw ? lw[(int64_t)A.w_count * L + s2] == 0 : *limb(lw, L, A.w_count, s2) == 0) continue;
          if (!hashed && whole) {
            store_local(A, lw, L, s2, P.table + (int64_t)s2 * P.stride + 1, raw, P.row_offset);
            continue;
          }
          const int64_t gs = hashed ? global_slot(P, lkeys[s2], 0) : s2;
          if (gs < 0) continue;
          if (raw) merge_raw(A, lw + s2, L, P.table + gs * P.stride + 1);
          else merge_local(A, lw, L, s2, P.table + gs * P.stride + 1, P.row_offset);
        }
      }
      __syncthreads();
    }
  }
}

// ---- windows of a large direct table (qm_win_spec) --------------------------------
// The fused scan updates such a table with four or more reductions a row,
// bound by the L2's rate for them (85 G/s).  Here a row costs one record
// written and read (8 bytes and 8 a value column), and its updates are
// shared-memory atomics.  200M rows, 16.7M slots (4,096 windows), key and one
// value column: count 0.42 ms, scatter 2.3, aggregation 1.05, against 9.2 ms
// of key-range passes of the scan.

// The slots of the warp tile of 256 rows at e0: rows e0 + 32 * j + lane that
// pass (slot[j], or QM_NO_SLOT).  Returns the rows that passed (all lanes').
#define QM_NO_SLOT 0xffffffffu
template <int KK>
__device__ __forceinline__ int win_slots(const qm_scan_args &a, int64_t e0, int lane, uint32_t (&slot)[QM_R]) {
  uint32_t m;
  const int64_t r0 = e0 + (int64_t)lane * QM_R;
  if (a.vec_ok && e0 + QM_TILE_ROWS <= a.n) {
    uint32_t want;
    m = eval_pred_contig<1>(a.pred, r0, (1u << QM_R) - 1, want);
  } else {
    int64_t rowv[QM_R];
    m = 0;
#pragma unroll
    for (int j = 0; j < QM_R; ++j) {
      m |= (uint32_t)(r0 + j < a.n) << j;
      rowv[j] = r0 + j;
    }
    auto rowf = [&](int j) { return rowv[j]; };
    m = eval_pred(a.pred, rowf, m);
  }
  // lane l's eight rows follow one another; its keys are read 32 rows apart
  uint64_t key[QM_R];
  int special[QM_R];
  uint32_t pass = 0;
#pragma unroll
  for (int j = 0; j < QM_R; ++j) {
    const uint32_t b = __shfl_sync(QM_FULL, m, j * 4 + (lane >> 3));
    pass |= ((b >> (lane & 7)) & 1) << j;
    key[j] = 0;
    special[j] = 0;
    if ((pass >> j) & 1) key[j] = row_key<KK>(a.key, e0 + j * 32 + lane, special[j]);
  }
#pragma unroll
  for (int j = 0; j < QM_R; ++j) {
    // (global_slot of a direct table: its hash branch and a special for keys that
    // have none spilled the scatter's registers, 3.0 -> 2.3 ms)
    const uint64_t d = key[j] - (uint64_t)a.key.base;
    slot[j] = QM_NO_SLOT;
    if ((pass >> j) & 1) {
      if (KK == QM_KK_ANY && special[j] == 2) slot[j] = (uint32_t)a.n_slots;
      else if (d < (uint64_t)a.n_slots) slot[j] = (uint32_t)d;
      else set_error(a.status, QM_DEV_RANGE);
    }
  }
  return (int)__reduce_add_sync(QM_FULL, (unsigned)__popc(m));
}

// Pulls `rows` cells of a column from row r0 on into L2 (one thread).
__device__ __forceinline__ void win_prefetch(const void *data, int dtype, int64_t r0, int rows) {
  const int elem = dtype == QM_I32 || dtype == QM_F32 ? 4 : 8;
  if (((uintptr_t)data & 15) == 0)  // (and r0 is a multiple of 256)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const char *)data + r0 * elem), "r"(rows * elem) : "memory");
}

// Records of each window: a block's counts in shared memory, then its totals.
template <int KK>
__global__ void __launch_bounds__(QM_SCAN_THREADS)
    qm_win_count(const __grid_constant__ qm_scan_args a, const __grid_constant__ qm_win_spec ws) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t *cnt = reinterpret_cast<uint32_t *>(smem);
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  for (int p = threadIdx.x; p < ws.windows; p += blockDim.x) cnt[p] = 0;
  __syncthreads();
  const int64_t n_tiles = (a.n + QM_TILE_ROWS - 1) / QM_TILE_ROWS;
  const int64_t n_virtual = a.zones ? a.n_zone_tiles : n_tiles;
  unsigned long long selected = 0;
  for (int64_t v = (int64_t)blockIdx.x * warps + (threadIdx.x >> 5); v < n_virtual; v += (int64_t)gridDim.x * warps) {
    const int64_t tile = a.zones ? (int64_t)a.zones[v / QM_ZONE_TILES] * QM_ZONE_TILES + v % QM_ZONE_TILES : v;
    if (tile >= n_tiles) continue;
    uint32_t slot[QM_R];
    const int64_t nxt = (v + (int64_t)gridDim.x * warps) * QM_TILE_ROWS;
    if (!a.zones && nxt + QM_TILE_ROWS <= a.n && lane < a.key.n_cols)
      win_prefetch(a.key.data[lane], a.key.dtype[lane], nxt, QM_TILE_ROWS);
    selected += win_slots<KK>(a, tile * QM_TILE_ROWS, lane, slot);
#pragma unroll
    for (int j = 0; j < QM_R; ++j)
      if (slot[j] != QM_NO_SLOT) atomicAdd(&cnt[slot[j] >> ws.shift], 1u);
  }
  if (lane == 0 && selected) atomicAdd(&a.status->rows_selected, selected);
  __syncthreads();
  for (int p = threadIdx.x; p < ws.windows; p += blockDim.x)
    if (cnt[p]) atomicAdd(&ws.counts[p], cnt[p]);
}

// Exclusive prefix of one value a thread over a block of T threads.
template <int T>
__device__ __forceinline__ uint32_t win_block_scan(uint32_t v, uint32_t *warp_sums, uint32_t &total) {
  const int lane = threadIdx.x & 31;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(QM_FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t w = lane < T / 32 ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(QM_FULL, w, o);
      if (lane >= o) w += y;
    }
    if (lane < T / 32) warp_sums[lane] = w;
  }
  __syncthreads();
  total = warp_sums[T / 32 - 1];
  return x - v + (threadIdx.x >= 32 ? warp_sums[(threadIdx.x >> 5) - 1] : 0);
}

// One block: first records and first chunks of the windows.
__global__ void __launch_bounds__(QM_WIN_THREADS) qm_win_offsets(const __grid_constant__ qm_win_spec ws) {
  __shared__ uint32_t sums[32];
  const int per = (ws.windows + QM_WIN_THREADS - 1) / QM_WIN_THREADS;
  const int p0 = min(ws.windows, (int)threadIdx.x * per), p1 = min(ws.windows, p0 + per);
  uint32_t n = 0, k = 0;
  for (int p = p0; p < p1; ++p) {
    n += ws.counts[p];
    k += (uint32_t)((ws.counts[p] + ws.chunk - 1) / ws.chunk);
  }
  uint32_t n_all, k_all;
  uint32_t b = win_block_scan<QM_WIN_THREADS>(n, sums, n_all);
  __syncthreads();
  uint32_t i = win_block_scan<QM_WIN_THREADS>(k, sums, k_all);
  for (int p = p0; p < p1; ++p) {
    ws.bases[p] = ws.cursor[p] = b;
    ws.items[p] = i;
    b += ws.counts[p];
    i += (uint32_t)((ws.counts[p] + ws.chunk - 1) / ws.chunk);
  }
  if (threadIdx.x == 0) {
    ws.bases[ws.windows] = n_all;
    ws.items[ws.windows] = k_all;
  }
}

// A block's 8,192 rows ordered by window in shared memory, then written to
// the windows' lists in runs (places claimed with one global atomic a window
// and tile): with 4,096 windows a list's open sector is soon filled by
// another block, in L2.  Bound by the L2's write requests (36 G/s: records
// written in row order, without the ordering, 5.6 ms) and, with the runs eight
// long (1,024 windows, 1.8 ms), by the latency of a tile's phases.  While this
// took 3.0 ms, tiles of 12,288 rows on 768 threads took 3.7 and 4,096 rows on
// two blocks of 512 3.5.
template <int NV, int KK>
__global__ void __launch_bounds__(QM_WIN_THREADS, 1)
    qm_win_scatter(const __grid_constant__ qm_scan_args a, const __grid_constant__ qm_win_spec ws) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t sums[32];
  uint64_t *stage = reinterpret_cast<uint64_t *>(smem);  // [1 + NV][QM_WIN_ROWS]
  uint32_t *cnt = reinterpret_cast<uint32_t *>(stage + (1 + NV) * QM_WIN_ROWS);  // counts, then first places here
  uint32_t *delta = cnt + ws.windows;                                            // place in the list less place here
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t n_tiles = (a.n + QM_WIN_ROWS - 1) / QM_WIN_ROWS;
  constexpr int CLAIMS = 4;
  constexpr int ZT = QM_ZONE_ROWS / QM_WIN_ROWS;  // block tiles of a zone
  const int64_t n_virtual = a.zones ? a.n_zone_tiles / QM_ZONE_TILES * ZT : n_tiles;
  const int per = (ws.windows + QM_WIN_THREADS - 1) / QM_WIN_THREADS;
  const int p0 = min(ws.windows, (int)threadIdx.x * per), p1 = min(ws.windows, p0 + per);
  for (int p = threadIdx.x; p < ws.windows; p += blockDim.x) cnt[p] = 0;
  __syncthreads();
  for (int64_t v = blockIdx.x; v < n_virtual; v += gridDim.x) {
    const int64_t tile = a.zones ? (int64_t)a.zones[v / ZT] * ZT + v % ZT : v;
    if (tile >= n_tiles) continue;  // (the whole block)
    const int64_t e0 = tile * QM_WIN_ROWS + warp * QM_TILE_ROWS;
    uint32_t slot[QM_R], rank[QM_R];
    win_slots<KK>(a, e0, lane, slot);
#pragma unroll
    for (int j = 0; j < QM_R; ++j)
      if (slot[j] != QM_NO_SLOT) rank[j] = atomicAdd(&cnt[slot[j] >> ws.shift], 1u);
    __syncthreads();
    // the columns would stand idle until this tile is written out
    const int64_t nxt = (v + gridDim.x) * QM_WIN_ROWS;
    if (!a.zones && nxt + QM_WIN_ROWS <= a.n) {
      if ((int)threadIdx.x < a.key.n_cols) win_prefetch(a.key.data[threadIdx.x], a.key.dtype[threadIdx.x], nxt, QM_WIN_ROWS);
      else if (threadIdx.x >= 32 && threadIdx.x < 32 + NV)
        win_prefetch(a.agg.vcol[threadIdx.x - 32].data, a.agg.vcol[threadIdx.x - 32].dtype, nxt, QM_WIN_ROWS);
    }
    uint32_t n = 0, total;
    for (int p = p0; p < p1; ++p) n += cnt[p];
    uint32_t at = win_block_scan<QM_WIN_THREADS>(n, sums, total);
    for (int p = p0; p < p1; ++p) {
      const uint32_t c = cnt[p];
      delta[p] = c;
      cnt[p] = at;
      at += c;
    }
    __syncthreads();
    // the lists' places: neighbouring windows by neighbouring lanes, in
    // flight while the rows are ordered
    uint32_t place[CLAIMS];
#pragma unroll
    for (int k = 0; k < CLAIMS; ++k) {
      const int p = (int)threadIdx.x + k * QM_WIN_THREADS;
      const uint32_t c = p < ws.windows ? delta[p] : 0;
      if (c) place[k] = atomicAdd(&ws.cursor[p], c);
    }
    for (int p = (int)threadIdx.x + CLAIMS * QM_WIN_THREADS; p < ws.windows; p += QM_WIN_THREADS) {
      const uint32_t c = delta[p];
      if (c) delta[p] = atomicAdd(&ws.cursor[p], c) - cnt[p];
    }
    // four rows' cells in flight (all eight take more registers than there are)
#pragma unroll
    for (int j0 = 0; j0 < QM_R; j0 += 4) {
      uint64_t vb[4][QM_MAX_VCOLS];
      uint32_t vn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (slot[j0 + j] != QM_NO_SLOT) gather_values<NV>(a.agg, e0 + (j0 + j) * 32 + lane, vb[j], vn[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t s = slot[j0 + j];
        if (s == QM_NO_SLOT) continue;
        const uint32_t i = cnt[s >> ws.shift] + rank[j0 + j];
        stage[i] = (uint64_t)(uint32_t)(e0 + (j0 + j) * 32 + lane) | (uint64_t)s << 32 |
                   (NV > 0 ? (uint64_t)vn[j] << (32 + QM_WIN_SLOT_BITS) : 0);
#pragma unroll
        for (int c = 0; c < NV; ++c) stage[(c + 1) * QM_WIN_ROWS + i] = vb[j][c];
      }
    }
#pragma unroll
    for (int k = 0; k < CLAIMS; ++k) {
      const int p = (int)threadIdx.x + k * QM_WIN_THREADS;
      if (p < ws.windows) delta[p] = place[k] - cnt[p];  // (not read where the tile has none)
    }
    __syncthreads();
    for (int p = threadIdx.x; p < ws.windows; p += blockDim.x) cnt[p] = 0;
    for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
      const uint64_t w0 = stage[i];
      const uint32_t p = ((uint32_t)(w0 >> 32) & ((1u << QM_WIN_SLOT_BITS) - 1)) >> ws.shift;
      const uint32_t to = delta[p] + i;
      if ((int64_t)to >= ws.rec_cap) {  // the columns changed since they were counted
        set_error(a.status, QM_DEV_OVERFLOW);
        continue;
      }
      uint64_t *rec = ws.records + (int64_t)to * (1 + NV);
      if constexpr (NV == 1) {
        *reinterpret_cast<ulonglong2 *>(rec) = make_ulonglong2(w0, stage[QM_WIN_ROWS + i]);
      } else {
        rec[0] = w0;
#pragma unroll
        for (int c = 0; c < NV; ++c) rec[c + 1] = stage[(c + 1) * QM_WIN_ROWS + i];
      }
    }
    __syncthreads();
  }
}

// Blocks claim chunks of the windows' lists and aggregate each in a
// shared-memory window of the table, four records a thread in flight; a
// window of one chunk is stored, a larger one's chunks are merged.
template <int NV, int FT>
__global__ void __launch_bounds__(QM_WIN_THREADS, 1)
    qm_win_agg(const __grid_constant__ qm_scan_args a, const __grid_constant__ qm_win_spec ws) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_item, s_window;
  const qm_aggspec &A = a.agg;
  const int lane = threadIdx.x & 31;
  const int L = 1 << ws.shift;
  uint64_t *lw = reinterpret_cast<uint64_t *>(smem);
  const int n_items = (int)ws.items[ws.windows];
  for (;;) {
    if (threadIdx.x == 0) {
      const int it = atomicAdd(ws.counter, 1);
      int lo = 0, hi = ws.windows - 1;  // the last window with items[p] <= it
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((int)ws.items[mid] <= it) lo = mid;
        else hi = mid - 1;
      }
      s_item = it;
      s_window = lo;
    }
    for (int i = threadIdx.x; i < L * A.n_words; i += blockDim.x) lw[i] = A.init[i >> ws.shift];
    __syncthreads();
    const int it = s_item, p = s_window;
    if (it >= n_items) break;
    const int k = it - (int)ws.items[p];
    const int64_t r0 = (int64_t)ws.bases[p] + k * ws.chunk;
    const int64_t r1 = min(min((int64_t)ws.bases[p + 1], r0 + ws.chunk), ws.rec_cap);
    for (int64_t b0 = r0 + (threadIdx.x & ~31u); b0 < r1; b0 += 4 * QM_WIN_THREADS) {  // (whole warps)
      const int64_t b = b0 + lane;
      uint64_t w[4][1 + NV];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const int64_t i = b + d * QM_WIN_THREADS;
        if (i >= r1) continue;
        const uint64_t *rec = ws.records + i * (1 + NV);
        if constexpr (NV == 1) {
          const ulonglong2 x = __ldcs(reinterpret_cast<const ulonglong2 *>(rec));
          w[d][0] = x.x;
          w[d][1] = x.y;
        } else {
#pragma unroll
          for (int c = 0; c <= NV; ++c) w[d][c] = __ldcs(reinterpret_cast<const unsigned long long *>(rec) + c);
        }
      }
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const bool act = b + d * QM_WIN_THREADS < r1;
        if (FT > QM_FT_DBL && !act) break;
        const uint32_t slot = (uint32_t)(w[d][0] >> 32) & ((1u << QM_WIN_SLOT_BITS) - 1);
        const uint32_t vnull = (uint32_t)(w[d][0] >> (32 + QM_WIN_SLOT_BITS));
        uint64_t vb[QM_MAX_VCOLS];
#pragma unroll
        for (int c = 0; c < QM_MAX_VCOLS; ++c) vb[c] = c < NV ? w[d][c < NV ? c + 1 : 0] : 0;
        if (act)
          agg_row_local<NV, FT>(a, lw, L, (int)(slot & (L - 1)), (uint64_t)a.key.base + slot, slot >= a.n_slots ? 2 : 0,
                                (uint32_t)w[d][0], vb, vnull);
        if (FT <= QM_FT_DBL) {
          __syncwarp();
          local_doubles<NV>(a, lw, L, act ? (int)(slot & (L - 1)) : -1, lane, vb, vnull);
          __syncwarp();
        }
      }
    }
    __syncthreads();
    const bool whole = ws.items[p + 1] - ws.items[p] == 1;
    const int64_t s0 = (int64_t)p << ws.shift;
    const int slots = (int)min((int64_t)L, ws.total_slots - s0);
    for (int s = threadIdx.x; s < slots; s += blockDim.x) {
      if (*limb(lw, L, A.w_count, s) == 0) continue;
      uint64_t *gp = a.table + (s0 + s) * a.stride + 1;
      if (whole) store_local(A, lw, L, s, gp, false, a.row_offset);
      else merge_local(A, lw, L, s, gp, a.row_offset);
    }
    __syncthreads();
  }
}

}  // namespace qm

using namespace qm;

size_t qm_part_scan_smem(int parts) {
  return (size_t)(QM_SCAN_THREADS / 32) * QM_PART_WQ * sizeof(uint32_t) + (size_t)(parts + 1) * sizeof(uint32_t);
}

size_t qm_part_agg_smem(int local_slots, int local_hash, int n_words) {
  return (size_t)local_slots * 8 * ((local_hash ? 1 : 0) + n_words);
}

namespace {

// Kernel attributes and occupancy are set up once per instantiation (the
// largest shared memory any launch may ask for), not per launch.
constexpr size_t PART_SCAN_SMEM_MAX = (size_t)(QM_SCAN_THREADS / 32) * QM_PART_WQ * 4 + (size_t)(8192 + 1) * 4;
constexpr size_t PART_AGG_SMEM_MAX = 200 * 1024;

template <auto Kernel>
cudaError_t set_smem_once(size_t bytes, int *per_sm_out = nullptr) {
  static qm_device_once once;  // one per kernel (the kernel is a template argument)
  const auto kernel = Kernel;
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  const qm_kernel_setup s = once.get(device, [&] {
    int per_sm = 1;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, QM_SCAN_THREADS, bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return qm_kernel_setup{(int)e, per_sm};
  });
  if (per_sm_out) *per_sm_out = s.per_sm;
  return (cudaError_t)s.error;
}

template <int PASS, int NV, int KK>
cudaError_t part_scan_one(const qm_scan_args &a, const qm_part_spec &ps, cudaStream_t st) {
  const size_t smem = qm_part_scan_smem(ps.parts);
  cudaError_t e = set_smem_once<qm_part_scan<PASS, NV, KK>>(PART_SCAN_SMEM_MAX);
  if (e != cudaSuccess) return e;
  qm_part_scan<PASS, NV, KK><<<ps.blocks, QM_SCAN_THREADS, smem, st>>>(a, ps);
  return cudaGetLastError();
}

template <int PASS, int NV>
cudaError_t part_scan_kk(const qm_scan_args &a, const qm_part_spec &ps, int kk, cudaStream_t st) {
  if (kk == QM_KK_I64) return part_scan_one<PASS, NV, QM_KK_I64>(a, ps, st);
  if (kk == QM_KK_I32) return part_scan_one<PASS, NV, QM_KK_I32>(a, ps, st);
  return part_scan_one<PASS, NV, QM_KK_ANY>(a, ps, st);
}

template <int PASS>
cudaError_t part_scan_nv(const qm_scan_args &a, const qm_part_spec &ps, int kk, cudaStream_t st) {
  switch (a.agg.n_vcols) {
    case 1: return part_scan_kk<PASS, 1>(a, ps, kk, st);
    case 2: return part_scan_kk<PASS, 2>(a, ps, kk, st);
    default: return part_scan_kk<PASS, QM_NV_ANY>(a, ps, kk, st);
  }
}

int part_key_kind(const qm_keyspec &K) {
  if (K.n_cols == 1 && K.pack == QP_RAW && K.nulls[0] == nullptr) {
    if (K.dtype[0] == QM_I64) return QM_KK_I64;
    if (K.dtype[0] == QM_I32) return QM_KK_I32;
  }
  return QM_KK_ANY;
}

template <int DD, int NV>
cudaError_t part_agg_one(const qm_scan_args &a, const qm_part_spec &ps, int sm_count, cudaStream_t st) {
  const size_t smem = qm_part_agg_smem(ps.local_slots, ps.direct ? 0 : 1, a.agg.n_words);
  cudaError_t e = set_smem_once<qm_part_agg<DD, NV>>(PART_AGG_SMEM_MAX);
  if (e != cudaSuccess) return e;
  // two blocks of 16 warps per SM when their tables fit (register bound)
  const int per_sm = smem <= 100 * 1024 ? 2 : 1;
  const int blocks = sm_count * per_sm;
  // chunks: about 8 per block over the planned records, at least a few
  // table sizes each (the merge of a partition's table is paid per chunk)
  int64_t chunk = std::max<int64_t>(ps.rec_cap / ((int64_t)blocks * 8), (int64_t)ps.local_slots * 16);
  chunk = std::max<int64_t>(chunk, 8192);
  qm_part_agg<DD, NV><<<blocks, QM_SCAN_THREADS, smem, st>>>(a, ps, chunk);
  return cudaGetLastError();
}

}  // namespace

int qm_part_scan_blocks(int sm_count, int parts) {
  (void)parts;
  int per_sm = 1;
  if (set_smem_once<qm_part_scan<0, QM_NV_ANY, QM_KK_ANY>>(PART_SCAN_SMEM_MAX, &per_sm) != cudaSuccess) {
    cudaGetLastError();
    per_sm = 1;
  }
  return sm_count * std::min(std::max(per_sm, 1), 2);
}

cudaError_t qm_launch_part_scan(int pass, const qm_scan_args &a, const qm_part_spec &ps, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const int kk = part_key_kind(a.key);
  return pass == 0 ? part_scan_nv<0>(a, ps, kk, st) : part_scan_nv<1>(a, ps, kk, st);
}

cudaError_t qm_launch_part_offsets(const qm_part_spec &ps, cudaStream_t st) {
  const int P1 = ps.parts + 1;
  const int blocks = (int)std::min<int64_t>(((int64_t)P1 * 32 + 255) / 256, 1024);
  qm_part_prefix<<<blocks, 256, 0, st>>>(ps);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  qm_part_bases<<<1, 1024, 0, st>>>(ps);
  return cudaGetLastError();
}

cudaError_t qm_launch_part_agg(const qm_scan_args &a, const qm_part_spec &ps, int sm_count, cudaStream_t st) {
  const bool fixed = [&] {
    for (int c = 0; c < a.agg.n_vcols; ++c)
      if (a.agg.vcol[c].flags & VF_FIXED) return true;
    return false;
  }();
  const int dd = a.dedupe != 0 ? 1 : 0;
  if (!fixed && a.agg.n_vcols == 1)
    return dd ? part_agg_one<1, 1>(a, ps, sm_count, st) : part_agg_one<0, 1>(a, ps, sm_count, st);
  if (!fixed && a.agg.n_vcols == 2)
    return dd ? part_agg_one<1, 2>(a, ps, sm_count, st) : part_agg_one<0, 2>(a, ps, sm_count, st);
  return dd ? part_agg_one<1, QM_NV_ANY>(a, ps, sm_count, st) : part_agg_one<0, QM_NV_ANY>(a, ps, sm_count, st);
}

// ---- windows of a large direct table ----------------------------------------------

namespace {
// (ws null: only the kernels' shared memory limits are set)
template <int KK>
cudaError_t win_count(const qm_scan_args &a, const qm_win_spec *ws, int sm_count, cudaStream_t st) {
  cudaError_t e = set_smem_once<qm_win_count<KK>>((size_t)QM_WIN_MAX * 4);
  if (e != cudaSuccess || !ws) return e;
  qm_win_count<KK><<<sm_count * 2, QM_SCAN_THREADS, (size_t)ws->windows * 4, st>>>(a, *ws);
  return cudaGetLastError();
}

template <int NV, int KK>
cudaError_t win_scatter(const qm_scan_args &a, const qm_win_spec *ws, int sm_count, cudaStream_t st) {
  cudaError_t e = set_smem_once<qm_win_scatter<NV, KK>>(QM_WIN_SMEM_MAX);
  if (e != cudaSuccess || !ws) return e;
  qm_win_scatter<NV, KK><<<sm_count, QM_WIN_THREADS, qm_win_scatter_smem(ws->windows, NV), st>>>(a, *ws);
  return cudaGetLastError();
}

template <int NV, int FT>
cudaError_t win_agg(const qm_scan_args &a, const qm_win_spec *ws, int sm_count, cudaStream_t st) {
  cudaError_t e = set_smem_once<qm_win_agg<NV, FT>>(QM_WIN_SMEM_MAX);
  if (e != cudaSuccess || !ws) return e;
  qm_win_agg<NV, FT><<<sm_count, QM_WIN_THREADS, ((size_t)a.agg.n_words * 8) << ws->shift, st>>>(a, *ws);
  return cudaGetLastError();
}

template <int NV>
cudaError_t win_run(const qm_scan_args &a, const qm_win_spec *ws, int sm_count, cudaStream_t st) {
  const int kk = part_key_kind(a.key);
  cudaError_t e = kk == QM_KK_I64   ? win_count<QM_KK_I64>(a, ws, sm_count, st)
                  : kk == QM_KK_I32 ? win_count<QM_KK_I32>(a, ws, sm_count, st)
                                    : win_count<QM_KK_ANY>(a, ws, sm_count, st);
  if (e != cudaSuccess) return e;
  if (ws) qm_win_offsets<<<1, QM_WIN_THREADS, 0, st>>>(*ws);
  if (ws && (e = cudaGetLastError()) != cudaSuccess) return e;
  e = kk == QM_KK_I64   ? win_scatter<NV, QM_KK_I64>(a, ws, sm_count, st)
      : kk == QM_KK_I32 ? win_scatter<NV, QM_KK_I32>(a, ws, sm_count, st)
                        : win_scatter<NV, QM_KK_ANY>(a, ws, sm_count, st);
  if (e != cudaSuccess) return e;
  if constexpr (NV > 0) {
    const int ft = qm_value_features(a.agg);
    if (ft == QM_FT_SUM) return win_agg<NV, QM_FT_SUM>(a, ws, sm_count, st);
    if (ft == QM_FT_DBL) return win_agg<NV, QM_FT_DBL>(a, ws, sm_count, st);
  }
  return win_agg<NV, QM_FT_GEN>(a, ws, sm_count, st);
}
}  // namespace

bool qm_win_supported(const qm_aggspec &A) {
  return A.n_vcols <= QM_WIN_NV_MAX && qm_value_features(A) != QM_FT_FULL;
}

size_t qm_win_scatter_smem(int windows, int n_vcols) {
  return (size_t)QM_WIN_ROWS * 8 * (1 + n_vcols) + (size_t)windows * 8;
}

cudaError_t qm_win_setup(const qm_scan_args &a) {
  switch (a.agg.n_vcols) {
    case 0: return win_run<0>(a, nullptr, 0, nullptr);
    case 1: return win_run<1>(a, nullptr, 0, nullptr);
    default: return win_run<2>(a, nullptr, 0, nullptr);
  }
}

cudaError_t qm_launch_windows(const qm_scan_args &a, const qm_win_spec &ws, int sm_count, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  switch (a.agg.n_vcols) {
    case 0: return win_run<0>(a, &ws, sm_count, st);
    case 1: return win_run<1>(a, &ws, sm_count, st);
    default: return win_run<2>(a, &ws, sm_count, st);
  }
}
