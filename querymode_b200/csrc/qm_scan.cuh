// qm_scan.cuh — the fused filter + GROUP BY scan kernel template.  Its
// instantiations live in several translation units (qm_kernels.cu: the
// run-time-plan kernels; qm_scan_nv*.cu: kernels specialised for a value
// column count and key kind) so they compile in parallel.
#pragma once

#include "qm_kernels.cuh"
#include "qm_launch.h"

namespace qm {

// Shared memory of one block: the block-local group table (keys, then the
// accumulator words structure-of-arrays), then one survivor queue per warp.
// Survivors a lane aggregates at once when all have block-local slots: their
// gathers overlap (200M rows, 16 groups, a third selected: 645 us with one,
// 578 with two, 556 with four).  Rows that may go to the global table stay at
// one: their atomics, not their gathers, bound them (100M events 709 us with
// one, 725 with two, 926 with four).
#define QM_DRAIN_ROWS 4
// Entries of a warp's queue: a tile's survivors and those left over from
// before, and both tiles' of a pair unless most of their rows pass (those go
// in tile by tile).  26 KB a block, so that block-local tables of 80 KB leave
// room for two blocks on an SM, and one of 200 KB fits: room for every pair's
// rows (640 entries, 40 KB) took the second block from 20M rows into 4,000
// hashed keys (SUM and COUNT(*), half of the rows: 0.49 ms a query, 0.60 so).
#define QM_WQ 416
static_assert(QM_WQ >= QM_TILE_ROWS + 32 * QM_DRAIN_ROWS, "a tile's survivors fit beside those left over");
static_assert(QM_LOCAL_MAX_BYTES + QM_SCAN_THREADS / 32 * QM_WQ * 4 <= QM_SCAN_SMEM_MAX, "the largest block-local table fits");

#define QM_LOCAL_TRIAL 32          // drains after which a warp judges the hashed block-local table

struct smem_layout {
  int L;
  size_t keys_off, words_off, queue_off, stage_off, stage_warp_bytes, bytes;
};

// Per warp staging region: QM_STAGE_MAX_DEPTH mbarriers (32 bytes), then
// `depth` tile buffers of tile_bytes each.
__host__ __device__ inline smem_layout make_smem_layout(int local_slots, int local_hash, int n_words, int warps,
                                                        int stage_tile_bytes = 0, int stage_depth = 0, int priv = 0) {
  smem_layout s;
  s.L = local_slots;
  s.keys_off = 0;
  size_t kb = (local_slots > 0 && local_hash) ? (size_t)local_slots * 8 : 0;
  s.words_off = kb;
  size_t wb = (size_t)local_slots * n_words * 8 * (priv ? warps : 1);  // priv: one copy per warp
  s.queue_off = (s.words_off + wb + 15) & ~(size_t)15;
  s.stage_off = (s.queue_off + (size_t)warps * QM_WQ * sizeof(uint32_t) + 127) & ~(size_t)127;
  s.stage_warp_bytes = stage_depth > 0 ? (size_t)(32 + stage_depth * stage_tile_bytes + 127) & ~(size_t)127 : 0;
  s.bytes = s.stage_off + (size_t)warps * s.stage_warp_bytes;
  return s;
}

// The fused scan.  Each warp takes tiles of QM_TILE_ROWS rows round robin,
// filters them, appends the survivors' row indices to its own queue in
// shared memory and aggregates 32 survivors at a time (one per lane): gather
// the key and value cells, find the slot in the block-local table (else the
// global table) and update the accumulators.  With STAGED, the filter
// columns of the warp's next tiles stream into its shared-memory buffers by
// bulk async copies (lane 0 issues, an mbarrier per buffer counts the bytes)
// while the current tile is evaluated.
// NV / KK: the value-column count and key kind the kernel is specialised
// for (QM_NV_ANY / QM_KK_ANY: read from the plan at run time); FT / LM: what
// its value columns need and where its rows go (QM_FT_*, QM_LM_*).
// The first of a lane's n places in the queue, and the warp's total.
__device__ __forceinline__ uint32_t warp_places(uint32_t n, int lane, uint32_t &total) {
  uint32_t off = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(QM_FULL, off, o);
    if (lane >= o) off += x;
  }
  total = __shfl_sync(QM_FULL, off, 31);
  return off - n;
}

template <bool SEL, bool STAGED, int DD, int NV, int KK, int FT, int LM>
__global__ void __launch_bounds__(QM_SCAN_THREADS)
    qm_scan_kernel(const __grid_constant__ qm_scan_args a) {
  constexpr int D = DD == 0 && !SEL && !STAGED && LM == QM_LM_DIRECT && FT >= QM_FT_MIX && NV <= 2
                        ? (FT == QM_FT_SUM || NV == 0 ? QM_DRAIN_ROWS : 2)
                        : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  const qm_aggspec &A = a.agg;
  const qm_staging &S = a.stage;
  const smem_layout lay =
      make_smem_layout(a.local_slots, a.local_hash, A.n_words, warps, STAGED ? S.tile_bytes : 0, STAGED ? S.depth : 0,
                       a.priv);
  const int L = lay.L;
  uint64_t *lkeys = reinterpret_cast<uint64_t *>(smem + lay.keys_off);
  uint64_t *lw = reinterpret_cast<uint64_t *>(smem + lay.words_off);
  // a private (per-warp) table: this warp's copy
  uint64_t *lwm = a.priv ? lw + (int64_t)warp * L * A.n_words : lw;
  uint32_t *queue = reinterpret_cast<uint32_t *>(smem + lay.queue_off) + warp * QM_WQ;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + lay.stage_off + warp * lay.stage_warp_bytes);
  uint8_t *sbuf = smem + lay.stage_off + warp * lay.stage_warp_bytes + 32;
  __shared__ unsigned long long blk_selected;

  if (threadIdx.x == 0) blk_selected = 0;
  if (L > 0) {
    if (a.local_hash)
      for (int s = threadIdx.x; s < L; s += blockDim.x) lkeys[s] = QM_EMPTY_KEY;
    const int per = L * A.n_words;
    for (int i = threadIdx.x; i < per * (a.priv ? warps : 1); i += blockDim.x) lw[i] = A.init[(i % per) / L];
  }
  if (STAGED && lane == 0) {
    for (int d = 0; d < S.depth; ++d) mbar_init(&mbar[d], 1);
    fence_async_shared();
  }
  // launched early behind the clearing of a small table (no effect otherwise)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __syncthreads();

  // (tile numbers fit 32 bits: rows do)
  const int tile_rows = STAGED ? QM_TILE_ROWS : (a.lane_rows ? 32 * a.lane_rows : QM_SCAN_ROWS);
  const int n_tiles = (int)((a.n + tile_rows - 1) / tile_rows);
  const int full_tiles = (int)(a.n / tile_rows);
  const int gwarps = (int)gridDim.x * warps;
  const int first = (int)blockIdx.x * warps + warp;
  const uint32_t lt = lanemask_lt();
  int qn = 0;  // warp-uniform queue length
  // a hashed block-local table that takes few of a warp's first rows (many
  // groups, no hot ones) costs more than it saves: that warp leaves it
  // (deduplicating plans keep it: their rows are merged ahead of the lookup)
  int Lw = L, trial = DD == 0 && a.local_hash && L > 0 ? QM_LOCAL_TRIAL : 0, hits = 0;
  // aggregates queue entries [at, at + count), count <= 32 * D
  auto drain = [&](int at, int count) {
    if constexpr (D > 1) {
      uint32_t row[D];
      bool act[D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        act[d] = d * 32 + lane < count;
        row[d] = act[d] ? queue[at + d * 32 + lane] : 0;
      }
      __syncwarp();
      drain_rows<NV, KK, FT, D>(a, lwm, L, lane, row, act);
    } else {
      const bool act = lane < count;
      const int64_t row = act ? (int64_t)queue[at + lane] : 0;
      __syncwarp();
      const bool hit = drain_round_any<DD, NV, KK, FT, LM>(a, lkeys, lwm, Lw, lane, act, row);
      if (DD == 0 && LM != QM_LM_DIRECT && trial > 0) {
        hits += __popc(__ballot_sync(QM_FULL, hit));
        if (--trial == 0 && hits < QM_LOCAL_TRIAL * 32 / 8) Lw = 0;
      }
    }
  };
  unsigned long long selected = 0;
  const char *pf_base;  // the filter column this lane prefetches
  int pf_elem;
  prefetch_column(a.pred, lane, pf_base, pf_elem);
  uint32_t pf_want = ~0u;
  int issued = 0;  // STAGED: tiles whose copies were issued (in order)
  bool failed = false;

  // lane 0 issues the copies of the warp's k-th tile into buffer k % depth
  auto issue = [&](int k) {
    const int64_t tile = first + (int64_t)k * gwarps;
    if (tile >= full_tiles) return;
    if (lane == 0) {
      fence_async_shared();
      const int b = (int)(k % S.depth);
      uint8_t *dst = sbuf + b * S.tile_bytes;
      mbar_expect_tx(&mbar[b], (uint32_t)S.tile_bytes);
      for (int c = 0; c < S.n; ++c)
        bulk_g2s(dst + S.off[c], reinterpret_cast<const uint8_t *>(S.data[c]) + tile * QM_TILE_ROWS * S.elem[c],
                 (uint32_t)(QM_TILE_ROWS * S.elem[c]), &mbar[b]);
    }
    issued = k + 1;
  };
  if (STAGED)
    for (int k = 0; k < S.depth - 1; ++k) issue(k);

  // with zone maps, virtual tile v walks the kept zones' tiles
  // (STAGED and short tiles have none)
  constexpr int ZONE = QM_ZONE_ROWS / QM_SCAN_ROWS;
  const int n_virtual = a.zones ? (int)(a.n_zone_tiles / (QM_ZONE_TILES / ZONE)) : n_tiles;
  auto tile_of = [&](int v) -> int {
    return a.zones ? (int)(a.zones[v / ZONE] * ZONE + v % ZONE) : v;
  };
  int k = 0;
  for (int v = first; v < n_virtual; v += gwarps, ++k) {
    const int tile = tile_of(v);
    if (tile >= n_tiles) continue;  // the table's last zone is partial
    const int64_t e0 = (int64_t)tile * tile_rows;
    uint32_t m = 0;
    bool fill = false;  // m's rows are not in the queue yet
    if (STAGED && tile < full_tiles) {
      __syncwarp();
      issue(k + S.depth - 1);
      const int b = (int)(k % S.depth);
      if (!mbar_wait(&mbar[b], (uint32_t)((k / S.depth) & 1))) {
        set_error(a.status, QM_DEV_TIMEOUT);
        failed = true;
        break;
      }
      m = eval_pred_staged(a.pred, S, sbuf + b * S.tile_bytes, e0, lane, (1u << QM_R) - 1);
      // append survivors (rows e0 + j*32 + lane)
      uint32_t base = (uint32_t)qn;
#pragma unroll
      for (int j = 0; j < QM_R; ++j) {
        const uint32_t bal = __ballot_sync(QM_FULL, (m >> j) & 1);
        if ((m >> j) & 1) queue[base + __popc(bal & lt)] = (uint32_t)(e0 + j * 32 + lane);
        base += __popc(bal);
      }
      const int tot = (int)base - qn;
      qn = (int)base;
      selected += tot;
    } else if (!SEL && a.lane_rows && a.lane_rows < QM_R) {
      // few rows: short tiles, a row of the warp's 32 per lane and step, so
      // that the serial drains of a tile spread over the idle warps
      for (int j = 0; j < a.lane_rows; ++j) {
        const int64_t row = e0 + j * 32 + lane;
        const bool pass = eval_pred_row(a.pred, row, row < a.n);
        const uint32_t bal = __ballot_sync(QM_FULL, pass);
        if (pass) queue[qn + __popc(bal & lt)] = (uint32_t)row;
        qn += __popc(bal);
        selected += __popc(bal);
      }
    } else {
      if (!SEL && a.vec_ok && e0 + tile_rows <= a.n) {
        // full dense tiles: the lane's rows are r0 .. r0 + 7 in each
        const int64_t r0 = e0 + (int64_t)lane * QM_R;
        const int nxt = v + gwarps < n_virtual ? tile_of(v + gwarps) : n_tiles;
        if (nxt < full_tiles) prefetch_tile_l2(pf_base, pf_elem, pf_want, (int64_t)nxt * tile_rows, tile_rows, lane);
        m = a.lane_rows ? eval_pred_contig<1>(a.pred, r0, (1u << QM_R) - 1, pf_want)
                        : eval_pred_contig<QM_SCAN_TILES>(a.pred, r0, (1u << (QM_SCAN_TILES * QM_R)) - 1, pf_want);
      } else {
#pragma unroll 1
        for (int h = 0; h * QM_TILE_ROWS < tile_rows; ++h) {
          const int64_t r0 = e0 + h * QM_TILE_ROWS + (int64_t)lane * QM_R;  // this lane's first element
          int64_t rowv[QM_R];
          uint32_t mh = 0;
#pragma unroll
          for (int j = 0; j < QM_R; ++j) {
            const bool in = r0 + j < a.n;
            mh |= (uint32_t)in << j;
            rowv[j] = r0 + j;
          }
          if (SEL) {
#pragma unroll
            for (int j = 0; j < QM_R; ++j) rowv[j] = ((mh >> j) & 1) ? (int64_t)__ldg(a.sel + r0 + j) : 0;
          }
          auto rowf = [&](int j) { return rowv[j]; };
          m |= eval_pred(a.pred, rowf, mh) << (h * QM_R);
        }
      }
      fill = true;
    }
    do {
      if (fill) {  // (order inside the queue does not matter: FIRST is a min)
        uint32_t now = m, tot;
        uint32_t q = qn + warp_places(__popc(now), lane, tot);
        fill = qn + tot > QM_WQ;
        if (fill) {  // the first tile's rows, then the second's
          now &= (1u << QM_R) - 1;
          m ^= now;
          q = qn + warp_places(__popc(now), lane, tot);
        }
        const uint32_t r0u = (uint32_t)(e0 + lane * QM_R);
        for (uint32_t mm = now; mm; mm &= mm - 1) {
          const uint32_t j = (uint32_t)(__ffs(mm) - 1);
          const uint32_t row = r0u + (j & (QM_R - 1)) + (j / QM_R) * QM_TILE_ROWS;
          queue[q++] = SEL ? __ldg(a.sel + row) : row;
        }
        qn += (int)tot;
        selected += tot;
      }
      __syncwarp();
      while (qn >= 32 * D) {
        drain(qn - 32 * D, 32 * D);
        qn -= 32 * D;
      }
    } while (fill);
  }
  if (STAGED && failed) {
    // let every copy still in flight land before the block's memory goes
    for (int j = k; j < issued; ++j)
      if (!mbar_wait(&mbar[j % S.depth], (uint32_t)((j / S.depth) & 1))) break;
  }
  if (qn > 0) drain(0, qn);

  if (lane == 0 && selected) atomicAdd(&blk_selected, selected);
  __syncthreads();
  if (threadIdx.x == 0 && blk_selected) atomicAdd(&a.status->rows_selected, blk_selected);

  // merge the block-local table into the global table
  if (L > 0) {
    if (a.priv) {  // fold the per-warp copies into copy 0
      const int cw = A.w_count;
      for (int s = threadIdx.x; s < L; s += blockDim.x)
        for (int w = 1; w < warps; ++w) {
          const uint64_t *src = lw + (int64_t)w * L * A.n_words + s;
          if (src[(int64_t)cw * L] != 0) merge_plain(A, lw + s, src, L);
        }
      __syncthreads();
    }
    merge_block(a, lkeys, lw);
  }
}

// Launch of one instantiation: `early`, overlapping the end of the clearing
// launch ahead of it (the kernel waits for it before it touches the table).
// per_sm non-null: asks how many of its blocks fit an SM instead.
template <class KERNEL>
inline cudaError_t launch_scan_kernel(KERNEL kernel, const qm_scan_args &a, int blocks, size_t smem, cudaStream_t st,
                                      int *per_sm) {
  if (per_sm) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, QM_SCAN_THREADS, smem);
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)blocks);
  c.blockDim = dim3(QM_SCAN_THREADS);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = a.early ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&c, kernel, a);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, not by the next launch
  return e;
}

}  // namespace qm
