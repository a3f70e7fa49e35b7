// qm_kernels.cuh — device code of the fused filter -> GROUP BY path.
//
// One warp owns a tile of QM_TILE_ROWS consecutive rows (or selection
// entries).  Per tile:
//   1. predicates: each lane tests QM_R rows (lane, lane+32, ...), one term at
//      a time; a term's column is read only for rows still alive, so a
//      selective first term skips the sectors of later columns;
//   2. compaction: __ballot_sync masks + popcount prefix sums put the
//      surviving row offsets, in ascending row order, into a per-warp list;
//   3. aggregation: 32 survivors at a time, the lane gathers its row's key and
//      value cells and updates the block-local shared-memory table (or the
//      global table when the key misses it).  The block-local words are built
//      from native 32-bit shared-memory atomics (see agg_row_local).
// At block end the shared-memory table is merged into the global table with
// atomics.  Float sums are compensated (TwoSum of every atomic add: the old
// value returned by atomicAdd gives the exact rounding error, which goes to a
// second word), integer sums are exact 128-bit, MIN/MAX are integer atomics
// on an order-preserving image of the value.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/qm_gpu.h"
#include "qm_plan.h"

#define QM_FULL 0xffffffffu

namespace qm {

// murmur3 fmix64 finaliser — the hash the reference's LinearHashTable uses
// (wasm/src/query/vector_engine.zig:209-250)
__host__ __device__ __forceinline__ uint64_t fmix64(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdULL;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ULL;
  k ^= k >> 33;
  return k;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ---- column access ----------------------------------------------------------
// Column cells are read once per query: cache-streaming loads keep the group
// table (read-modify-written by atomics) resident in L2.
// A miss fetches 64 bytes from DRAM instead of the default 128 (measured on
// one 8-byte cell in every 128 bytes of 800 MB: 800 -> 400 MB, 117 -> 65 us):
// the gathers of a filtered scan touch cells far apart.
__device__ __forceinline__ int ld64(const int *p) {
  int v;
  asm("ld.global.cs.L2::64B.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ long long ld64(const long long *p) {
  long long v;
  asm("ld.global.cs.L2::64B.s64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld64(const float *p) {
  float v;
  asm("ld.global.cs.L2::64B.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld64(const double *p) {
  double v;
  asm("ld.global.cs.L2::64B.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld64(const int4 *p) {
  int4 v;
  asm("ld.global.cs.L2::64B.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ longlong2 ld64(const longlong2 *p) {
  longlong2 v;
  asm("ld.global.cs.L2::64B.v2.s64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld64(const float4 *p) {
  float4 v;
  asm("ld.global.cs.L2::64B.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld64(const double2 *p) {
  double2 v;
  asm("ld.global.cs.L2::64B.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

template <typename T>
__device__ __forceinline__ T ldcs(const void *p, int64_t r) {
  return ld64(reinterpret_cast<const T *>(p) + r);
}

__device__ __forceinline__ bool cell_null(const uint32_t *nb, int64_t r) {
  return nb != nullptr && ((__ldg(nb + (r >> 5)) >> (r & 31)) & 1u);
}

__device__ __forceinline__ int64_t ld_int(const void *p, int dtype, int64_t r) {
  return dtype == QM_I32 ? (int64_t)ldcs<int>(p, r) : (int64_t)ldcs<long long>(p, r);
}

__device__ __forceinline__ double ld_flt(const void *p, int dtype, int64_t r) {
  return dtype == QM_F32 ? (double)ldcs<float>(p, r) : ldcs<double>(p, r);
}

// order-preserving image of a double in int64 (after -0 -> +0)
__host__ __device__ __forceinline__ int64_t f2ord(double d) {
  int64_t b;
#ifdef __CUDA_ARCH__
  b = __double_as_longlong(d);
#else
  memcpy(&b, &d, 8);
#endif
  return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}

__host__ __device__ __forceinline__ double ord2f(int64_t o) {
  int64_t b = o >= 0 ? o : (o ^ 0x7fffffffffffffffLL);
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double d;
  memcpy(&d, &b, 8);
  return d;
#endif
}

// ---- predicates -------------------------------------------------------------
__device__ __forceinline__ bool fcmp(double v, int op, double t) {
  switch (op) {
    case QC_EQ: return v == t;
    case QC_NEQ: return v != t;
    case QC_LT: return v < t;
    case QC_LTE: return v <= t;
    case QC_GT: return v > t;
    default: return v >= t;
  }
}

// JS: coerceCompare(number v, bigint b) -> BigInt(trunc(v)) <op> b, with a
// non-finite v compared as a number (src/decode.ts:480-485).
__device__ __forceinline__ bool fbig(double v, int op, int64_t b) {
  if (isnan(v)) return op == QC_NEQ;
  int c;
  if (isinf(v)) {
    c = v > 0 ? 1 : -1;
    if (op == QC_EQ) return false;
    if (op == QC_NEQ) return true;
  } else {
    double t = trunc(v);
    if (t >= 9223372036854775808.0) c = 1;
    else if (t < -9223372036854775808.0) c = -1;
    else {
      long long ti = (long long)t;
      c = ti < b ? -1 : (ti > b ? 1 : 0);
    }
  }
  switch (op) {
    case QC_EQ: return c == 0;
    case QC_NEQ: return c != 0;
    case QC_LT: return c < 0;
    case QC_LTE: return c <= 0;
    case QC_GT: return c > 0;
    default: return c >= 0;
  }
}

__device__ __forceinline__ bool fterm(const qm_term &t, double v) {
  switch (t.kind) {
    case QT_FRANGE:
      return ((t.op & 1) ? v >= t.f0 : v > t.f0) && ((t.op & 2) ? v <= t.f1 : v < t.f1);
    case QT_FCMP: return fcmp(v, t.op, t.f0);
    case QT_FBETWEEN: return v >= t.f0 && v <= t.f1;
    case QT_FNBETWEEN: return v < t.f0 || v > t.f1;
    default: return fbig(v, t.op, t.lo);
  }
}

// Tests term `t` on the lane's alive rows (bit j of m = row[j] alive).
template <typename ROWS>
__device__ __forceinline__ uint32_t eval_term(const qm_term &t, const ROWS &row, uint32_t m) {
  uint32_t pass = 0;
  if (t.kind <= QT_FALSE) {
    pass = t.kind == QT_TRUE ? ((1u << QM_R) - 1) : 0u;
  } else if (t.dtype == QM_I32 || t.dtype == QM_I64) {
    int64_t v[QM_R];
    if (t.dtype == QM_I32) {
#pragma unroll
      for (int j = 0; j < QM_R; ++j) v[j] = ((m >> j) & 1) ? (int64_t)ldcs<int>(t.data, row(j)) : 0;
    } else {
#pragma unroll
      for (int j = 0; j < QM_R; ++j) v[j] = ((m >> j) & 1) ? (int64_t)ldcs<long long>(t.data, row(j)) : 0;
    }
    const bool inr = t.kind == QT_IRANGE;
#pragma unroll
    for (int j = 0; j < QM_R; ++j) {
      bool in = v[j] >= t.lo && v[j] <= t.hi;
      pass |= (uint32_t)(in == inr) << j;
    }
  } else {
    double v[QM_R];
    if (t.dtype == QM_F32) {
#pragma unroll
      for (int j = 0; j < QM_R; ++j) v[j] = ((m >> j) & 1) ? (double)ldcs<float>(t.data, row(j)) : 0.0;
    } else {
#pragma unroll
      for (int j = 0; j < QM_R; ++j) v[j] = ((m >> j) & 1) ? ldcs<double>(t.data, row(j)) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < QM_R; ++j) pass |= (uint32_t)fterm(t, v[j]) << j;
  }
  if (t.nulls != nullptr) {
#pragma unroll
    for (int j = 0; j < QM_R; ++j)
      if (((m >> j) & 1) && cell_null(t.nulls, row(j)))
        pass = (pass & ~(1u << j)) | ((uint32_t)t.null_pass << j);
  }
  return m & pass;
}

// H full dense tiles one after another, lane owns rows r0 + h * QM_TILE_ROWS + j
// (j < 8, r0 = first row + 8 * lane): its runs of a column in 16-byte loads
// (one or two 32-byte sectors each), NULL bits as one byte a run.  Bit h * 8 + j
// of a mask is row j of tile h.
template <int H, typename V, typename T, int PER>
__device__ __forceinline__ void load_contig(const void *data, int64_t r0, T (&v)[H * QM_R]) {
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const V *p = reinterpret_cast<const V *>(reinterpret_cast<const T *>(data) + r0 + h * QM_TILE_ROWS);
#pragma unroll
    for (int k = 0; k < QM_R / PER; ++k) {
      const V x = ld64(p + k);
      const T *xs = reinterpret_cast<const T *>(&x);
#pragma unroll
      for (int i = 0; i < PER; ++i) v[h * QM_R + k * PER + i] = xs[i];
    }
  }
}

template <int H>
__device__ __forceinline__ uint32_t eval_term_contig(const qm_term &t, int64_t r0, uint32_t m) {
  constexpr int R = H * QM_R;
  constexpr uint32_t ALL = (1u << R) - 1;
  uint32_t pass = 0;
  if (m == 0) return 0;  // a lane without rows left reads nothing
  if (t.kind <= QT_FALSE) {
    pass = t.kind == QT_TRUE ? ALL : 0u;
  } else if (t.dtype == QM_I32) {
    // the planner clamps int32 bounds to the int32 range: one unsigned
    // compare per cell tests lo <= v <= hi
    int w[R];
    load_contig<H, int4, int, 4>(t.data, r0, w);
    const int lo = (int)t.lo;
    const uint32_t span = (uint32_t)((int)t.hi - lo);
#pragma unroll
    for (int j = 0; j < R; ++j) pass |= (uint32_t)((uint32_t)(w[j] - lo) <= span) << j;
    if (t.kind == QT_INRANGE) pass = ~pass & ALL;
  } else if (t.dtype == QM_I64) {
    long long w[R];
    load_contig<H, longlong2, long long, 2>(t.data, r0, w);
    const uint64_t span = (uint64_t)t.hi - (uint64_t)t.lo;
#pragma unroll
    for (int j = 0; j < R; ++j) pass |= (uint32_t)((uint64_t)w[j] - (uint64_t)t.lo <= span) << j;
    if (t.kind == QT_INRANGE) pass = ~pass & ALL;
  } else {
    double v[R];
    if (t.dtype == QM_F32) {
      float w[R];
      load_contig<H, float4, float, 4>(t.data, r0, w);
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = w[j];
    } else {
      load_contig<H, double2, double, 2>(t.data, r0, v);
    }
    if (t.kind == QT_FRANGE) {  // bounds are inclusive after planning
#pragma unroll
      for (int j = 0; j < R; ++j) pass |= (uint32_t)(v[j] >= t.f0 && v[j] <= t.f1) << j;
    } else {
#pragma unroll
      for (int j = 0; j < R; ++j) pass |= (uint32_t)fterm(t, v[j]) << j;
    }
  }
  if (t.nulls != nullptr) {
    // r0 is a multiple of 8: the lane's 8 NULL bits are one byte
    uint32_t nb = 0;
#pragma unroll
    for (int h = 0; h < H; ++h)
      nb |= ((__ldg(t.nulls + ((r0 + h * QM_TILE_ROWS) >> 5)) >> (r0 & 31)) & 0xffu) << (h * 8);
    const uint32_t np = t.null_pass ? ALL : 0u;
    pass = (pass & ~nb) | (np & nb);
  }
  return m & pass;
}

// Pulls `rows` rows of the filter columns into L2 ahead of their evaluation:
// lane i issues one bulk prefetch for term i if bit i of `want` is set (base:
// its column, or null; elem: bytes of a cell).
__device__ __forceinline__ void prefetch_tile_l2(const char *base, int elem, uint32_t want, int64_t e0, int rows,
                                                 int lane) {
  if (base != nullptr && ((want >> lane) & 1))
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base + e0 * elem), "r"(rows * elem) : "memory");
}

__device__ __forceinline__ void prefetch_column(const qm_pred &P, int lane, const char *&base, int &elem) {
  const int nt = P.n_groups > 0 ? P.group_end[P.n_groups - 1] : P.n_and;
  base = nullptr;
  elem = 0;
  if (lane < nt && P.t[lane].kind > QT_FALSE) {
    base = reinterpret_cast<const char *>(P.t[lane].data);
    elem = (P.t[lane].dtype == QM_I32 || P.t[lane].dtype == QM_F32) ? 4 : 8;
  }
}

// A term's tile is worth prefetching while at least this many of the warp's
// 32 runs of 8 rows still have a row when the term is reached: below that the
// prefetch reads more of the column than the term does (a 1 % flag ahead of a
// second column, 200M rows: query 1.33 -> 1.18 ms without it; a month of a
// year leaves half the runs of the second column, which is faster with it).
#define QM_PREFETCH_RUNS 8

// want: bit i set if term i of the next tile should be prefetched, judged by
// this tile.
template <int H>
__device__ __forceinline__ uint32_t eval_pred_contig(const qm_pred &P, int64_t r0, uint32_t m, uint32_t &want) {
  want = 0;
  for (int i = 0; i < P.n_and; ++i) {
    const int runs = __popc(__ballot_sync(QM_FULL, m != 0));
    if (runs == 0) return 0;
    if (runs >= QM_PREFETCH_RUNS) want |= 1u << i;
    m = eval_term_contig<H>(P.t[i], r0, m);
  }
  if (P.n_groups > 0) {
    uint32_t any = 0;
    int b = P.n_and;
    for (int g = 0; g < P.n_groups; ++g) {
      uint32_t mg = m & ~any;
      const int e = P.group_end[g];
      for (int i = b; i < e; ++i) {
        const int runs = __popc(__ballot_sync(QM_FULL, mg != 0));
        if (runs == 0) break;
        if (runs >= QM_PREFETCH_RUNS) want |= 1u << i;
        mg = eval_term_contig<H>(P.t[i], r0, mg);
      }
      any |= mg;
      b = e;
    }
    m = any;
  }
  return m;
}

// ---- bulk async copies into shared memory (cp.async.bulk + mbarrier) ------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// global -> shared bulk copy; dst, src and bytes are multiples of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

#define QM_WAIT_LIMIT (1 << 22)

// Bounded wait for a phase of an mbarrier; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  for (int i = 0; i < QM_WAIT_LIMIT; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Term evaluation on a staged tile: rows e0 + j*32 + lane, cells read from
// the shared-memory copy (consecutive lanes, consecutive addresses).
__device__ __forceinline__ uint32_t eval_term_staged(const qm_term &t, const qm_staging &S, const uint8_t *buf,
                                                     int64_t e0, int lane, uint32_t m) {
  uint32_t pass = 0;
  if (t.kind <= QT_FALSE) {
    pass = t.kind == QT_TRUE ? ((1u << QM_R) - 1) : 0u;
  } else {
    const uint8_t *col = buf + S.off[t.sidx];
    if (t.dtype == QM_I32 || t.dtype == QM_I64) {
      const bool inr = t.kind == QT_IRANGE;
#pragma unroll
      for (int j = 0; j < QM_R; ++j) {
        const int64_t v = t.dtype == QM_I32 ? (int64_t)reinterpret_cast<const int *>(col)[j * 32 + lane]
                                            : (int64_t)reinterpret_cast<const long long *>(col)[j * 32 + lane];
        pass |= (uint32_t)((v >= t.lo && v <= t.hi) == inr) << j;
      }
    } else {
#pragma unroll
      for (int j = 0; j < QM_R; ++j) {
        const double v = t.dtype == QM_F32 ? (double)reinterpret_cast<const float *>(col)[j * 32 + lane]
                                           : reinterpret_cast<const double *>(col)[j * 32 + lane];
        pass |= (uint32_t)fterm(t, v) << j;
      }
    }
  }
  if (t.nulls != nullptr) {
#pragma unroll
    for (int j = 0; j < QM_R; ++j) {
      const uint32_t w = __ldg(t.nulls + ((e0 >> 5) + j));
      if ((w >> lane) & 1) pass = (pass & ~(1u << j)) | ((uint32_t)t.null_pass << j);
    }
  }
  return m & pass;
}

__device__ __forceinline__ uint32_t eval_pred_staged(const qm_pred &P, const qm_staging &S, const uint8_t *buf,
                                                     int64_t e0, int lane, uint32_t m) {
  for (int i = 0; i < P.n_and; ++i) {
    if (!__any_sync(QM_FULL, m)) return 0;
    m = eval_term_staged(P.t[i], S, buf, e0, lane, m);
  }
  if (P.n_groups > 0) {
    uint32_t any = 0;
    int b = P.n_and;
    for (int g = 0; g < P.n_groups; ++g) {
      uint32_t mg = m & ~any;
      const int e = P.group_end[g];
      for (int i = b; i < e; ++i) {
        if (!__any_sync(QM_FULL, mg)) break;
        mg = eval_term_staged(P.t[i], S, buf, e0, lane, mg);
      }
      any |= mg;
      b = e;
    }
    m = any;
  }
  return m;
}

// AND terms, then the OR of the groups' AND chains (src/decode.ts:558-578).
template <typename ROWS>
__device__ __forceinline__ uint32_t eval_pred(const qm_pred &P, const ROWS &row, uint32_t m) {
  for (int i = 0; i < P.n_and; ++i) {
    if (!__any_sync(QM_FULL, m)) return 0;
    m = eval_term(P.t[i], row, m);
  }
  if (P.n_groups > 0) {
    uint32_t any = 0;
    int b = P.n_and;
    for (int g = 0; g < P.n_groups; ++g) {
      uint32_t mg = m & ~any;
      const int e = P.group_end[g];
      for (int i = b; i < e; ++i) {
        if (!__any_sync(QM_FULL, mg)) break;
        mg = eval_term(P.t[i], row, mg);
      }
      any |= mg;
      b = e;
    }
    m = any;
  }
  return m;
}

// One row per lane (act: this lane has one).
__device__ __forceinline__ bool eval_term_row(const qm_term &t, int64_t r, bool act) {
  bool pass = t.kind == QT_TRUE;
  if (act && t.kind > QT_FALSE) {
    if (t.dtype == QM_I32 || t.dtype == QM_I64) {
      const int64_t v = ld_int(t.data, t.dtype, r);
      pass = (v >= t.lo && v <= t.hi) == (t.kind == QT_IRANGE);
    } else {
      pass = fterm(t, ld_flt(t.data, t.dtype, r));
    }
  }
  if (act && cell_null(t.nulls, r)) pass = t.null_pass != 0;
  return act && pass;
}

__device__ __forceinline__ bool eval_pred_row(const qm_pred &P, int64_t r, bool act) {
  for (int i = 0; i < P.n_and; ++i) {
    if (!__any_sync(QM_FULL, act)) return false;
    act = eval_term_row(P.t[i], r, act);
  }
  if (P.n_groups > 0) {
    bool any = false;
    int b = P.n_and;
    for (int g = 0; g < P.n_groups; ++g) {
      bool mg = act && !any;
      const int e = P.group_end[g];
      for (int i = b; i < e; ++i) {
        if (!__any_sync(QM_FULL, mg)) break;
        mg = eval_term_row(P.t[i], r, mg);
      }
      any = any || mg;
      b = e;
    }
    act = any;
  }
  return act;
}

// ---- group keys -------------------------------------------------------------
// Key word of one row.  special: 0 ordinary, 1 the key equals the empty-slot
// sentinel (hash mode), 2 NULL key.
// Key kinds a scan kernel can be specialised for (KK): 0 any plan; 1 one
// int64 column without NULLs; 2 one int32 column without NULLs; 3 no GROUP BY.
#define QM_KK_ANY 0
#define QM_KK_I64 1
#define QM_KK_I32 2
#define QM_KK_NONE 3
// Value-column counts (NV): 0..QM_MAX_VCOLS exactly, or QM_NV_ANY (read the
// plan's n_vcols at run time).
#define QM_NV_ANY (QM_MAX_VCOLS + 1)
#define QM_NV_BOUND(NV) ((NV) > QM_MAX_VCOLS ? QM_MAX_VCOLS : (NV))
// What the value columns of a plan can need (FT): 0 anything, fixed-point
// sums included; 1 anything but those; 2 every float sum kept as block-local
// integers (qm_vcol.lim, planned from statistics); 3 as 2 without NULLs and
// 128-bit integer sums; 4 as 3, and every column is a float one with a SUM
// only.  A path a kernel leaves out costs its drain no instructions: the flags
// are tested once per row and column otherwise.
#define QM_FT_FULL 0
#define QM_FT_DBL 1
#define QM_FT_GEN 2
#define QM_FT_MIX 3
#define QM_FT_SUM 4
// Where rows go (LM): 0 as planned; 1 every row has a slot of the
// block-local table (a dense key range, or no GROUP BY); 2 a hash table with
// aligned slots (qm_scan_args.head), through a hashed block-local table or not.
#define QM_LM_ANY 0
#define QM_LM_DIRECT 1
#define QM_LM_HASH 2

template <int KK = QM_KK_ANY>
__device__ __forceinline__ uint64_t row_key(const qm_keyspec &K, int64_t r, int &special) {
  special = 0;
  if (KK == QM_KK_NONE) return 0;
  if (KK == QM_KK_I64 || KK == QM_KK_I32) {
    const uint64_t k = KK == QM_KK_I64 ? (uint64_t)ldcs<long long>(K.data[0], r)
                                       : (uint64_t)(int64_t)ldcs<int>(K.data[0], r);
    if (K.mode == QK_HASH && k == QM_EMPTY_KEY) special = 1;
    return k;
  }
  if (K.n_cols == 0) return 0;
  uint64_t k;
  if (K.pack == QP_CONCAT) {
    uint32_t a = (uint32_t)ldcs<int>(K.data[0], r), b = (uint32_t)ldcs<int>(K.data[1], r);
    k = ((uint64_t)a << 32) | b;
  } else if (K.pack == QP_DIGITS) {
    k = 0;
    for (int i = 0; i < K.n_cols; ++i) {
      uint64_t d;
      if (K.knullable[i] && cell_null(K.nulls[i], r)) d = 0;
      else d = (uint64_t)(ld_int(K.data[i], K.dtype[i], r) - K.kbase[i]) + (uint64_t)K.knullable[i];
      k += d * K.kmul[i];
    }
  } else {
    if (cell_null(K.nulls[0], r)) {
      special = 2;
      return 0;
    }
    switch (K.dtype[0]) {
      case QM_I32: k = (uint64_t)(int64_t)ldcs<int>(K.data[0], r); break;
      case QM_I64: k = (uint64_t)ldcs<long long>(K.data[0], r); break;
      default: {
        // String(v) identity: -0 and 0 share "0", every NaN is "NaN"
        double d = ld_flt(K.data[0], K.dtype[0], r);
        if (d == 0.0) d = 0.0;
        k = isnan(d) ? 0x7ff8000000000000ULL : (uint64_t)__double_as_longlong(d);
      }
    }
  }
  if (K.mode == QK_HASH && k == QM_EMPTY_KEY) special = 1;
  return k;
}

__device__ __forceinline__ void set_error(qm_status *st, int code) {
  atomicCAS(&st->error, 0, code);
}

// Home slot of a key among n_slots (any number): the hash as a fraction of them.
__device__ __forceinline__ uint64_t home_slot(uint64_t key, int64_t n_slots) {
  return __umul64hi(fmix64(key), (uint64_t)n_slots);
}

// Linear probing with a CAS claim of the key word.  Accumulator words are
// pre-initialised, so a claimed slot is immediately usable.
__device__ __forceinline__ int64_t global_find(uint64_t *table, int stride, int64_t n_slots,
                                               uint64_t key, int max_probe, qm_status *st) {
  uint64_t s = home_slot(key, n_slots);
  for (int p = 0; p < max_probe; ++p) {
    unsigned long long *kp = reinterpret_cast<unsigned long long *>(table + s * stride);
    uint64_t k = *reinterpret_cast<volatile unsigned long long *>(kp);
    if (k == key) return (int64_t)s;
    if (k == QM_EMPTY_KEY) {
      uint64_t prev = atomicCAS(kp, QM_EMPTY_KEY, key);
      if (prev == QM_EMPTY_KEY) {
        atomicAdd(&st->groups_inserted, 1ULL);
        return (int64_t)s;
      }
      if (prev == key) return (int64_t)s;
    }
    if (++s == (uint64_t)n_slots) s = 0;
  }
  return -1;
}

__device__ __forceinline__ int64_t global_slot(const qm_scan_args &a, uint64_t key, int special) {
  if (a.key.mode == QK_NONE) return 0;
  if (a.key.mode == QK_DIRECT) {
    if (special == 2) return a.n_slots;
    uint64_t d = key - (uint64_t)a.key.base;
    if (d >= (uint64_t)a.n_slots) {
      set_error(a.status, QM_DEV_RANGE);
      return -1;
    }
    return (int64_t)d;
  }
  if (special) return a.n_slots + special - 1;
  int64_t s = global_find(a.table, a.stride, a.n_slots, key, a.max_probe, a.status);
  if (s < 0) set_error(a.status, QM_DEV_OVERFLOW);
  return s;
}

// The slot of an ordinary key of a hash table with aligned slots, and the
// words beside the key as the probe that ended there read them.
__device__ __forceinline__ int64_t global_find_head(const qm_scan_args &a, uint64_t key, uint64_t (&w)[QM_HEAD_WORDS]) {
  uint64_t s = home_slot(key, a.n_slots);
  for (int p = 0; p < a.max_probe; ++p) {
    uint64_t *slot = a.table + s * a.stride;
    uint64_t k;
    asm volatile("ld.global.cg.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(k), "=l"(w[0]), "=l"(w[1]), "=l"(w[2])
                 : "l"(slot)
                 : "memory");
    if (k == QM_EMPTY_KEY) {
      k = atomicCAS(reinterpret_cast<unsigned long long *>(slot), QM_EMPTY_KEY, key);
      if (k == QM_EMPTY_KEY) {
        atomicAdd(&a.status->groups_inserted, 1ULL);
        return (int64_t)s;
      }
    }
    if (k == key) return (int64_t)s;
    if (++s == (uint64_t)a.n_slots) s = 0;
  }
  set_error(a.status, QM_DEV_OVERFLOW);
  return -1;
}

// A group's slot from its key, without inserting (the key is in the table).
__device__ __forceinline__ int64_t find_slot(const qm_scan_args &a, uint64_t key, int special) {
  if (a.key.mode == QK_NONE) return 0;
  if (a.key.mode == QK_DIRECT) {
    if (special == 2) return a.n_slots;
    const uint64_t d = key - (uint64_t)a.key.base;
    return d < (uint64_t)a.n_slots ? (int64_t)d : -1;
  }
  if (special) return a.n_slots + special - 1;
  uint64_t s = home_slot(key, a.n_slots);
  for (int p = 0; p < a.max_probe; ++p) {
    const uint64_t k = a.table[s * a.stride];
    if (k == key) return (int64_t)s;
    if (k == QM_EMPTY_KEY) return -1;
    if (++s == (uint64_t)a.n_slots) s = 0;
  }
  return -1;
}

// Block-local lookup: slots in buckets of four (two 16-byte reads); a key may
// sit in any slot of its bucket, the first keys to come take the slots and a
// key that finds its bucket full goes to the global table.  No probe loop:
// its lanes leave at different steps, and a miss walks it to the end (against
// eight probes of a half-full table, 20M rows into 500,000 groups 1,045 ->
// 1,015 us and 100M events no slower; buckets of two hold fewer hot keys, 725
// against 709 us).
//
// The bucket comes from the hash's high bits, which differ for keys that
// follow one another (its low bits put 15 of the keys 0..15 on the same bank:
// 20M rows pushed, half of them kept, 330 us of scan, 189 so), and the slot of a bucket
// that a key tries first from its low ones: first slots alone are eight banks.
#define QM_LOCAL_BUCKET 4
__device__ __forceinline__ int local_find(uint64_t *lkeys, int L, uint64_t key) {
  // a multiplicative hash of the folded key: this table only fronts the
  // global one, so a poor spread costs misses, not correctness
  const uint32_t h = ((uint32_t)key * 0x9e3779b1u) ^ ((uint32_t)(key >> 32) * 0x85ebca6bu);
  const uint32_t s = __umulhi(h, (uint32_t)L) & ~(uint32_t)(QM_LOCAL_BUCKET - 1);
  uint64_t k[QM_LOCAL_BUCKET];
  asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(k[0]), "=l"(k[1]) : "r"(smem_u32(lkeys + s)));
  asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(k[2]), "=l"(k[3]) : "r"(smem_u32(lkeys + s + 2)));
  int at = -1;
  bool room = false;
#pragma unroll
  for (int i = 0; i < QM_LOCAL_BUCKET; ++i) {
    if (k[i] == key) at = (int)s + i;
    room = room || k[i] == QM_EMPTY_KEY;
  }
  if (at < 0 && room) {  // (every lane with this key tries the slots in the same order)
    for (uint32_t i = 0; i < QM_LOCAL_BUCKET; ++i) {
      const uint32_t x = s + ((i ^ (h >> 3)) & (QM_LOCAL_BUCKET - 1));
      const uint64_t prev = atomicCAS(reinterpret_cast<unsigned long long *>(lkeys + x), QM_EMPTY_KEY, key);
      if (prev == QM_EMPTY_KEY || prev == key) {
        at = (int)x;
        break;
      }
    }
  }
  return at;
}

// ---- accumulator updates ------------------------------------------------------
__device__ __forceinline__ void add128(uint64_t *lo, uint64_t *hi, uint64_t vlo, int64_t vhi) {
  if (vlo != 0) {
    uint64_t old = atomicAdd(reinterpret_cast<unsigned long long *>(lo), (unsigned long long)vlo);
    if (old + vlo < old) vhi += 1;
  }
  if (vhi != 0) atomicAdd(reinterpret_cast<unsigned long long *>(hi), (unsigned long long)vhi);
}

// Compensated atomic add: atomicAdd returns the old value, so the rounding
// error of old + x is recovered exactly (TwoSum) and added, with the
// contribution's own low part xc, to the low word.
__device__ __forceinline__ void fsum_add(uint64_t *hp, uint64_t *lp, double x, double xc) {
  if (x == 0.0 && xc == 0.0) return;
  double old = atomicAdd(reinterpret_cast<double *>(hp), x);
  double s = old + x;
  if (!isfinite(s)) return;
  double bb = s - old;
  double err = (old - (s - bb)) + (x - bb);
  double add = xc + err;
  if (add != 0.0) atomicAdd(reinterpret_cast<double *>(lp), add);
}

// Split summation: x = xh + xl exactly; the high words only ever hold
// multiples of ulp(split) below split in magnitude, so their atomic adds are
// exact in any order and need no returned value.  Non-finite x goes to the
// high word as it is (Infinity / NaN propagate as in the reference's sum).
__device__ __forceinline__ void split_parts(double x, double split, double &xh, double &xl) {
  if (!isfinite(x)) {
    xh = x;
    xl = 0.0;
    return;
  }
  xh = __dsub_rn(__dadd_rn(x, split), split);
  xl = __dsub_rn(x, xh);
}

__device__ __forceinline__ void split_words_add(uint64_t *hp, uint64_t *lp, double xh, double xl) {
  if (xh != 0.0 || isnan(xh)) atomicAdd(reinterpret_cast<double *>(hp), xh);
  if (xl != 0.0) atomicAdd(reinterpret_cast<double *>(lp), xl);
}

__device__ __forceinline__ void split_add(uint64_t *hp, uint64_t *lp, double x, double split) {
  double xh, xl;
  split_parts(x, split, xh, xl);
  split_words_add(hp, lp, xh, xl);
}

__device__ __forceinline__ void two_sum_acc(double &s, double &c, double x) {
  double t = s + x;
  if (isfinite(t)) {
    double bb = t - s;
    c += (s - (t - bb)) + (x - bb);
  }
  s = t;
}

// ---- fixed-point float sums (VF_FIXED) -------------------------------------
// A finite x as round(x / 2^fxe) (ties to even), a 128-bit two's-complement
// integer.  Planning keeps |x| < 2^(fxe + 126), so the value fits; sums of
// these integers are exact and do not depend on the order of the adds.
__device__ __forceinline__ void fx_parts(double x, int fxe, uint64_t &lo, int64_t &hi) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  uint64_t m = b & ((1ULL << 52) - 1);
  int e2 = -1074;  // zero or subnormal: m * 2^-1074
  if (ex != 0) {
    m |= 1ULL << 52;
    e2 = ex - 1075;
  }
  const int sh = e2 - fxe;  // x = m * 2^sh units
  unsigned __int128 v = 0;
  if (m != 0) {
    if (sh >= 0) {
      v = (unsigned __int128)m << sh;
    } else if (sh > -64) {
      const int r = -sh;
      uint64_t q = m >> r;
      const uint64_t rem = m & ((1ULL << r) - 1), half = 1ULL << (r - 1);
      if (rem > half || (rem == half && (q & 1))) q++;
      v = q;
    }
  }
  if (b >> 63) v = (unsigned __int128)0 - v;
  lo = (uint64_t)v;
  hi = (int64_t)(uint64_t)(v >> 64);
}

// One cell of a fixed-point SUM column: its integer value, or its
// non-finite bit (NaN 1, +Infinity 2, -Infinity 4); `stale` when the cell is
// beyond the planned range.
__device__ __forceinline__ void fx_cell(const qm_vcol &vc, double x, uint64_t &lo, int64_t &hi, uint32_t &nf,
                                        bool &stale) {
  lo = 0;
  hi = 0;
  nf = 0;
  if (isnan(x)) {
    nf = 1;
  } else if (isinf(x)) {
    nf = x > 0 ? 2u : 4u;
  } else if (fabs(x) >= vc.fx_max) {
    stale = true;
  } else {
    fx_parts(x, vc.fx_exp, lo, hi);
  }
}

// A fixed-point sum's value: NaN if a NaN or both infinities were seen, else
// the infinity seen, else the integer scaled back (rounded once, to nearest).
__device__ __forceinline__ double i128_to_f64(uint64_t lo, int64_t hi);
__device__ __forceinline__ double fx_value(uint64_t lo, int64_t hi, uint64_t nf, int fxe) {
  if ((nf & 1) || (nf & 6) == 6) return __longlong_as_double(0x7ff8000000000000LL);
  if (nf & 2) return __longlong_as_double(0x7ff0000000000000LL);
  if (nf & 4) return __longlong_as_double((long long)0xfff0000000000000ULL);
  return ldexp(i128_to_f64(lo, hi), fxe);
}

__device__ __forceinline__ uint64_t pick(const uint64_t (&v)[QM_MAX_VCOLS], int i) {
  uint64_t r = 0;
#pragma unroll
  for (int c = 0; c < QM_MAX_VCOLS; ++c)
    if (c == i) r = v[c];
  return r;
}

// Value cell c of a row: a plain register when the kernel knows the column
// count (c is then a compile-time index), else a select over the array.
template <int NV>
__device__ __forceinline__ uint64_t vget(const uint64_t (&vb)[QM_MAX_VCOLS], int c) {
  if constexpr (NV > QM_MAX_VCOLS) return pick(vb, c);
  else return vb[c];
}

// Monotone updates: the word only ever decreases (min) or increases (max),
// so a plain read that already beats the value makes the atomic redundant.
__device__ __forceinline__ void min_u64(uint64_t *p, uint64_t v) {
  if (v < *reinterpret_cast<volatile uint64_t *>(p)) atomicMin(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v);
}
__device__ __forceinline__ void min_i64(uint64_t *p, int64_t v) {
  if (v < (int64_t)*reinterpret_cast<volatile uint64_t *>(p)) atomicMin(reinterpret_cast<long long *>(p), (long long)v);
}
__device__ __forceinline__ void max_i64(uint64_t *p, int64_t v) {
  if (v > (int64_t)*reinterpret_cast<volatile uint64_t *>(p)) atomicMax(reinterpret_cast<long long *>(p), (long long)v);
}
// In the global table the read test costs an L2 round trip that the warp
// waits for; there the atomics go out unconditionally (no returned value, so
// they are fire-and-forget reductions).
__device__ __forceinline__ void upd_min_u64(uint64_t *p, uint64_t v, bool local) {
  if (local) min_u64(p, v);
  else atomicMin(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v);
}
__device__ __forceinline__ void upd_min_i64(uint64_t *p, int64_t v, bool local) {
  if (local) min_i64(p, v);
  else atomicMin(reinterpret_cast<long long *>(p), (long long)v);
}
__device__ __forceinline__ void upd_max_i64(uint64_t *p, int64_t v, bool local) {
  if (local) max_i64(p, v);
  else atomicMax(reinterpret_cast<long long *>(p), (long long)v);
}

// Accumulator word updates, atomic or (plain = the slot is private to the
// calling lane's warp and only one lane writes it) a plain read-modify-write.
__device__ __forceinline__ void acc_add_u64(uint64_t *p, uint64_t v, bool plain) {
  if (plain) *p += v;
  else atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)v);
}
__device__ __forceinline__ void acc_add_f64(uint64_t *p, double v, bool plain) {
  if (plain) *reinterpret_cast<double *>(p) += v;
  else atomicAdd(reinterpret_cast<double *>(p), v);
}
__device__ __forceinline__ void acc_min_u64(uint64_t *p, uint64_t v, bool plain, bool local) {
  if (plain) *p = min(*p, v);
  else upd_min_u64(p, v, local);
}
__device__ __forceinline__ void acc_min_i64(uint64_t *p, int64_t v, bool plain) {
  if (plain) *p = (uint64_t)min((int64_t)*p, v);
  else atomicMin(reinterpret_cast<long long *>(p), (long long)v);
}
__device__ __forceinline__ void acc_max_i64(uint64_t *p, int64_t v, bool plain) {
  if (plain) *p = (uint64_t)max((int64_t)*p, v);
  else atomicMax(reinterpret_cast<long long *>(p), (long long)v);
}
__device__ __forceinline__ void acc_add128(uint64_t *lo, uint64_t *hi, uint64_t vlo, int64_t vhi, bool plain) {
  if (!plain) {
    add128(lo, hi, vlo, vhi);
    return;
  }
  const uint64_t o = *lo, n = o + vlo;
  *lo = n;
  *hi = (uint64_t)((int64_t)*hi + vhi + (n < o ? 1 : 0));
}
__device__ __forceinline__ void acc_fsum(uint64_t *hp, uint64_t *lp, double x, double xc, bool plain) {
  if (!plain) {
    fsum_add(hp, lp, x, xc);
    return;
  }
  if (x == 0.0 && xc == 0.0) return;
  const double old = __longlong_as_double((long long)*hp);
  const double s = old + x;
  *hp = (uint64_t)__double_as_longlong(s);
  if (!isfinite(s)) return;
  const double bb = s - old;
  const double add = xc + ((old - (s - bb)) + (x - bb));
  if (add != 0.0) *reinterpret_cast<double *>(lp) += add;
}

// Butterfly reductions over all 32 lanes (every lane gets the result): the
// peer loops below are O(peers), this is O(log 32) for the common case of a
// whole warp in one group (no GROUP BY, or a dominant key).
template <class T, class OP>
__device__ __forceinline__ T warp_allreduce(T v, OP op) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = op(v, __shfl_xor_sync(QM_FULL, v, o));
  return v;
}

// Reduction of `v` over the calling lane's peer group, for every lane of
// `act` (the lanes executing this; peers is a subset of act).  One loop of
// `iters` steps (the largest group's size - 1) runs in lockstep for all
// groups, so groups do not serialise on divergent loops; a whole-warp group
// takes the butterfly.
template <class T, class OP>
__device__ __forceinline__ T group_reduce(T v, unsigned act, unsigned peers, int lane, int iters, OP op) {
  if (peers == QM_FULL) return warp_allreduce(v, op);
  T r = v;
  unsigned rem = peers & ~(1u << lane);
  for (int it = 0; it < iters; ++it) {
    const int src = rem ? __ffs(rem) - 1 : lane;
    const T x = __shfl_sync(act, v, src);
    if (rem) {
      r = op(r, x);
      rem &= rem - 1;
    }
  }
  return r;
}

// Apply one compacted row (merged with its equal-key peers) to a slot whose
// accumulator word w lives at tp[w * ws].  Every lane of `act` executes this
// (the shuffles need them); only group leaders, with tp != nullptr, write.
// iters = (largest peer group in act) - 1.
// FX: the kernel carries the fixed-point (VF_FIXED) sum paths; kernels
// specialised for a column count and key kind leave them out (their plans
// never use them, and the extra paths cost the hot loop instructions).
template <bool FX = true>
__device__ __forceinline__ void apply_row(const qm_aggspec &A, uint64_t *tp, int ws, bool local, unsigned act,
                                          unsigned peers, int iters, int lane, uint64_t grow,
                                          const uint64_t (&vb)[QM_MAX_VCOLS], uint32_t vnull, bool plain = false,
                                          qm_status *st = nullptr) {
  const bool full = peers == QM_FULL;
  auto umin = [](uint64_t x, uint64_t y) { return min(x, y); };
  auto imin = [](int64_t x, int64_t y) { return min(x, y); };
  auto imax = [](int64_t x, int64_t y) { return max(x, y); };
  auto iadd = [](int64_t x, int64_t y) { return x + y; };
  auto fadd = [](double x, double y) { return x + y; };
  for (int i = 0; i < A.n_accs; ++i) {
    __syncwarp(act);  // the lanes part ways at their probes and at each update: meet again
    const qm_acc ac = A.acc[i];
    uint64_t *w0 = tp ? tp + (int64_t)ac.word * ws : nullptr;
    uint64_t *w1 = tp ? tp + (int64_t)(ac.word + 1) * ws : nullptr;
    if (ac.kind == QA_COUNT) {
      if (tp) acc_add_u64(w0, (uint64_t)__popc(peers), plain);
      continue;
    }
    if (ac.kind == QA_FIRST) {
      const uint64_t first = iters > 0 ? group_reduce(grow, act, peers, lane, iters, umin) : grow;
      if (tp) acc_min_u64(w0, first, plain, local);
      continue;
    }
    const bool valid = !((vnull >> ac.vcol) & 1);
    const uint64_t raw = pick(vb, ac.vcol);
    switch (ac.kind) {
      case QA_NN: {
        const unsigned nn = __popc(__ballot_sync(act, valid) & peers);
        if (tp && nn) acc_add_u64(w0, (uint64_t)nn, plain);
        break;
      }
      case QA_ISUM: {
        const int64_t v = valid ? (int64_t)raw : 0;
        if (!ac.wide) {
          const int64_t s = iters > 0 ? group_reduce(v, act, peers, lane, iters, iadd) : v;
          if (tp && s != 0) {
            if (local || ac.narrow) acc_add_u64(w0, (uint64_t)s, plain);
            else add128(w0, w1, (uint64_t)s, s < 0 ? -1 : 0);
          }
        } else {
          // 128-bit sum of up to 32 int64 cells
          uint64_t lo = (uint64_t)v;
          int64_t hi = v < 0 ? -1 : 0;
          if (full) {
#pragma unroll
            for (int o = 16; o; o >>= 1) {
              const uint64_t xl = __shfl_xor_sync(QM_FULL, lo, o);
              const int64_t xh = __shfl_xor_sync(QM_FULL, hi, o);
              const uint64_t nlo = lo + xl;
              hi += xh + (nlo < lo ? 1 : 0);
              lo = nlo;
            }
          } else {
            unsigned rem = peers & ~(1u << lane);
            for (int it = 0; it < iters; ++it) {
              const int src = rem ? __ffs(rem) - 1 : lane;
              const int64_t x = __shfl_sync(act, v, src);
              if (rem) {
                const uint64_t nlo = lo + (uint64_t)x;
                hi += (x < 0 ? -1 : 0) + (nlo < lo ? 1 : 0);
                lo = nlo;
                rem &= rem - 1;
              }
            }
          }
          if (tp && (lo != 0 || hi != 0)) acc_add128(w0, w1, lo, hi, plain);
        }
        break;
      }
      case QA_FSUM: {
        const double v = valid ? __longlong_as_double((long long)raw) : 0.0;
        const qm_vcol &fv = A.vcol[ac.vcol];
        if (FX && (fv.flags & VF_FIXED)) {
          uint64_t lo;
          int64_t hi;
          uint32_t nf;
          bool stale = false;
          fx_cell(fv, v, lo, hi, nf, stale);
          if (stale && st) set_error(st, QM_DEV_STALE);
          if (full) {
            nf = warp_allreduce(nf, [](uint32_t x, uint32_t y) { return x | y; });
#pragma unroll
            for (int o = 16; o; o >>= 1) {
              const uint64_t xl = __shfl_xor_sync(QM_FULL, lo, o);
              const int64_t xh = __shfl_xor_sync(QM_FULL, hi, o);
              const uint64_t nlo = lo + xl;
              hi += xh + (nlo < lo ? 1 : 0);
              lo = nlo;
            }
          } else {
            const uint64_t lo0 = lo;
            const int64_t hi0 = hi;
            const uint32_t nf0 = nf;
            unsigned rem = peers & ~(1u << lane);
            for (int it = 0; it < iters; ++it) {
              const int src = rem ? __ffs(rem) - 1 : lane;
              const uint64_t xl = __shfl_sync(act, lo0, src);
              const int64_t xh = __shfl_sync(act, hi0, src);
              const uint32_t xn = __shfl_sync(act, nf0, src);
              if (rem) {
                const uint64_t nlo = lo + xl;
                hi += xh + (nlo < lo ? 1 : 0);
                lo = nlo;
                nf |= xn;
                rem &= rem - 1;
              }
            }
          }
          if (tp) {
            if (lo != 0 || hi != 0) acc_add128(w0, w1, lo, hi, plain);
            if (nf) {
              uint64_t *wn = tp + (int64_t)fv.w_nf * ws;
              if (plain) *wn |= nf;
              else atomicOr(reinterpret_cast<unsigned long long *>(wn), (unsigned long long)nf);
            }
          }
          break;
        }
        const double split = fv.split;
        if (split != 0.0) {
          double h, l;
          split_parts(v, split, h, l);
          if (iters > 0) {
            h = group_reduce(h, act, peers, lane, iters, fadd);  // exact: multiples of ulp(split) below split
            l = group_reduce(l, act, peers, lane, iters, fadd);
          }
          if (tp) {
            if (h != 0.0 || isnan(h)) acc_add_f64(w0, h, plain);
            if (l != 0.0) acc_add_f64(w1, l, plain);
          }
          break;
        }
        double s = v, c = 0.0;
        if (full) {
#pragma unroll
          for (int o = 16; o; o >>= 1) {
            const double xs = __shfl_xor_sync(QM_FULL, s, o);
            const double xc = __shfl_xor_sync(QM_FULL, c, o);
            double cc = c + xc;
            two_sum_acc(s, cc, xs);
            c = cc;
          }
        } else {
          unsigned rem = peers & ~(1u << lane);
          for (int it = 0; it < iters; ++it) {
            const int src = rem ? __ffs(rem) - 1 : lane;
            const double x = __shfl_sync(act, v, src);
            if (rem) {
              two_sum_acc(s, c, x);
              rem &= rem - 1;
            }
          }
        }
        if (tp) acc_fsum(w0, w1, s, c, plain);
        break;
      }
      case QA_IMIN:
      case QA_IMAX: {
        const bool mx = ac.kind == QA_IMAX;
        int64_t v = valid ? (int64_t)raw : (mx ? INT64_MIN : INT64_MAX);
        if (iters > 0) v = mx ? group_reduce(v, act, peers, lane, iters, imax) : group_reduce(v, act, peers, lane, iters, imin);
        if (tp && v != (mx ? INT64_MIN : INT64_MAX)) {
          if (mx) acc_max_i64(w0, v, plain);
          else acc_min_i64(w0, v, plain);
        }
        break;
      }
      case QA_FMIN:
      case QA_FMAX: {
        const bool mx = ac.kind == QA_FMAX;
        const double d = __longlong_as_double((long long)raw);
        const bool ok = valid && !isnan(d);  // NaN never wins '<' / '>' (src/partial-agg.ts:80-81)
        int64_t o = ok ? f2ord(d == 0.0 ? 0.0 : d) : (mx ? INT64_MIN : INT64_MAX);
        if (iters > 0) o = mx ? group_reduce(o, act, peers, lane, iters, imax) : group_reduce(o, act, peers, lane, iters, imin);
        if (tp && o != (mx ? INT64_MIN : INT64_MAX)) {
          if (mx) acc_max_i64(w0, o, plain);
          else acc_min_i64(w0, o, plain);
        }
        break;
      }
      case QA_FZERO: {
        const double d = __longlong_as_double((long long)raw);
        const bool z = valid && d == 0.0;
        uint64_t code = z ? ((grow << 1) | (raw >> 63)) : ~0ULL;
        if (__any_sync(act, z) && iters > 0) code = group_reduce(code, act, peers, lane, iters, umin);
        if (tp && code != ~0ULL) acc_min_u64(w0, code, plain, false);
        break;
      }
    }
  }
}

// One row's update of the global slot whose words start at tp: straight
// line per value column, values already gathered into vb (NULL bits in
// vnull) so the cell loads overlap the key lookup.  The atomics return
// nothing (fire-and-forget reductions): a read test of its own would cost an
// L2 round trip that the warp waits for.  But the probe of a hash slot brings
// the words beside its key (h: head, where h.on), and FIRST and the first MIN
// and MAX sit there: their atomics go out only where the row beats the word
// read.  A word only moves one way, so a stale read can cause an unneeded
// atomic, never skip one.
struct slot_head {
  bool on;
  uint64_t w[QM_HEAD_WORDS];
  __device__ __forceinline__ uint64_t word(int i) const { return i == 0 ? w[0] : (i == 1 ? w[1] : w[2]); }
  __device__ __forceinline__ bool above_u(int i, uint64_t v) const { return !on || i >= QM_HEAD_WORDS || v < word(i); }
  __device__ __forceinline__ bool above(int i, int64_t v) const { return !on || i >= QM_HEAD_WORDS || v < (int64_t)word(i); }
  __device__ __forceinline__ bool below(int i, int64_t v) const { return !on || i >= QM_HEAD_WORDS || v > (int64_t)word(i); }
};
struct no_head {  // tables whose lookup reads nothing
  __device__ __forceinline__ bool above_u(int, uint64_t) const { return true; }
  __device__ __forceinline__ bool above(int, int64_t) const { return true; }
  __device__ __forceinline__ bool below(int, int64_t) const { return true; }
};

template <int NV = QM_NV_ANY, int FT = QM_FT_FULL, class HEAD = no_head>
__device__ __forceinline__ void agg_row(const qm_aggspec &A, uint64_t *tp, uint64_t grow,
                                        const uint64_t (&vb)[QM_MAX_VCOLS], uint32_t vnull, const HEAD &h,
                                        qm_status *st = nullptr) {
  atomicAdd(reinterpret_cast<unsigned long long *>(tp + A.w_count), 1ULL);
  if (A.w_first >= 0 && h.above_u(A.w_first, grow))
    atomicMin(reinterpret_cast<unsigned long long *>(tp + A.w_first), (unsigned long long)grow);
  // (run-time plans in a loop: unrolled for every column a plan may have, this
  // and agg_row_local outgrow the instruction cache; 20M rows into 20,000
  // hashed groups, five columns: scan 1.44 -> 1.17 ms)
  constexpr int UNROLL = NV > QM_MAX_VCOLS ? 1 : QM_MAX_VCOLS;
#pragma unroll UNROLL
  for (int c = 0; c < QM_NV_BOUND(NV); ++c) {
    if (NV > QM_MAX_VCOLS && c >= A.n_vcols) break;
    if (FT <= QM_FT_GEN && ((vnull >> c) & 1)) continue;
    const qm_vcol &vc = A.vcol[c];
    const int f = vc.flags;
    if (FT <= QM_FT_GEN && (f & VF_NN)) atomicAdd(reinterpret_cast<unsigned long long *>(tp + vc.w_nn), 1ULL);
    if (FT <= QM_FT_MIX && (vc.dtype == QM_I32 || vc.dtype == QM_I64)) {
      const int64_t v = (int64_t)vget<NV>(vb, c);
      if ((f & VF_SUM) && v != 0) {
        uint64_t *w0 = tp + vc.w_sum;
        if (f & VF_NARROW) atomicAdd(reinterpret_cast<unsigned long long *>(w0), (unsigned long long)v);
        else add128(w0, w0 + 1, (uint64_t)v, v < 0 ? -1 : 0);
      }
      if ((f & VF_MIN) && h.above(vc.w_min, v)) atomicMin(reinterpret_cast<long long *>(tp + vc.w_min), (long long)v);
      if ((f & VF_MAX) && h.below(vc.w_max, v)) atomicMax(reinterpret_cast<long long *>(tp + vc.w_max), (long long)v);
    } else {
      const double d = __longlong_as_double((long long)vget<NV>(vb, c));
      if (FT == QM_FT_SUM || (f & VF_SUM)) {
        uint64_t *w0 = tp + vc.w_sum;
        if (FT == QM_FT_FULL && (f & VF_FIXED)) {
          uint64_t lo;
          int64_t hi;
          uint32_t nf;
          bool stale = false;
          fx_cell(vc, d, lo, hi, nf, stale);
          if (stale && st) set_error(st, QM_DEV_STALE);
          if (lo != 0 || hi != 0) add128(w0, w0 + 1, lo, hi);
          if (nf) atomicOr(reinterpret_cast<unsigned long long *>(tp + vc.w_nf), (unsigned long long)nf);
        } else if (FT >= QM_FT_GEN || vc.split != 0.0) {
          split_add(w0, w0 + 1, d, vc.split);
        } else {
          fsum_add(w0, w0 + 1, d, 0.0);
        }
      }
      if (FT <= QM_FT_MIX) {
        if ((f & (VF_MIN | VF_MAX)) && !isnan(d)) {  // NaN never wins '<' / '>'
          const int64_t o = f2ord(d == 0.0 ? 0.0 : d);
          if ((f & VF_MIN) && h.above(vc.w_min, o)) atomicMin(reinterpret_cast<long long *>(tp + vc.w_min), (long long)o);
          if ((f & VF_MAX) && h.below(vc.w_max, o)) atomicMax(reinterpret_cast<long long *>(tp + vc.w_max), (long long)o);
        }
        if ((f & VF_ZERO) && d == 0.0)
          atomicMin(reinterpret_cast<unsigned long long *>(tp + vc.w_zero),
                    (unsigned long long)((grow << 1) | (vget<NV>(vb, c) >> 63)));
      }
    }
  }
}

// ---- block-local words ---------------------------------------------------------
// Shared memory has native 32-bit atomics only; a 64-bit integer or double
// atomic is a compare-and-swap loop (measured per warp and SM: 18 cycles on
// 4,096 random slots, 24 on 512, 56 on 64, 111 on 16, against 1 for a 32-bit
// add and 4 for two limbs with a carry), and merging equal slots first costs
// more than it saves (__match_any_sync: 53-62 cycles on random slots).  So
// the words of a block-local table that take an add per row are split into
// 32-bit limbs: word w of slot s has its low limb at lw32(w)[s] and its high
// limb at lw32(w)[L + s], where lw32(w) is the word's 8 * L bytes.
//   COUNT, NN       low limb only (a block counts fewer than 2^32 rows)
//   FIRST           low limb: the row within this launch (32-bit in the queue)
//   integer sums    two limbs a 64-bit word, carries passed on
//   split float sum two 64-bit integers in limbs (local_fsum)
//   fixed-point sum 128 bits in limbs
// MIN / MAX / FZERO (read first: most rows change nothing), FNF and the
// doubles of local_doubles stay 64-bit words at
// lw[w * L + s].
// Against 64-bit atomics with equal slots merged through __match_any_sync
// (whole queries, B200): 200M rows into 16 groups 1.23 -> 0.76 ms, 5M rows
// without GROUP BY 0.29 -> 0.17 ms, 100M events into 65,536 groups 0.78 ->
// 0.71 ms.
__device__ __forceinline__ uint32_t *limb(uint64_t *lw, int L, int w, int s) {
  return reinterpret_cast<uint32_t *>(lw + (int64_t)w * L) + s;
}

// p[0] += v (64-bit, limbs p[0] and p[L]); returns the carry out of bit 63.
__device__ __forceinline__ uint32_t limb_add64(uint32_t *p, int L, uint64_t v) {
  const uint32_t v0 = (uint32_t)v;
  uint64_t v1 = v >> 32;
  if (v0) {
    const uint32_t o = atomicAdd(p, v0);
    v1 += (o + v0) < o ? 1 : 0;
  }
  uint32_t carry = (uint32_t)(v1 >> 32);
  const uint32_t h = (uint32_t)v1;
  if (h) {
    const uint32_t o = atomicAdd(p + L, h);
    carry += (o + h) < o ? 1 : 0;
  }
  return carry;
}

// As limb_add64 where the sum is read modulo 2^64 (no carry out).
__device__ __forceinline__ void limb_add64w(uint32_t *p, int L, uint64_t v) {
  // (adding a zero limb costs less than the branch around it)
  const uint32_t v0 = (uint32_t)v;
  const uint32_t o = atomicAdd(p, v0);
  atomicAdd(p + L, (uint32_t)(v >> 32) + ((o + v0) < o ? 1u : 0u));
}

__device__ __forceinline__ void limb_add128(uint32_t *p, int L, uint64_t lo, int64_t hi) {
  hi += (int64_t)limb_add64(p, L, lo);
  if (hi != 0) limb_add64w(p + 2 * L, L, (uint64_t)hi);
}

// A cell of a split column added to its block-local integers.  x + sa rounds
// x to a multiple of ga; the bits of that sum less the bits of sa are the
// multiple itself, an integer below 2^(62 - b) for a table of fewer than
// 2^(b - 1) rows, so the integers of a slot add up without overflow and
// exactly, in any order.  The rest (at most ga / 2) goes to the second
// integer in units of gb the same way; what is left below that (only cells
// smaller than 2^(2b - 73) of the column's bound have any: 2^-17 of it at 100M
// rows, 2^-31 at 1M) is returned for the group's global low word.
// Returns false for a cell outside the planned range (NaN, Infinity, or a
// column rewritten after its statistics): it goes to the global words whole.
__device__ __forceinline__ bool local_fsum(uint32_t *p, int L, const qm_vcol &vc, double x, double &rest) {
  rest = 0.0;
  if (!(fabs(x) < vc.lim)) return false;
  const double ta = __dadd_rn(x, vc.sa);
  const double xb = __dsub_rn(x, __dsub_rn(ta, vc.sa));
  const double tb = __dadd_rn(xb, vc.sb);
  rest = __dsub_rn(xb, __dsub_rn(tb, vc.sb));
  limb_add64w(p, L, (uint64_t)(__double_as_longlong(ta) - __double_as_longlong(vc.sa)));
  limb_add64w(p + 2 * L, L, (uint64_t)(__double_as_longlong(tb) - __double_as_longlong(vc.sb)));
  return true;
}

// One row's update of block-local slot ls (key / special: its group, for the
// rare parts of a float sum that go to the global slot).
template <int NV = QM_NV_ANY, int FT = QM_FT_FULL>
__device__ __forceinline__ void agg_row_local(const qm_scan_args &a, uint64_t *lw, int L, int ls, uint64_t key,
                                              int special, uint32_t row, const uint64_t (&vb)[QM_MAX_VCOLS],
                                              uint32_t vnull) {
  const qm_aggspec &A = a.agg;
  atomicAdd(limb(lw, L, A.w_count, ls), 1u);
  if (A.w_first >= 0) atomicMin(limb(lw, L, A.w_first, ls), row);
  constexpr int UNROLL = NV > QM_MAX_VCOLS ? 1 : QM_MAX_VCOLS;
#pragma unroll UNROLL
  for (int c = 0; c < QM_NV_BOUND(NV); ++c) {
    if (NV > QM_MAX_VCOLS && c >= A.n_vcols) break;
    if (FT <= QM_FT_GEN && ((vnull >> c) & 1)) continue;
    const qm_vcol &vc = A.vcol[c];
    const int f = vc.flags;
    if (FT <= QM_FT_GEN && (f & VF_NN)) atomicAdd(limb(lw, L, vc.w_nn, ls), 1u);
    if (FT <= QM_FT_MIX && (vc.dtype == QM_I32 || vc.dtype == QM_I64)) {
      const int64_t v = (int64_t)vget<NV>(vb, c);
      if (f & VF_SUM) {
        uint32_t *p = limb(lw, L, vc.w_sum, ls);
        if (FT <= QM_FT_GEN && (f & VF_WIDE)) limb_add128(p, L, (uint64_t)v, v < 0 ? -1 : 0);
        else limb_add64w(p, L, (uint64_t)v);
      }
      if (f & VF_MIN) min_i64(lw + (int64_t)vc.w_min * L + ls, v);
      if (f & VF_MAX) max_i64(lw + (int64_t)vc.w_max * L + ls, v);
    } else {
      const double d = __longlong_as_double((long long)vget<NV>(vb, c));
      if (FT == QM_FT_SUM || (f & VF_SUM)) {
        if (FT == QM_FT_FULL && (f & VF_FIXED)) {
          uint64_t lo;
          int64_t hi;
          uint32_t nf;
          bool stale = false;
          fx_cell(vc, d, lo, hi, nf, stale);
          if (stale) set_error(a.status, QM_DEV_STALE);
          limb_add128(limb(lw, L, vc.w_sum, ls), L, lo, hi);
          if (nf) atomicOr(reinterpret_cast<unsigned long long *>(lw + (int64_t)vc.w_nf * L + ls), (unsigned long long)nf);
        } else if (FT >= QM_FT_GEN || vc.lim != 0.0) {
          double rest;
          const bool in = local_fsum(limb(lw, L, vc.w_sum, ls), L, vc, d, rest);
          if (!in || rest != 0.0) {
            const int64_t gs = global_slot(a, key, special);
            if (gs >= 0) {
              uint64_t *w0 = a.table + gs * a.stride + 1 + vc.w_sum;
              if (in) atomicAdd(reinterpret_cast<double *>(w0 + 1), rest);
              else split_add(w0, w0 + 1, d, vc.split);
            }
          }
        }  // (sums kept as doubles: local_doubles)
      }
      if (FT <= QM_FT_MIX) {
        if ((f & (VF_MIN | VF_MAX)) && !isnan(d)) {  // NaN never wins '<' / '>'
          const int64_t o = f2ord(d == 0.0 ? 0.0 : d);
          if (f & VF_MIN) min_i64(lw + (int64_t)vc.w_min * L + ls, o);
          if (f & VF_MAX) max_i64(lw + (int64_t)vc.w_max * L + ls, o);
        }
        if ((f & VF_ZERO) && d == 0.0)
          min_u64(lw + (int64_t)vc.w_zero * L + ls, (((uint64_t)(a.row_offset) + row) << 1) | (vget<NV>(vb, c) >> 63));
      }
    }
  }
}

// The float sums of the warp's rows that the block-local table keeps as two
// doubles a slot (columns without statistics: pushed batches; split columns
// whose cells differ too much in size for integers: wide_cells).  Lane l's row
// goes to slot ls (below 0: none); all lanes call this.  An add to a double in
// shared memory is a compare-and-swap loop, so the lanes of a slot sum theirs
// first (each takes over its next peer's sum, then that one's: five steps at
// most) and the lowest adds once, to its warp's copy where slots have copies.
// 20M rows pushed, half of them kept, SUM and COUNT(*), us of scan against an add
// a row: one group 2,152 -> 204, 16 502 -> 207, 1,000 371 -> 256.
template <int NV = QM_NV_ANY>
__device__ __forceinline__ void local_doubles(const qm_scan_args &a, uint64_t *lw, int L, int ls, int lane,
                                              const uint64_t (&vb)[QM_MAX_VCOLS], uint32_t vnull) {
  const qm_aggspec &A = a.agg;
  const unsigned act = __ballot_sync(QM_FULL, ls >= 0);
  if (ls < 0) return;
  const int slot = ls >> a.local_rep;
  const unsigned peers = __match_any_sync(act, slot);
  const unsigned above = lane == 31 ? 0u : peers & (~0u << (lane + 1));
  const bool lowest = lane == __ffs(peers) - 1;
  const int at = (slot << a.local_rep) | ((int)(threadIdx.x >> 5) & ((1 << a.local_rep) - 1));
#pragma unroll 1
  for (int c = 0; c < QM_NV_BOUND(NV); ++c) {
    if (NV > QM_MAX_VCOLS && c >= A.n_vcols) break;
    const qm_vcol &vc = A.vcol[c];
    if (!(vc.flags & VF_SUM) || (vc.flags & VF_FIXED) || vc.lim != 0.0 || vc.dtype == QM_I32 || vc.dtype == QM_I64) continue;
    double s = (vnull >> c) & 1 ? 0.0 : __longlong_as_double((long long)pick(vb, c)), r = 0.0;
    if (vc.split != 0.0) split_parts(s, vc.split, s, r);
    bool more = above != 0;
    int next = more ? __ffs(above) - 1 : lane;
    while (__any_sync(act, more)) {
      const double s2 = __shfl_sync(act, s, next), r2 = __shfl_sync(act, r, next);
      const int n2 = __shfl_sync(act, next, next);
      if (more) {
        two_sum_acc(s, r, s2);
        r += r2;
      }
      more = more && n2 != next;  // (the last peer's next is itself)
      next = more ? n2 : lane;
    }
    uint64_t *w0 = lw + (int64_t)vc.w_sum * L + at;
    if (lowest) {
      if (vc.split != 0.0) split_words_add(w0, w0 + L, s, r);
      else fsum_add(w0, w0 + L, s, r);
    }
  }
}

// Gather a row's value cells (float32 widened to double, as JS numbers).
template <int NV = QM_NV_ANY, int FT = QM_FT_FULL>
__device__ __forceinline__ void gather_values(const qm_aggspec &A, int64_t row, uint64_t (&vb)[QM_MAX_VCOLS],
                                              uint32_t &vnull) {
  vnull = 0;
#pragma unroll
  for (int c = 0; c < QM_MAX_VCOLS; ++c) {
    vb[c] = 0;
    if (c < QM_NV_BOUND(NV) && (NV <= QM_MAX_VCOLS || c < A.n_vcols)) {
      const qm_vcol &vc = A.vcol[c];
      if (FT <= QM_FT_GEN && cell_null(vc.nulls, row)) vnull |= 1u << c;
      else if (FT <= QM_FT_MIX && (vc.dtype == QM_I32 || vc.dtype == QM_I64)) vb[c] = (uint64_t)ld_int(vc.data, vc.dtype, row);
      else vb[c] = (uint64_t)__double_as_longlong(ld_flt(vc.data, vc.dtype, row));
    }
  }
}

// Merge one block-local slot of a deduplicating plan (words in the global
// table's form, word w at lp[w * L]) into global slot words gp.
__device__ __forceinline__ void merge_raw(const qm_aggspec &A, const uint64_t *lp, int L, uint64_t *gp) {
  for (int i = 0; i < A.n_accs; ++i) {
    const qm_acc ac = A.acc[i];
    const uint64_t v0 = lp[(int64_t)ac.word * L];
    uint64_t *g0 = gp + ac.word, *g1 = gp + ac.word + 1;
    switch (ac.kind) {
      case QA_COUNT:
      case QA_NN:
        if (v0) atomicAdd(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
        break;
      case QA_FIRST:
      case QA_FZERO:
        if (v0 != ~0ULL) atomicMin(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
        break;
      case QA_ISUM:
        if (ac.wide) add128(g0, g1, v0, (int64_t)lp[(int64_t)(ac.word + 1) * L]);
        else if (v0 && ac.narrow) atomicAdd(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
        else if (v0) add128(g0, g1, v0, (int64_t)v0 < 0 ? -1 : 0);
        break;
      case QA_FNF:
        if (v0) atomicOr(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
        break;
      case QA_FSUM:
        if (A.vcol[ac.vcol].flags & VF_FIXED) {
          const uint64_t v1 = lp[(int64_t)(ac.word + 1) * L];
          if (v0 || v1) add128(g0, g1, v0, (int64_t)v1);
        } else if (A.vcol[ac.vcol].split != 0.0) {
          const double h = __longlong_as_double((long long)v0);
          const double l = __longlong_as_double((long long)lp[(int64_t)(ac.word + 1) * L]);
          if (h != 0.0 || isnan(h)) atomicAdd(reinterpret_cast<double *>(g0), h);
          if (l != 0.0) atomicAdd(reinterpret_cast<double *>(g1), l);
        } else {
          fsum_add(g0, g1, __longlong_as_double((long long)v0),
                   __longlong_as_double((long long)lp[(int64_t)(ac.word + 1) * L]));
        }
        break;
      case QA_IMIN:
      case QA_FMIN:
        if ((int64_t)v0 != (int64_t)A.init[ac.word]) atomicMin(reinterpret_cast<long long *>(g0), (long long)v0);
        break;
      case QA_IMAX:
      case QA_FMAX:
        if ((int64_t)v0 != (int64_t)A.init[ac.word]) atomicMax(reinterpret_cast<long long *>(g0), (long long)v0);
        break;
    }
  }
}

// The value of one accumulator of block-local slot s (agg_row_local's words):
// v0, v1 as 64-bit integers (split sums: the two integers; FIRST: the row
// within the launch).
__device__ __forceinline__ void local_load(const qm_aggspec &A, const qm_acc &ac, uint64_t *lw, int L, int s,
                                           uint64_t &v0, uint64_t &v1) {
  const uint32_t *p = limb(lw, L, ac.word, s);
  v1 = 0;
  switch (ac.kind) {
    case QA_COUNT:
    case QA_NN:
    case QA_FIRST: v0 = p[0]; break;
    case QA_ISUM:
    case QA_FSUM:
      if (ac.kind == QA_FSUM && !(A.vcol[ac.vcol].flags & VF_FIXED) && A.vcol[ac.vcol].lim == 0.0) {
        v0 = lw[(int64_t)ac.word * L + s];
        v1 = lw[(int64_t)(ac.word + 1) * L + s];
      } else {
        v0 = p[0] | (uint64_t)p[L] << 32;
        v1 = p[2 * L] | (uint64_t)p[3 * L] << 32;
        if (ac.kind == QA_ISUM && !ac.wide) v1 = 0;
      }
      break;
    default: v0 = lw[(int64_t)ac.word * L + s];
  }
}

// (v0, v1) of another copy of the slot folded into this one's.
__device__ __forceinline__ void local_fold(const qm_aggspec &A, const qm_acc &ac, uint64_t &v0, uint64_t &v1,
                                           uint64_t x0, uint64_t x1) {
  switch (ac.kind) {
    case QA_COUNT:
    case QA_NN: v0 += x0; break;
    case QA_FIRST:
    case QA_FZERO: v0 = min(v0, x0); break;
    case QA_FNF: v0 |= x0; break;
    case QA_IMIN:
    case QA_FMIN: v0 = (uint64_t)min((int64_t)v0, (int64_t)x0); break;
    case QA_IMAX:
    case QA_FMAX: v0 = (uint64_t)max((int64_t)v0, (int64_t)x0); break;
    case QA_ISUM: {
      const uint64_t n = v0 + x0;
      v1 += x1 + (n < v0 ? 1 : 0);
      v0 = n;
      break;
    }
    case QA_FSUM:
      if (A.vcol[ac.vcol].flags & VF_FIXED) {
        const uint64_t n = v0 + x0;
        v1 += x1 + (n < v0 ? 1 : 0);
        v0 = n;
      } else if (A.vcol[ac.vcol].lim != 0.0) {
        v0 += x0;
        v1 += x1;
      } else {
        double s = __longlong_as_double((long long)v0);
        double c = __longlong_as_double((long long)v1) + __longlong_as_double((long long)x1);
        two_sum_acc(s, c, __longlong_as_double((long long)x0));
        v0 = (uint64_t)__double_as_longlong(s);
        v1 = (uint64_t)__double_as_longlong(c);
      }
      break;
  }
}

// A split sum's two integers as the global table's double words: hi the
// multiple of ulp(split) nearest the first, lo the rest.
__device__ __forceinline__ void split_words(const qm_vcol &vc, int64_t ai, int64_t bi, double &hi, double &lo) {
  const int64_t h = (ai + ((int64_t)1 << vc.lsh >> 1)) >> vc.lsh;
  const int64_t r = ai - (h << vc.lsh);
  hi = (double)h * (vc.ga * (double)((int64_t)1 << vc.lsh));  // |h| < 2^53: exact
  lo = (double)r * vc.ga + (double)bi * vc.gb;
}

// One accumulator's value (local_load) into global slot words gp.
__device__ __forceinline__ void merge_value(const qm_aggspec &A, const qm_acc &ac, uint64_t v0, uint64_t v1, uint64_t *gp,
                                            int64_t row_offset) {
  uint64_t *g0 = gp + ac.word, *g1 = gp + ac.word + 1;
  switch (ac.kind) {
    case QA_COUNT:
    case QA_NN:
      if (v0) atomicAdd(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
      break;
    case QA_FIRST:  // an occupied slot has a row
      atomicMin(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)row_offset + (unsigned long long)v0);
      break;
    case QA_FZERO:
      if (v0 != ~0ULL) atomicMin(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
      break;
    case QA_ISUM:
      if (ac.wide) add128(g0, g1, v0, (int64_t)v1);
      else if (v0 && ac.narrow) atomicAdd(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
      else if (v0) add128(g0, g1, v0, (int64_t)v0 < 0 ? -1 : 0);
      break;
    case QA_FNF:
      if (v0) atomicOr(reinterpret_cast<unsigned long long *>(g0), (unsigned long long)v0);
      break;
    case QA_FSUM:
      if (A.vcol[ac.vcol].flags & VF_FIXED) {
        if (v0 || v1) add128(g0, g1, v0, (int64_t)v1);
      } else if (A.vcol[ac.vcol].lim != 0.0) {
        double h, l;
        split_words(A.vcol[ac.vcol], (int64_t)v0, (int64_t)v1, h, l);
        if (h != 0.0) atomicAdd(reinterpret_cast<double *>(g0), h);
        if (l != 0.0) atomicAdd(reinterpret_cast<double *>(g1), l);
      } else {
        const double h = __longlong_as_double((long long)v0), l = __longlong_as_double((long long)v1);
        if (A.vcol[ac.vcol].split != 0.0) split_words_add(g0, g1, h, l);
        else fsum_add(g0, g1, h, l);
      }
      break;
    case QA_IMIN:
    case QA_FMIN:
      if ((int64_t)v0 != (int64_t)A.init[ac.word]) atomicMin(reinterpret_cast<long long *>(g0), (long long)v0);
      break;
    case QA_IMAX:
    case QA_FMAX:
      if ((int64_t)v0 != (int64_t)A.init[ac.word]) atomicMax(reinterpret_cast<long long *>(g0), (long long)v0);
      break;
  }
}

// Block-local slot s (agg_row_local's words) into global slot words gp.
__device__ __forceinline__ void merge_local(const qm_aggspec &A, uint64_t *lw, int L, int s, uint64_t *gp,
                                            int64_t row_offset) {
  for (int i = 0; i < A.n_accs; ++i) {
    const qm_acc ac = A.acc[i];
    uint64_t v0, v1;
    local_load(A, ac, lw, L, s, v0, v1);
    merge_value(A, ac, v0, v1, gp, row_offset);
  }
}

// A whole block's local table into the global table (every thread of the
// block calls this after a barrier).  With copies, the lanes of a copy group
// fold theirs by shuffles first, so the block adds once per slot and word.
__device__ __forceinline__ void merge_block(const qm_scan_args &a, const uint64_t *lkeys, uint64_t *lw) {
  const qm_aggspec &A = a.agg;
  const int L = a.local_slots;
  if (a.dedupe) {
    for (int s = threadIdx.x; s < L; s += blockDim.x) {
      if (lw[(int64_t)A.w_count * L + s] == 0) continue;
      const int64_t gs = a.local_hash ? global_slot(a, lkeys[s], 0) : s;
      if (gs >= 0) merge_raw(A, lw + s, L, a.table + gs * a.stride + 1);
    }
    return;
  }
  if (a.local_rep == 0) {
    for (int s = threadIdx.x; s < L; s += blockDim.x) {
      if (*limb(lw, L, A.w_count, s) == 0) continue;
      const int64_t gs = a.local_hash ? global_slot(a, lkeys[s], 0) : s;
      if (gs >= 0) merge_local(A, lw, L, s, a.table + gs * a.stride + 1, a.row_offset);
    }
    return;
  }
  const int copies = 1 << a.local_rep;
  for (int s0 = threadIdx.x & ~31; s0 < L; s0 += blockDim.x) {  // whole warps: L is a multiple of the copies, not of 32
    const int s = s0 + (threadIdx.x & 31);
    const bool in = s < L;
    unsigned any = __ballot_sync(QM_FULL, in && *limb(lw, L, A.w_count, s) != 0);
    any = (any >> ((threadIdx.x & 31) & ~(copies - 1))) & (copies == 32 ? QM_FULL : (1u << copies) - 1u);
    uint64_t *gp = a.table + (int64_t)(s >> a.local_rep) * a.stride + 1;
    for (int i = 0; i < A.n_accs; ++i) {
      const qm_acc ac = A.acc[i];
      uint64_t v0 = 0, v1 = 0;
      if (in) local_load(A, ac, lw, L, s, v0, v1);
      for (int o = copies >> 1; o; o >>= 1) {
        const uint64_t x0 = __shfl_xor_sync(QM_FULL, v0, o), x1 = __shfl_xor_sync(QM_FULL, v1, o);
        local_fold(A, ac, v0, v1, x0, x1);
      }
      if (any && in && (s & (copies - 1)) == 0) merge_value(A, ac, v0, v1, gp, a.row_offset);
    }
  }
}

// Fold block-local slot words src[w * L] into dst[w * L] (both in this
// block's shared memory, no other writer): the per-warp copies of a private
// table collapse into one before the global merge.
__device__ __forceinline__ void merge_plain(const qm_aggspec &A, uint64_t *dst, const uint64_t *src, int L) {
  for (int i = 0; i < A.n_accs; ++i) {
    const qm_acc ac = A.acc[i];
    const int64_t w0 = (int64_t)ac.word * L, w1 = (int64_t)(ac.word + 1) * L;
    switch (ac.kind) {
      case QA_COUNT:
      case QA_NN: dst[w0] += src[w0]; break;
      case QA_FIRST:
      case QA_FZERO: dst[w0] = min(dst[w0], src[w0]); break;
      case QA_ISUM:
        if (ac.wide) acc_add128(dst + w0, dst + w1, src[w0], (int64_t)src[w1], true);
        else dst[w0] += src[w0];
        break;
      case QA_FNF: dst[w0] |= src[w0]; break;
      case QA_FSUM:
        if (A.vcol[ac.vcol].flags & VF_FIXED) {
          acc_add128(dst + w0, dst + w1, src[w0], (int64_t)src[w1], true);
        } else if (A.vcol[ac.vcol].split != 0.0) {
          acc_add_f64(dst + w0, __longlong_as_double((long long)src[w0]), true);
          acc_add_f64(dst + w1, __longlong_as_double((long long)src[w1]), true);
        } else {
          acc_fsum(dst + w0, dst + w1, __longlong_as_double((long long)src[w0]),
                   __longlong_as_double((long long)src[w1]), true);
        }
        break;
      case QA_IMIN:
      case QA_FMIN: acc_min_i64(dst + w0, (int64_t)src[w0], true); break;
      case QA_IMAX:
      case QA_FMAX: acc_max_i64(dst + w0, (int64_t)src[w0], true); break;
    }
  }
}

// Applies one survivor per lane (key word, special flag, row within the
// launch and gathered cells; lanes with active = false sit out) to the
// block-local table or else the global table.  Returns whether the row found
// a slot of a hashed block-local table.
template <int DD = 2, int NV = QM_NV_ANY, int FT = QM_FT_FULL, int LM = QM_LM_ANY>
__device__ __forceinline__ bool drain_apply(const qm_scan_args &a, uint64_t *lkeys, uint64_t *lw, int L, int lane,
                                            bool active, uint64_t key, int special, uint32_t row,
                                            const uint64_t (&vb)[QM_MAX_VCOLS], uint32_t vnull) {
  const qm_aggspec &A = a.agg;
  if (DD == 2 ? a.dedupe != 0 : DD == 1) {
    const unsigned act = __ballot_sync(QM_FULL, active);
    if (!active) return false;
    unsigned peers = __match_any_sync(act, key);
    if (__any_sync(act, special != 0)) peers &= __match_any_sync(act, special);
    const bool leader = lane == __ffs(peers) - 1;
    uint64_t *tp = nullptr;
    int ws = 1;
    bool local = false;
    if (leader) {
      int ls = -1;
      if (L > 0) {
        if (!a.local_hash) ls = (int)global_slot(a, key, special);
        else if (special == 0) ls = local_find(lkeys, L, key);
      }
      if (ls >= 0) {
        tp = lw + ls;
        ws = L;
        local = true;
      } else if (!(L > 0 && !a.local_hash)) {
        const int64_t gs = global_slot(a, key, special);
        if (gs >= 0) tp = a.table + gs * a.stride + 1;
      }
    }
    const int iters = (int)__reduce_max_sync(act, (unsigned)__popc(peers)) - 1;
    apply_row<FT == QM_FT_FULL>(A, tp, ws, local, act, peers, iters, lane, (uint64_t)a.row_offset + row, vb, vnull,
                                local && a.priv, FT == QM_FT_FULL ? a.status : nullptr);
    return false;
  }
  int ls = -1;
  if (LM == QM_LM_DIRECT) {
    if (active) {
      const int64_t s = global_slot(a, key, special);
      if (s >= 0) {
        ls = ((int)s << a.local_rep) | (lane & ((1 << a.local_rep) - 1));
        agg_row_local<NV, FT>(a, lw, L, ls, key, special, row, vb, vnull);
      }
    }
    __syncwarp();
    if (FT <= QM_FT_DBL && a.doubles) local_doubles<NV>(a, lw, L, ls, lane, vb, vnull);
    return false;
  }
  bool global = active;
  if (L > 0 && active) {
    if (LM != QM_LM_HASH && !a.local_hash) {
      const int64_t s = global_slot(a, key, special);
      global = false;
      if (s >= 0) ls = ((int)s << a.local_rep) | (lane & ((1 << a.local_rep) - 1));
    } else if (special == 0) {
      ls = local_find(lkeys, L, key);
      global = ls < 0;
    }
  }
  // the lanes leave the probe loops at different steps: meet again before the
  // updates, or each lane walks them alone
  __syncwarp();
  if (ls >= 0) agg_row_local<NV, FT>(a, lw, L, ls, key, special, row, vb, vnull);
  __syncwarp();
  if (FT <= QM_FT_DBL && a.doubles) {
    local_doubles<NV>(a, lw, L, ls, lane, vb, vnull);
    __syncwarp();
  }
  int64_t gs = -1;
  if constexpr (LM == QM_LM_HASH) {
    slot_head h;
    h.on = special == 0;
    if (global) gs = h.on ? global_find_head(a, key, h.w) : a.n_slots + special - 1;
    __syncwarp();
    if (gs >= 0)
      agg_row<NV, FT>(A, a.table + gs * a.stride + 1, (uint64_t)a.row_offset + row, vb, vnull, h,
                      FT == QM_FT_FULL ? a.status : nullptr);
  } else {
    if (global) gs = global_slot(a, key, special);
    __syncwarp();
    if (gs >= 0)
      agg_row<NV, FT>(A, a.table + gs * a.stride + 1, (uint64_t)a.row_offset + row, vb, vnull, no_head(),
                      FT == QM_FT_FULL ? a.status : nullptr);
  }
  return ls >= 0;
}

// Aggregates one survivor per lane (lanes with active = false sit out):
// gathers its key and value cells, then drain_apply.
// DD: 0 / 1 = the plan's dedupe flag fixed at compile time (separate kernels
// keep each path's registers and code apart), 2 = read it from the plan.
template <int DD = 2, int NV = QM_NV_ANY, int KK = QM_KK_ANY, int FT = QM_FT_FULL, int LM = QM_LM_ANY>
__device__ __forceinline__ bool drain_round_any(const qm_scan_args &a, uint64_t *lkeys, uint64_t *lw, int L,
                                                int lane, bool active, int64_t row) {
  uint64_t key = 0;
  int special = 0;
  uint64_t vb[QM_MAX_VCOLS];
  uint32_t vnull = 0;
  if (active) {
    key = row_key<KK>(a.key, row, special);
    gather_values<NV, FT>(a.agg, row, vb, vnull);
  }
  return drain_apply<DD, NV, FT, LM>(a, lkeys, lw, L, lane, active, key, special, (uint32_t)row, vb, vnull);
}


// D survivors per lane at once (act: this lane has a d-th one) of a plan whose
// rows all have block-local slots: the cells of all D are gathered before any
// is used.
template <int NV, int KK, int FT, int D>
__device__ __forceinline__ void drain_rows(const qm_scan_args &a, uint64_t *lw, int L, int lane, const uint32_t (&row)[D],
                                           const bool (&act)[D]) {
  uint64_t key[D];
  int special[D];
  uint64_t vb[D][QM_MAX_VCOLS];
  uint32_t vnull[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    key[d] = 0;
    special[d] = 0;
    vnull[d] = 0;
    if (act[d]) {
      key[d] = row_key<KK>(a.key, row[d], special[d]);
      gather_values<NV, FT>(a.agg, row[d], vb[d], vnull[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < D; ++d) {
    if (act[d]) {
      const int64_t s = global_slot(a, key[d], special[d]);
      if (s >= 0)
        agg_row_local<NV, FT>(a, lw, L, ((int)s << a.local_rep) | (lane & ((1 << a.local_rep) - 1)), key[d], special[d],
                              row[d], vb[d], vnull[d]);
    }
    __syncwarp();
  }
}

// Number(bigint): round to nearest, ties to even.
__device__ __forceinline__ double i128_to_f64(uint64_t lo, int64_t hi) {
  const bool neg = hi < 0;
  if (neg) {  // negate the 128-bit value
    lo = ~lo + 1;
    hi = ~hi + (lo == 0 ? 1 : 0);
  }
  const uint64_t uhi = (uint64_t)hi;
  double r;
  if (uhi == 0) {
    r = __ull2double_rn(lo);
  } else {
    const int shift = 64 - __clzll((long long)uhi);  // drop `shift` bits
    const uint64_t top = (uhi << (64 - shift)) | (lo >> shift);
    const bool sticky = (lo << (64 - shift)) != 0;
    uint64_t keep = top >> 11;
    const uint64_t rem = top & 0x7ff;
    const bool guard = (rem >> 10) & 1;
    const bool st = sticky || (rem & 0x3ff);
    if (guard && (st || (keep & 1))) keep++;
    r = ldexp((double)keep, shift + 11);
  }
  return neg ? -r : r;
}

__device__ __forceinline__ void set_null(unsigned char *out, int64_t null_offset, int64_t i) {
  atomicOr(reinterpret_cast<unsigned *>(out + null_offset) + (i >> 5), 1u << (i & 31));
}

// Finalize slot `s` of a group table into output row `i` (keys, then each
// aggregate; NULL bits in the output's word bitmaps).
// BYTES: NULL flags go to one byte per output row at nullbytes + nboff[k]
// (every nullable output writes 0 or 1, so no clearing is needed);
// otherwise set bits in the word bitmap at out + null_offset.
// A NULL output cell: its flag, and zero in the data cell (the output
// buffer is not cleared beforehand).
__device__ __forceinline__ void zero_cell(unsigned char *col, int dtype, int64_t i) {
  if (dtype == QM_I32 || dtype == QM_F32) {
    reinterpret_cast<uint32_t *>(col)[i] = 0;
  } else if (dtype == QM_I128) {
    reinterpret_cast<uint64_t *>(col)[2 * i] = 0;
    reinterpret_cast<uint64_t *>(col)[2 * i + 1] = 0;
  } else {
    reinterpret_cast<uint64_t *>(col)[i] = 0;
  }
}
#define NULL_OUT()                                  \
  do {                                              \
    if (BYTES) nullbytes[nboff[k] + i] = 1;         \
    else set_null(out, o.null_offset, i);           \
    zero_cell(col, o.dtype, i);                     \
  } while (0)
template <bool BYTES>
__device__ __forceinline__ void emit_group(const uint64_t *t, int stride, uint64_t s, int64_t i, const qm_keyspec &K,
                                           int64_t n_slots, const qm_outspec &O, unsigned char *out,
                                           unsigned char *nullbytes, const int64_t *nboff) {
  const uint64_t *w = t + s * stride + 1;
  // reconstruct the key word
  bool knull = false;
  uint64_t key = 0;
  if (K.mode == QK_DIRECT) {
    if ((int64_t)s == n_slots) knull = true;
    else key = (uint64_t)K.base + s;
  } else if (K.mode == QK_HASH) {
    if ((int64_t)s == n_slots) key = QM_EMPTY_KEY;
    else if ((int64_t)s == n_slots + 1) knull = true;
    else key = t[s * stride];
  }
  for (int k = 0; k < O.n_out; ++k) {
    const qm_out &o = O.o[k];
    unsigned char *col = out + o.offset;
    if (BYTES && nboff[k] >= 0) nullbytes[nboff[k] + i] = 0;
    if (o.kind == QO_KEY) {
      if (knull) {
        NULL_OUT();
        continue;
      }
      if (K.pack == QP_CONCAT) {
        reinterpret_cast<int32_t *>(col)[i] = (int32_t)(o.src == 0 ? (key >> 32) : key);
      } else if (K.pack == QP_DIGITS) {
        const int c = o.src;
        const uint64_t d = (key / K.kmul[c]) % K.kradix[c];
        if (K.knullable[c] && d == 0) {
          NULL_OUT();
          continue;
        }
        const int64_t v = K.kbase[c] + (int64_t)(d - (uint64_t)K.knullable[c]);
        if (o.dtype == QM_I32) reinterpret_cast<int32_t *>(col)[i] = (int32_t)v;
        else reinterpret_cast<int64_t *>(col)[i] = v;
      } else if (o.dtype == QM_I32) {
        reinterpret_cast<int32_t *>(col)[i] = (int32_t)(int64_t)key;
      } else {
        reinterpret_cast<uint64_t *>(col)[i] = key;
      }
      continue;
    }
    if (o.kind == QO_COUNT) {
      reinterpret_cast<int64_t *>(col)[i] = (int64_t)w[o.word];
      continue;
    }
    const uint64_t nn = w[o.nn_word];
    if (nn == 0) {
      NULL_OUT();
      continue;
    }
    switch (o.kind) {
      case QO_SUM_F:
      case QO_AVG_F: {
        double s2 = o.fixed ? fx_value(w[o.word], (int64_t)w[o.word + 1], w[o.nf_word], o.fx_exp)
                            : __longlong_as_double((long long)w[o.word]) + __longlong_as_double((long long)w[o.word + 1]);
        reinterpret_cast<double *>(col)[i] = o.kind == QO_SUM_F ? s2 : s2 / (double)nn;
        break;
      }
      case QO_SUM_I2F:
      case QO_AVG_I2F: {
        const int64_t hi = o.narrow ? ((int64_t)w[o.word] >> 63) : (int64_t)w[o.word + 1];
        double s2 = i128_to_f64(w[o.word], hi);
        reinterpret_cast<double *>(col)[i] = o.kind == QO_SUM_I2F ? s2 : s2 / (double)nn;
        break;
      }
      case QO_SUM_I128:
        reinterpret_cast<uint64_t *>(col)[2 * i] = w[o.word];
        reinterpret_cast<uint64_t *>(col)[2 * i + 1] = w[o.word + 1];
        break;
      case QO_AVG_BIG: {
        // bigAvg(bigSum, 0, count): Number(sum / n) + Number(sum % n) / n
        const __int128 sum = (__int128)(((unsigned __int128)(uint64_t)w[o.word + 1] << 64) | w[o.word]);
        const __int128 q = sum / (__int128)nn, r = sum % (__int128)nn;
        const double qd = i128_to_f64((uint64_t)q, (int64_t)(q >> 64));
        const double rd = i128_to_f64((uint64_t)r, (int64_t)(r >> 64));
        reinterpret_cast<double *>(col)[i] = qd + (rd + 0.0) / (double)nn;
        break;
      }
      case QO_MIN_I:
      case QO_MAX_I:
        if (o.dtype == QM_I32) reinterpret_cast<int32_t *>(col)[i] = (int32_t)(int64_t)w[o.word];
        else reinterpret_cast<int64_t *>(col)[i] = (int64_t)w[o.word];
        break;
      case QO_MIN_F:
      case QO_MAX_F: {
        const int64_t ov = (int64_t)w[o.word];
        double d = ord2f(ov);
        // a zero result takes the sign of the first zero seen (strict
        // '<' / '>' keep the first of -0 and 0, src/partial-agg.ts:80-81)
        if (ov == 0 && o.zero_word >= 0 && w[o.zero_word] != ~0ULL && (w[o.zero_word] & 1)) d = -0.0;
        reinterpret_cast<double *>(col)[i] = d;
        break;
      }
    }
  }
}

#undef NULL_OUT

__device__ __forceinline__ void emit_group_bytes(const uint64_t *t, int stride, uint64_t s, int64_t i,
                                                 const qm_keyspec &K, int64_t n_slots, const qm_outspec &O,
                                                 unsigned char *out, unsigned char *nullbytes, const int64_t *nboff) {
  emit_group<true>(t, stride, s, i, K, n_slots, O, out, nullbytes, nboff);
}

}  // namespace qm
