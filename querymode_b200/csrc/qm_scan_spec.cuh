// qm_scan_spec.cuh — instantiations of the scan kernel for one value-column
// count (QM_SPEC_NV, defined by the including qm_scan_nv*.cu): the plans the
// planner produces by key kind, value features and row placement, plus their
// shared-memory attribute setter and launcher.
#include "qm_scan.cuh"

#define QM_PASTE2(a, b) a##b
#define QM_PASTE(a, b) QM_PASTE2(a, b)
#define QM_SPEC_FN(x) QM_PASTE(QM_PASTE(qm_scan_nv, QM_SPEC_NV), x)

// (dedupe, key kind, features, placement), narrowest first: a launch takes
// the first entry that covers its plan.  Deduplication is a launch-shape
// knob, so its kernel exists for any key only; without value columns there is
// nothing for the features to leave out.
#if QM_SPEC_NV > 0 && QM_SPEC_NV <= 2
#define QM_SPEC_SUM(X)                                                                                              \
  X(0, QM_KK_I64, QM_FT_SUM, QM_LM_DIRECT) X(0, QM_KK_I32, QM_FT_SUM, QM_LM_DIRECT)                                 \
  X(0, QM_KK_I64, QM_FT_SUM, QM_LM_HASH) X(0, QM_KK_I64, QM_FT_SUM, QM_LM_ANY) X(0, QM_KK_I32, QM_FT_SUM, QM_LM_ANY)
#else
#define QM_SPEC_SUM(X)
#endif
#define QM_SPEC_MIX(X)                                                                                              \
  X(0, QM_KK_I64, QM_FT_MIX, QM_LM_DIRECT) X(0, QM_KK_I32, QM_FT_MIX, QM_LM_DIRECT)                                 \
  X(0, QM_KK_NONE, QM_FT_MIX, QM_LM_DIRECT) X(0, QM_KK_ANY, QM_FT_MIX, QM_LM_DIRECT)                                \
  X(0, QM_KK_I64, QM_FT_MIX, QM_LM_HASH) X(0, QM_KK_ANY, QM_FT_MIX, QM_LM_HASH)                                     \
  X(0, QM_KK_I64, QM_FT_MIX, QM_LM_ANY) X(0, QM_KK_I32, QM_FT_MIX, QM_LM_ANY)
#if QM_SPEC_NV > 0
#define QM_SPEC_GEN(X)                                                                                              \
  X(0, QM_KK_NONE, QM_FT_GEN, QM_LM_DIRECT)                                                                         \
  X(0, QM_KK_I64, QM_FT_GEN, QM_LM_HASH) X(0, QM_KK_ANY, QM_FT_GEN, QM_LM_HASH)                                     \
  X(0, QM_KK_I64, QM_FT_GEN, QM_LM_ANY) X(0, QM_KK_I32, QM_FT_GEN, QM_LM_ANY) X(0, QM_KK_ANY, QM_FT_GEN, QM_LM_ANY) \
  X(0, QM_KK_NONE, QM_FT_DBL, QM_LM_DIRECT)                                                                         \
  X(0, QM_KK_I64, QM_FT_DBL, QM_LM_HASH) X(0, QM_KK_ANY, QM_FT_DBL, QM_LM_HASH) X(0, QM_KK_I64, QM_FT_DBL, QM_LM_ANY) \
  X(0, QM_KK_I32, QM_FT_DBL, QM_LM_ANY) X(0, QM_KK_ANY, QM_FT_DBL, QM_LM_ANY) X(1, QM_KK_ANY, QM_FT_DBL, QM_LM_ANY)
#else
#define QM_SPEC_GEN(X) X(0, QM_KK_ANY, QM_FT_GEN, QM_LM_ANY) X(1, QM_KK_ANY, QM_FT_GEN, QM_LM_ANY)
#endif
#define QM_SPEC_LIST(X) QM_SPEC_SUM(X) QM_SPEC_MIX(X) QM_SPEC_GEN(X)

cudaError_t QM_SPEC_FN(_attr)(int max_smem) {
  using namespace qm;
  cudaError_t e = cudaSuccess;
#define QM_ATTR_(DD, KK, FT, LM)                                                                    \
  if (e == cudaSuccess)                                                                             \
    e = cudaFuncSetAttribute(qm_scan_kernel<false, false, DD, QM_SPEC_NV, KK, FT, LM>,              \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  QM_SPEC_LIST(QM_ATTR_)
#undef QM_ATTR_
  return e;
}

cudaError_t QM_SPEC_FN(_launch)(const qm_scan_args &a, int dd, int kk, int ft, int lm, int blocks, size_t smem,
                                cudaStream_t st, int *per_sm) {
  using namespace qm;
#define QM_LAUNCH_(DD, KK, FT, LM)                                                                              \
  if (dd == DD && (kk == KK || KK == QM_KK_ANY) && ft >= FT && (lm == LM || LM == QM_LM_ANY)) {                 \
    return launch_scan_kernel(qm_scan_kernel<false, false, DD, QM_SPEC_NV, KK, FT, LM>, a, blocks, smem, st,     \
                              per_sm);                                                                          \
  }
  QM_SPEC_LIST(QM_LAUNCH_)
#undef QM_LAUNCH_
  return cudaErrorInvalidValue;
}
