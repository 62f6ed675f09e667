// One matrix-vector product of a sparse two-site plan in one call: psi panels, L.psi, the
// sparse product of both MPO sites, .R and the sum over operators (top1 .. top4 of HVecQt,
// source/mpo_dmrg_kernelQt.py:301-316), launched back to back.
//
// Bound at small bonds: the launches.  K=6, D=16 keeps the device busy for 19 us; six calls
// from Python with their stream and pointer look-ups took 51 us, this one 25 us (split TF32 at a
// like size: 73 and 33 us).
#include <cuda_runtime.h>
#include "qc_types.h"
#include "../../include/qcmpodmrg_b200.h"

__attribute__((visibility("hidden"))) int qc_internal_reduce(const void *part, int f32, int nops, long long n,
                                                             double *out, cudaStream_t s);

extern "C" int qc_sigma_panels(const qc_sigma_plan *p, const void *lpan, const void *rpan, const double *x,
                               void *psi, void *t1, void *t3, void *part, double *y, void *stream) {
  if (!p || !x || !psi || !t1 || !t3 || !part || !y) return QC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const bool f32 = p->f32 != 0, split = p->f32 == 2;
  int rc = split ? qc_gather_split_f32(x, p->psi_idx, p->npsi, (float *)psi, (float *)psi + p->npsi, stream)
           : f32 ? qc_gather_pad_f32(x, p->psi_idx, p->npsi, (float *)psi, stream)
               : qc_gather_pad_f64(x, p->psi_idx, p->npsi, (double *)psi, stream);
  if (rc != QC_OK) return rc;
  const qc_sigma_panel &a = p->first, &b = p->last;
  rc = split ? qc_tcpanel_seg_f32(a.units, a.nwork, lpan, a.ops, a.table, (float *)t1, stream)
       : f32 ? qc_dpanel_f32(a.units, a.work, a.nwork, a.ops, nullptr, a.table, (const float *)lpan,
                           (const float *)psi, (float *)t1, stream)
           : qc_dpanel_f64(a.units, a.work, a.nwork, a.ops, nullptr, a.table, (const double *)lpan,
                           (const double *)psi, (double *)t1, stream);
  for (int i = 0; i < 3 && rc == QC_OK; ++i) {
    const qc_sigma_tiles &w = p->tiles[i];
    if (w.n <= 0) continue;
    rc = f32 ? qc_wsparse_f32(w.items, w.n, w.tile, p->deltas, p->groups, p->rows, p->dops, p->octs, p->ent_w,
                              p->ent_r, p->wops, w.maxr, w.maxo, (const float *)t1, (float *)t3, stream)
             : qc_wsparse_f64(w.items, w.n, w.tile, p->deltas, p->groups, p->rows, p->dops, p->octs, p->ent_w,
                              p->ent_r, p->wops, w.maxr, w.maxo, (const double *)t1, (double *)t3, stream);
  }
  if (rc != QC_OK) return rc;
  // partial vectors that .R writes only in part
  if (p->clear && cudaMemsetAsync(part, 0, (size_t)p->nops * p->ndim * (f32 ? 4 : 8), s) != cudaSuccess)
    return QC_ERR_CUDA;
  rc = split ? qc_tcpanel_f32(b.units, b.nwork, rpan, b.ops, (const long long *)b.table, (float *)part, stream)
       : f32 ? qc_dpanel_f32(b.units, b.work, b.nwork, b.ops, (const long long *)b.table, nullptr, (const float *)t3,
                           (const float *)rpan, (float *)part, stream)
           : qc_dpanel_f64(b.units, b.work, b.nwork, b.ops, (const long long *)b.table, nullptr, (const double *)t3,
                           (const double *)rpan, (double *)part, stream);
  return rc == QC_OK ? qc_internal_reduce(part, f32, p->nops, p->ndim, y, s) : rc;
}
