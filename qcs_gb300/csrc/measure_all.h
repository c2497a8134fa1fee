/* measure_all.h -- measurement of all qubits in one launch (readout.cu), for the
 * qc_* layer (host/qcs_api.c).  Not exported from the library. */
#ifndef QCS_MEASURE_ALL_H
#define QCS_MEASURE_ALL_H

#include "qcs_cuda.h"

#ifdef __cplusplus
extern "C" {
#endif

/* What qcs_cuda_measure of qubits 0 .. n-1 in turn does, with one draw each.
 * QCS_CUDA_EUNSUP, and nothing done, for a state of more than 128 KB. */
__attribute__((visibility("hidden"))) int
qcs_measure_all(qcs_cuda_state *s, const double *random_vals, int *outcomes);

#ifdef __cplusplus
}
#endif

#endif
