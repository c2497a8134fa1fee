/* measure.h -- all qubits of a small state measured in one launch. */
#ifndef QCS_MEASURE_H
#define QCS_MEASURE_H

#include "../../include/qcs_cuda.h"

#ifdef __cplusplus
extern "C" {
#endif

/* What qcs_cuda_measure of qubits 0 .. n-1 in turn does, with one draw each.
 * QCS_CUDA_EUNSUP, and nothing done, for a state of more than 128 KB. */
int qcs_measure_all(qcs_cuda_state *s, const double *random_vals, int *outcomes);

#ifdef __cplusplus
}
#endif
#endif
