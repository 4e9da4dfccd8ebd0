/* lanczos.h -- TEST INFRASTRUCTURE ONLY.
 *
 * The entry point that the drop-in defines (eigen/include/lanczos.h:365-391 of
 * the reference declares it; its argument list is the drop-in's interface),
 * for machines without a NEMO-3D tree.
 */
#ifndef TBGPU_STANDIN_LANCZOS_H
#define TBGPU_STANDIN_LANCZOS_H

#include "nml_types.h"

int eigensolve_lanczos(nml_dvector **values, int check_start, int check_every, int iterations_max,
                       int wanted1, int wanted2, nml_extent length, int *argument[],
                       nml_dscalar low1, nml_dscalar high1, nml_dscalar low2, nml_dscalar high2,
                       nml_dscalar tolerance, int verbose, const char *trace_file,
                       const char *tridiagonal_file, const char *eigenvalue_file,
                       nml_dcvector *r, const nml_dcvector *start, nml_dcvector *q,
                       nml_dcvector *q_before, nml_dcvector **complex_values,
                       nml_dcmatrix **vectors,
                       void (*product)(const int **, nml_dcscalar *, const nml_dcscalar *),
                       int restore);

#endif
