/* nml_types.h -- TEST INFRASTRUCTURE ONLY.
 *
 * The types of the nml interface that eigensolve_lanczos's signature and the
 * drop-in use, for machines without a NEMO-3D tree: scalars are double, a
 * complex scalar is a pair (r, i), a vector is a pointer to its first element,
 * a matrix an array of row pointers, an extent a size_t.  Where the tree is
 * present the recipe compiles against its own headers instead.
 */
#ifndef TBGPU_STANDIN_NML_TYPES_H
#define TBGPU_STANDIN_NML_TYPES_H

#include <stddef.h>

typedef size_t nml_extent;
typedef double nml_dscalar;
typedef nml_dscalar nml_dvector;
typedef struct {
  double r, i;
} nml_dcscalar;
typedef nml_dcscalar nml_dcvector;
typedef nml_dcscalar *nml_dcmatrix;

nml_dvector *nml_dv_new(nml_extent n);
nml_dcvector *nml_dcv_new(nml_extent n);
nml_dcmatrix *nml_dcm_new(nml_extent m, nml_extent n);

#endif
