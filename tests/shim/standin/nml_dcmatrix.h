/* TEST INFRASTRUCTURE ONLY: see nml_types.h */
#include "nml_types.h"
