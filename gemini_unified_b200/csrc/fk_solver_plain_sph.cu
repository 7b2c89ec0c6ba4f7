// FK solver, parity build, spheroidal phase (see fk_solver_plain.cu).
#define GEM_NS gem_plain
#define GEM_FAST 0
#define GEM_PHASE 1
#include "fk_solver_tu.cuh"
