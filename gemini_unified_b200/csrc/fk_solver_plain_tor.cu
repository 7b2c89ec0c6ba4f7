// FK solver, parity build, toroidal phase (see fk_solver_plain.cu).
#define GEM_NS gem_plain
#define GEM_FAST 0
#define GEM_PHASE 0
#include "fk_solver_tu.cuh"
