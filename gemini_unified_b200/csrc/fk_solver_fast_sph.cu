// FK solver, fast build, spheroidal phase (see fk_solver_fast.cu).
#define GEM_NS gem_fast
#define GEM_FAST 1
#define GEM_PHASE 1
#include "fk_solver_tu.cuh"
