// Cluster multi-shift CG: a whole small solve in one launch.
#pragma once
#include <cuda_runtime.h>

#include "msolve_mk.h"
#include "solver_core.cuh"

namespace polar {

// Bytes of the graph's row order, places and neighbour lists for a cluster solve, and their
// pointers inside the workspace.
size_t cl_graph_bytes(const polar_graph* g, int nA);
size_t cl_graph_layout(const polar_graph* g, int nA, char* base, ClGraph* C);

// True when the cluster kernel is the faster one for a solve of this shape (ld: the padded R)
// and this thread may take it.
bool cl_takes(const polar_graph* g, int precision, int R, int ld, int p, int nA);

// Runs a whole solve (blocking).
template <typename T>
int cl_solve_one(const SolvePrm<T>& P, cudaStream_t st, MkResult* out);

}  // namespace polar
