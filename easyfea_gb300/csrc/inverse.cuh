// Host interface of the coarse matrix's inverse (inverse.cu).
#pragma once

#include "pcg_types.cuh"

namespace gfea {

// C.Ac (nc x nc, SPD) regularised -- a diagonal entry at most zero_tol times
// the largest is replaced by it, the others shifted by 'shift' times it --
// and inverted in place on st: a launch per 16 unknowns, none of which waits on
// another CTA.
int coarse_inverse(const CoarseDev& C, double zero_tol, double shift, cudaStream_t st);

}  // namespace gfea
