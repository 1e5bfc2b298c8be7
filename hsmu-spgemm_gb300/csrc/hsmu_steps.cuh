// Positions of walks that read several strides ahead.  CSR positions go up to
// INT_MAX, so a position plus the strides ahead of it does not fit int; as
// unsigned it does (the strides of a round are a few thousand), and the
// comparison with the end costs no more.
#pragma once

#ifdef __CUDACC__
#define HSMU_STEP_FN __host__ __device__ __forceinline__
#else
#define HSMU_STEP_FN inline
#endif

namespace hsmu {

typedef unsigned StepPos;  // a position of a walk: for (StepPos p = first; step_in(p, 0, end); p += strides)

// whether p + off lies below the end (p: at most INT_MAX and one round)
HSMU_STEP_FN bool step_in(StepPos p, int off, int end) { return p + (unsigned)off < (unsigned)end; }

}  // namespace hsmu
