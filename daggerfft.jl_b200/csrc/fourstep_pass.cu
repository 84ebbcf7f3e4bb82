// Instantiations of the first pass of a four-step axis (four_step_first).
// Columns per tile: rows of 32 bytes at least, and 256 CTAs for 2^20 points.
#define DFFT_PACKED_F32 1
#include "fourstep_pass.cuh"
#include "dfft_internal.h"

namespace dfft {

#define DFFT_FS(X)                                                                                          \
  X(float, 0, 4, 8, 8, 16, 8) X(float, 0, 4, 8, 10, 16, 10) X(float, 0, 4, 8, 12, 16, 12)                   \
  X(float, 0, 4, 8, 15, 15, 15) X(float, 0, 4, 8, 16, 15, 16) X(float, 0, 4, 8, 16, 16, 16)                 \
  X(float, 0, 4, 8, 10, 32, 10) X(float, 0, 4, 8, 15, 24, 15) X(float, 0, 4, 8, 16, 24, 16)                 \
  X(float, 0, 3, 8, 15, 32, 15) X(float, 0, 3, 8, 16, 32, 16) X(float, 0, 2, 4, 24, 24, 24)                 \
  X(float, 0, 2, 4, 24, 32, 24) X(float, 0, 2, 4, 32, 32, 32)                                               \
  X(double, 1, 2, 8, 8, 16, 8) X(double, 1, 2, 4, 10, 16, 10) X(double, 1, 2, 4, 12, 16, 12)                \
  X(double, 1, 2, 4, 15, 15, 15) X(double, 1, 2, 4, 16, 15, 16) X(double, 1, 2, 4, 16, 16, 16)              \
  X(double, 1, 2, 4, 10, 32, 10) X(double, 1, 2, 4, 15, 24, 15) X(double, 1, 2, 4, 16, 24, 16)              \
  X(double, 1, 2, 4, 15, 32, 15) X(double, 1, 2, 4, 16, 32, 16) X(double, 1, 2, 4, 24, 24, 24)              \
  X(double, 1, 2, 2, 24, 32, 24) X(double, 1, 2, 2, 32, 32, 32)

#define INST(T, DBL, MINB, CS, P, R0, R1)                                                                   \
  template __global__ void four_step_first<T, MINB, CS, P, R0, R1>(const cvec<T>::type*,                    \
                                                                   cvec<T>::type*,                          \
                                                                   const __grid_constant__ FourStepGeom);
DFFT_FS(INST)
#undef INST

#define ENTRY(T, DBL, MINB, CS, P, R0, R1)                                                                  \
  {DBL, R0* R1, R0, R1, P, CS, (const void*)&four_step_first<T, MINB, CS, P, R0, R1>,                       \
   sizeof(cvec<T>::type) * (FourStepTile<cvec<T>::type, CS, R0, R1>::ELEMS + kTwSplit)},
static const FourStepKernel kFourStep[] = {DFFT_FS(ENTRY)};
#undef ENTRY

const FourStepKernel* find_four_step_kernel(int dbl, int M) {
  for (const FourStepKernel& k : kFourStep)
    if (k.dbl == dbl && k.M == M) return &k;
  return nullptr;
}

}  // namespace dfft
