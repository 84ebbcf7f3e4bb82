// Instantiations of the one-launch Bluestein pass for plain complex axes
// (axis_pass_chirp) and their launch shapes, shortest convolution first.
#define DFFT_PACKED_F32 1  // issue-bound butterflies
#include "chirp_pass.cuh"
#include "dfft_internal.h"

namespace dfft {

#define DFFT_CHIRP_INST(T, MINB, CS, P, R0, R1)                                                        \
  template __global__ void axis_pass_chirp<T, MINB, true, CS, P, R0, R1>(const __grid_constant__ PassDesc);  \
  template __global__ void axis_pass_chirp<T, MINB, false, CS, P, R0, R1>(const __grid_constant__ PassDesc);
#define K(T, MINB, CS, P, R0, R1)                                                                      \
  P, CS, (const void*)&axis_pass_chirp<T, MINB, true, CS, P, R0, R1>,                                  \
      (const void*)&axis_pass_chirp<T, MINB, false, CS, P, R0, R1>,                                    \
      sizeof(cvec<T>::type) * ChirpTile<cvec<T>::type, true, CS, R0 * R1>::ELEMS,                      \
      sizeof(cvec<T>::type) * ChirpTile<cvec<T>::type, false, CS, R0 * R1>::ELEMS

// R0 is even (DftHalf) and the larger radix, so that its stages give every
// thread one butterfly where P = R1
DFFT_CHIRP_INST(float, 4, 16, 8, 8, 8)
DFFT_CHIRP_INST(float, 4, 16, 8, 12, 8)
DFFT_CHIRP_INST(float, 4, 16, 8, 16, 8)
DFFT_CHIRP_INST(float, 4, 16, 8, 24, 8)
DFFT_CHIRP_INST(float, 3, 16, 16, 16, 16)
DFFT_CHIRP_INST(float, 2, 16, 16, 24, 16)
DFFT_CHIRP_INST(float, 2, 16, 16, 32, 16)
DFFT_CHIRP_INST(float, 2, 8, 24, 32, 24)
DFFT_CHIRP_INST(float, 2, 8, 32, 32, 32)
DFFT_CHIRP_INST(double, 4, 8, 8, 8, 8)
DFFT_CHIRP_INST(double, 4, 8, 8, 12, 8)
DFFT_CHIRP_INST(double, 4, 8, 8, 16, 8)
DFFT_CHIRP_INST(double, 3, 8, 12, 16, 12)
DFFT_CHIRP_INST(double, 3, 8, 16, 16, 16)
DFFT_CHIRP_INST(double, 2, 8, 16, 24, 16)
DFFT_CHIRP_INST(double, 2, 8, 16, 32, 16)

static const ChirpKernel kChirpKernels[] = {
    // dbl, M, R0, R1, P, columns, strided and contiguous kernels, their shared memory
    {0, 64, 8, 8, K(float, 4, 16, 8, 8, 8)},       {0, 96, 12, 8, K(float, 4, 16, 8, 12, 8)},
    {0, 128, 16, 8, K(float, 4, 16, 8, 16, 8)},    {0, 192, 24, 8, K(float, 4, 16, 8, 24, 8)},
    {0, 256, 16, 16, K(float, 3, 16, 16, 16, 16)}, {0, 384, 24, 16, K(float, 2, 16, 16, 24, 16)},
    {0, 512, 32, 16, K(float, 2, 16, 16, 32, 16)}, {0, 768, 32, 24, K(float, 2, 8, 24, 32, 24)},
    {0, 1024, 32, 32, K(float, 2, 8, 32, 32, 32)}, {1, 64, 8, 8, K(double, 4, 8, 8, 8, 8)},
    {1, 96, 12, 8, K(double, 4, 8, 8, 12, 8)},     {1, 128, 16, 8, K(double, 4, 8, 8, 16, 8)},
    {1, 192, 16, 12, K(double, 3, 8, 12, 16, 12)}, {1, 256, 16, 16, K(double, 3, 8, 16, 16, 16)},
    {1, 384, 24, 16, K(double, 2, 8, 16, 24, 16)}, {1, 512, 32, 16, K(double, 2, 8, 16, 32, 16)},
};

#undef K

const ChirpKernel* find_chirp_kernel(int dbl, int N) {
  for (const ChirpKernel& k : kChirpKernels)
    if (k.dbl == dbl && k.M >= 2 * N - 1) return &k;
  return nullptr;
}

}  // namespace dfft
