// Instantiations of the one-launch Bluestein passes, shortest convolution
// first: plain complex axes (axis_pass_chirp) with their launch shapes, and
// the general one-tile kernel (axis_pass_any) for the other sides and the
// longer convolutions.
#define DFFT_PACKED_F32 1  // issue-bound butterflies
#include "any_pass.cuh"
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

// The general kernel: dtype, launch bound, length, threads per column, radices.
// Lengths at most a third apart from 36 up: 298455 Float64 columns of 17
// points, DCT-III, 282 us through 64 points, within 2 % of the 240 of two
// passes through 36.  Beyond 2048 a column is one CTA and with few of them its time a chain of
// latencies: four stages with more threads a column (64 x 1083 Float32 DCT-II:
// 2304 as 12 x 12 x 16 on 192 threads 29.8 us, as 6 x 6 x 8 x 8 on 384 20).
#define DFFT_CHIRP_ANY(X)                                                                              \
  X(float, 0, 1024, 36, 6, 6, 6) X(float, 0, 1024, 48, 8, 8, 6)                                        \
  X(float, 0, 1024, 64, 8, 8, 8) X(float, 0, 1024, 80, 8, 10, 8)                                       \
  X(float, 0, 1024, 96, 8, 12, 8) X(float, 0, 1024, 128, 8, 16, 8)                                     \
  X(float, 0, 1024, 160, 16, 16, 10) X(float, 0, 512, 192, 12, 12, 16)                                 \
  X(float, 0, 1024, 256, 16, 16, 16) X(float, 0, 1024, 320, 40, 5, 8, 8)                               \
  X(float, 0, 1024, 384, 48, 6, 8, 8) X(float, 0, 1024, 512, 64, 8, 8, 8)                              \
  X(float, 0, 1024, 640, 64, 10, 8, 8) X(float, 0, 1024, 768, 64, 12, 8, 8)                            \
  X(float, 0, 1024, 1024, 64, 16, 8, 8) X(float, 0, 1024, 1280, 128, 10, 16, 8)                        \
  X(float, 0, 1024, 1536, 128, 12, 16, 8) X(float, 0, 1024, 2048, 128, 16, 16, 8)                      \
  X(float, 0, 1024, 2304, 384, 6, 6, 8, 8) X(float, 0, 1024, 2560, 512, 5, 8, 8, 8)                    \
  X(float, 0, 1024, 3072, 256, 12, 16, 16) X(float, 0, 1024, 3200, 400, 10, 8, 8, 5) X(float, 0, 1024, 3600, 360, 10, 10, 6, 6)                    \
  X(float, 0, 1024, 4096, 512, 8, 8, 8, 8) X(double, 1, 512, 36, 6, 6, 6)                              \
  X(double, 1, 512, 48, 8, 8, 6) X(double, 1, 512, 64, 8, 8, 8)                                        \
  X(double, 1, 512, 80, 8, 10, 8) X(double, 1, 512, 96, 8, 12, 8)                                      \
  X(double, 1, 512, 128, 8, 16, 8) X(double, 1, 512, 160, 16, 16, 10)                                  \
  X(double, 1, 512, 192, 12, 12, 16) X(double, 1, 512, 256, 16, 16, 16)                                \
  X(double, 1, 512, 320, 40, 5, 8, 8) X(double, 1, 512, 384, 48, 6, 8, 8)                              \
  X(double, 1, 512, 512, 64, 8, 8, 8) X(double, 1, 512, 640, 64, 10, 8, 8)                             \
  X(double, 1, 512, 768, 64, 12, 8, 8) X(double, 1, 512, 1024, 64, 16, 8, 8)                           \
  X(double, 1, 512, 1280, 128, 10, 16, 8) X(double, 1, 512, 1536, 128, 12, 16, 8)                      \
  X(double, 1, 512, 2048, 128, 16, 16, 8)

#define INST(T, DBL, LB, L, P, ...) \
  template __global__ void axis_pass_any<T, LB, true, L, P, __VA_ARGS__>(const __grid_constant__ PassDesc);
DFFT_CHIRP_ANY(INST)
#undef INST

#define ENTRY(T, DBL, LB, L, P, ...) {DBL, L, P, LB, {__VA_ARGS__}, (const void*)&axis_pass_any<T, LB, true, L, P, __VA_ARGS__>},
static const ChirpAnyKernel kChirpAny[] = {DFFT_CHIRP_ANY(ENTRY)};
#undef ENTRY

const ChirpAnyKernel* find_chirp_any(int dbl, int least) {
  for (const ChirpAnyKernel& k : kChirpAny)
    if (k.dbl == dbl && k.L >= least) return &k;
  return nullptr;
}

}  // namespace dfft
