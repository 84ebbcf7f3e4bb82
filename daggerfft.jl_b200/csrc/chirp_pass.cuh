// Bluestein's algorithm (chirp-z) for plain complex axes in one launch, with
// a two-radix convolution length M = R0 * R1 >= 2N - 1:
//
//   forward FFT_M  radices R0, R1   of x_n w_n, zero-padded
//   times the filter spectrum, conjugated, in registers
//   inverse FFT_M  radices R1, R0   (the forward transform of the conjugate)
//   conjugated, times w_k, for k < N
//
// Both FFTs are Stockham transforms, and the last stage of the first leaves
// butterfly j holding the outputs j + r R0, exactly the inputs of butterfly
// j of the second one's first stage when its radices run the other way
// round: the filter multiply and that stage continue in registers.  So the
// tile makes two trips through shared memory in all (a stage at a time would
// be four exchanges, and five passes over the tile for the ends).  251 x 9800
// ComplexF32 columns, M = 512 (B200): 85 us in the general one-tile kernel,
// 29 us here, 1.4 TB/s of the columns' own bytes.  N <= M/2,
// so the first stage's second half of inputs is zero (DftHalf) and the last
// stage's second half of outputs is never formed.
//
// The kernel is bound by instruction issue.  A thread holds R0 (first and
// last stage) or ceil(R0/P) R1 elements.  Strided axes (CF): CS columns,
// column index fastest in the thread bits and in the tile, rows of 128
// bytes: every access is conflict-free.  Contiguous axis: a column per P
// lanes, padded.  Loads and stores go straight to global memory, in runs of
// CS elements or P elements.
#pragma once
#include "axis_pass.cuh"

namespace dfft {

template <typename V, bool CF, int CS, int M> struct ChirpTile {
  static constexpr int LD = M + M / (128 / (int)sizeof(V)) + 1;  // padded column
  static constexpr int ELEMS = CF ? M * CS : LD * CS;
  V* p;
  __device__ __forceinline__ ChirpTile(V* sm, int c) : p(CF ? sm + c : sm + c * LD) {}
  __device__ __forceinline__ V& at(int k) const { return p[CF ? k * CS : swz<V>(k)]; }
};

// d.in / d.out: complex sides of N = d.in.chirp_n elements per column, with
// the chirp table; d.tw: M entries exp(-2 pi i m / M); d.tw2: filter
// spectrum over M; d.scale at the store.
template <typename T, int MINB, bool CF, int CS, int P, int R0, int R1>
__global__ void __launch_bounds__(CS* P, MINB) axis_pass_chirp(const __grid_constant__ PassDesc d) {
  typedef typename cvec<T>::type V;
  constexpr int M = R0 * R1;
  constexpr int BA = (R1 + P - 1) / P;  // butterflies per thread of the radix-R0 stages
  constexpr int BB = (R0 + P - 1) / P;  // and of the radix-R1 stages
  extern __shared__ __align__(128) unsigned char smem_chirp[];
  const int tid = threadIdx.x;
  const int c = CF ? tid % CS : tid / P;
  const int t = CF ? tid / CS : tid % P;
  const ChirpTile<V, CF, CS, M> tile(reinterpret_cast<V*>(smem_chirp), c);
  const V* tw = reinterpret_cast<const V*>(d.tw);
  const V* filter = reinterpret_cast<const V*>(d.tw2);
  const V* chirp = reinterpret_cast<const V*>(d.in.chirp);
  const int N = d.in.chirp_n;
  const long long q = (long long)blockIdx.x * CS + c;
  const bool cv = q < d.Q;
  const long long qo = !cv ? 0 : d.I == 1 ? q : q / d.I;
  const long long qi = !cv || d.I == 1 ? 0 : q - qo * d.I;

  pass_entry();
  {  // radix R0 of the padded input
    const V* in = reinterpret_cast<const V*>(d.in.p) + (qi * d.in.si + io_outer(d.in, qo));
    const long long sk = d.in.sk;
#pragma unroll
    for (int b = 0; b < BA; ++b) {
      const int j = t + b * P;
      if (R1 % P != 0 && j >= R1) break;
      V v[R0];
#pragma unroll
      for (int r = 0; r < R0 / 2; ++r) {
        const int k = j + r * R1;
        v[r] = mk<V>((T)0, (T)0);
        if (cv && k < N) v[r] = in[k * sk];
      }
#pragma unroll
      for (int r = 0; r < R0 / 2; ++r) {
        const int k = j + r * R1;
        if (k < N) v[r] = cmul(v[r], ldg_c(chirp + k));
      }
      DftHalf<R0>::run(v);
#pragma unroll
      for (int r = 0; r < R0; ++r) tile.at(j * R0 + r) = v[r];
    }
  }
  __syncthreads();
  {  // radix R1, the filter, radix R1 of the inverse
    V v[BB][R1];
#pragma unroll
    for (int b = 0; b < BB; ++b) {
      const int j = t + b * P;
      if (R0 % P != 0 && j >= R0) break;
#pragma unroll
      for (int r = 0; r < R1; ++r) v[b][r] = tile.at(j + r * R0);
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < BB; ++b) {
      const int j = t + b * P;
      if (R0 % P != 0 && j >= R0) break;
#pragma unroll
      for (int r = 1; r < R1; ++r) v[b][r] = cmul(v[b][r], ldg_c(tw + j * r));
      Dft<R1>::run(v[b]);
#pragma unroll
      for (int r = 0; r < R1; ++r) v[b][r] = cconj(cmul(v[b][r], ldg_c(filter + j + r * R0)));
      Dft<R1>::run(v[b]);
#pragma unroll
      for (int r = 0; r < R1; ++r) tile.at(j * R1 + r) = v[b][r];
    }
  }
  __syncthreads();
  {  // radix R0 of the inverse
    V* out = reinterpret_cast<V*>(d.out.p) + (qi * d.out.si + io_outer(d.out, qo));
    const long long sk = d.out.sk;
    const T scale = (T)d.scale;
#pragma unroll
    for (int b = 0; b < BA; ++b) {
      const int j = t + b * P;
      if (R1 % P != 0 && j >= R1) break;
      V v[R0];
#pragma unroll
      for (int r = 0; r < R0; ++r) v[r] = tile.at(j + r * R1);
#pragma unroll
      for (int r = 1; r < R0; ++r) v[r] = cmul(v[r], ldg_c(tw + j * r));
      Dft<R0>::run(v);
#pragma unroll
      for (int r = 0; r < R0 / 2; ++r) {
        const int k = j + r * R1;
        if (cv && k < N) out[k * sk] = cscale(cmul(cconj(v[r]), ldg_c(chirp + k)), scale);
      }
    }
  }
}

}  // namespace dfft
