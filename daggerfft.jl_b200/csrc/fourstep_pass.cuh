// First pass of a four-step axis (L = L1 * M, unit inner stride): M-point
// transforms with two radices, M = R0 * R1, along the sub-axis n2 of the
// columns n1 (x[n1 + L1 n2]), times W_L^(n1 k2), written with the sub-axes
// swapped (k2 fastest), so that the second pass is an ordinary strided one.
//
// At these sizes a pass is one wave of CTAs and its time is the chain of
// latencies from the first load to the last store, not bandwidth (2^20
// ComplexF32: 8.4 MB each way, 2.6 us of memory time; 26 us in the general
// one-tile kernel, 12 us here).  So a thread's R0 loads go straight from global memory to
// registers, all in flight at once, there is one exchange, and the stores
// leave from registers.  The first stage maps lanes to columns (rows of CS
// elements are contiguous in the input), the second to butterflies (P
// consecutive elements of one column are contiguous in the output); the
// exchange in between carries the swap.  Tile layout: element q R0 + s of
// column c at c LD + q PITCH + s, PITCH the odd one of R0 and R0 + 1 and LD
// = 128 bytes / CS modulo 128 bytes, conflict-free on both sides.  The low part of the split twiddle
// table sits in shared memory: lanes read it n1 entries apart, which the L1
// serves a line at a time.
#pragma once
#include "axis_pass.cuh"

namespace dfft {

struct FourStepGeom {
  int L1;        // columns per transform
  int tiles;     // tiles of CS columns per transform
  long long in_o, out_o;  // elements between transforms
  // Bluestein around the pair: element n = n1 + L1 k2 of the input times
  // chirp[n] (zero from chirp_n on), or times mul[n]
  const void* chirp;
  const void* mul;
  int chirp_n;
  int inverse;
  const void* tw;   // M entries exp(-2 pi i m / M)
  const void* twl;  // split twiddle table of W_L
  int tw_log;       // log2 of its split
};

template <typename V, int CS, int R0, int R1> struct FourStepTile {
  static constexpr int ROW = 128 / (int)sizeof(V);
  static constexpr int STEP = CS < ROW ? ROW / CS : 1;
  static constexpr int PITCH = R0 | 1;  // odd: strides of R0 elements reach every bank
  static constexpr int RAW = R1 * PITCH;
  static constexpr int LD = RAW + ((STEP - RAW) % ROW + ROW) % ROW;
  static constexpr int ELEMS = CS * LD;
};

template <typename T, int MINB, int CS, int P, int R0, int R1>
__global__ void __launch_bounds__(CS* P, MINB)
    four_step_first(const typename cvec<T>::type* in, typename cvec<T>::type* out,
                    const __grid_constant__ FourStepGeom g) {
  typedef typename cvec<T>::type V;
  typedef FourStepTile<V, CS, R0, R1> Tile;
  constexpr int M = R0 * R1;
  constexpr int BB = (R0 + P - 1) / P;  // radix-R1 butterflies per thread
  static_assert(P == R1, "one radix-R0 butterfly per thread");
  extern __shared__ __align__(128) unsigned char smem_fs[];
  V* sm = reinterpret_cast<V*>(smem_fs);
  V* lo = sm + Tile::ELEMS;
  const int tid = threadIdx.x;
  const int o = blockIdx.x / g.tiles;
  const int n1_0 = (blockIdx.x - o * g.tiles) * CS;
  const V* twl = reinterpret_cast<const V*>(g.twl);
  const V* tw = reinterpret_cast<const V*>(g.tw);
  const int sh = g.tw_log;
  for (int i = tid; i < 1 << sh; i += CS * P) lo[i] = twl[i];
  pass_entry();
  {
    const int c = tid % CS, j = tid / CS;
    const int n1 = n1_0 + c;
    const V* src = in + o * g.in_o + n1;
    V v[R0];
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const int n = (j + r * R1) * g.L1;
      v[r] = mk<V>((T)0, (T)0);
      if (n1 < g.L1 && (!g.chirp || n1 + n < g.chirp_n)) v[r] = src[n];
    }
    if (g.chirp || g.mul) {
      const V* f = reinterpret_cast<const V*>(g.chirp ? g.chirp : g.mul) + n1;
#pragma unroll
      for (int r = 0; r < R0; ++r) {
        const int n = (j + r * R1) * g.L1;
        if (n1 < g.L1 && (!g.chirp || n1 + n < g.chirp_n)) v[r] = cmul(v[r], ldg_c(f + n));
      }
    }
    if (g.inverse) {
#pragma unroll
      for (int r = 0; r < R0; ++r) v[r].y = -v[r].y;
    }
    Dft<R0>::run(v);
    V* col = sm + c * Tile::LD + j * Tile::PITCH;
#pragma unroll
    for (int r = 0; r < R0; ++r) col[r] = v[r];
  }
  __syncthreads();
  {
    const int t = tid % P, c = tid / P;
    const int n1 = n1_0 + c;
    const V* col = sm + c * Tile::LD;
    V* dst = out + o * g.out_o + (long long)n1 * M;
    const V* hi = twl + (1 << sh);
#pragma unroll
    for (int b = 0; b < BB; ++b) {
      const int j = t + b * P;
      if (R0 % P != 0 && j >= R0) break;
      V v[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = col[r * Tile::PITCH + j];
#pragma unroll
      for (int r = 1; r < R1; ++r) v[r] = cmul(v[r], ldg_c(tw + j * r));
      Dft<R1>::run(v);
      if (n1 >= g.L1) continue;
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        const unsigned k = j + r * R0, m = (unsigned)n1 * k;
        if (g.inverse) v[r].y = -v[r].y;
        dst[k] = cmul(v[r], split_twiddle(lo[m & ((1u << sh) - 1)], hi + 2 * (m >> sh)));
      }
    }
  }
}

}  // namespace dfft
