// Tile-staged R2R passes for DCT-II / DCT-III (FFTW REDFT10 / REDFT01, the
// R2R(...) kinds of src/fft.jl:1-11 the README's 2-D DCT uses): a producer
// warp moves whole input tiles into NB shared-memory buffers -- C whole
// pencils, one 1-D bulk copy each, along the contiguous axis (STRIDED = 0), C
// columns x N rows by TMA boxes of the real tensor {I, N, O} along a strided
// axis (STRIDED = 1) -- and the output leaves from the same buffer by the
// same kind of copy, which the producer issues when the buffer is handed back.
//
// Both kinds are a permutation of N reals around a real transform, which runs
// as one complex FFT of M = N/2 points (x the input, v its permutation, w =
// exp(-2 pi i / N), c_j = exp(-i pi j / 2N)):
//   DCT-II: v_k = x_{2k} | x_{2N-2k-1}; z_m = v_{2m} + i v_{2m+1}; Z = FFT_M(z);
//     E = (Z_k + conj Z_{M-k})/2, T = -i w^k (Z_k - conj Z_{M-k})/2,
//     V_k = E + T, V_{M-k} = conj(E - T); with q = c_j V_j:
//     Y_j = 2 Re q, Y_{N-j} = -2 Im q.
//   DCT-III: V_j = conj(c_j) (x_j - i x_{N-j}), x_N = 0; A = V_k, B = conj
//     V_{M-k}, S = A + B, U = i conj(w^k) (A - B), Z_k = S + U, Z_{M-k} =
//     conj(S - U); z = IFFT_M(Z) (unnormalised); v_{2m} = Re z_m, v_{2m+1} =
//     Im z_m, stored at the permuted places.
// (A complex FFT of the N reals with zero imaginary parts took twice the
// FP64 work and shared-memory traffic: 256 x 256 x 32 Float64 DCT-II +
// DCT-III, four passes, 54 us.)  The FFT runs in a padded complex work
// buffer, one column per real column; columns stay independent of one
// another.  Bounded waits as in the other pipelined passes.
// Eight stage warps per SM: a tile's time is a chain of latencies, so the
// loops over k are unrolled (their table and tile reads go out together) and
// the planner launches no more CTAs than the rounds need.  256 x 256 Float64,
// DCT-II + DCT-III of 20, 41 and 58 planes (1.1, 2.2 and 3.1 rounds of CTAs):
// 49.0, 70.8 and 89.8 us with a round of k at a time on a full grid, 45.2,
// 62.9 and 78.8 so; 46.4, 63.8 and 85.1 by FFTs of N points.
#pragma once
#include "real_pass.cuh"

namespace dfft {

// Place of v_k in the data: x_{2k} | x_{2N-2k-1}.
template <int N> __device__ __forceinline__ int dct_place(int k) { return 2 * k < N ? 2 * k : 2 * N - 2 * k - 1; }
// The tile of one column / pencil as the packed sequence z_m (stride S
// between its elements: C in a strided tile, 1 in a contiguous one).
template <typename T, int N, int S> struct DctView {
  typedef typename cvec<T>::type V;
  T* p;
  __device__ __forceinline__ V ld(int b, int off) const {
    const int m = b + off;
    return mk<V>(p[dct_place<N>(2 * m) * S], p[dct_place<N>(2 * m + 1) * S]);
  }
  __device__ __forceinline__ void st(int b, int off, V v) const {
    const int m = b + off;
    p[dct_place<N>(2 * m) * S] = v.x;
    p[dct_place<N>(2 * m + 1) * S] = v.y;
  }
};

struct TiledGeom {
  long long ntiles;  // contiguous: ceil(pencils / C); strided: tiles_i * O
  long long pencils; // contiguous: pencils in all (the last tile may hold fewer than C)
  int tiles_i;       // strided: tiles along I
  int lb, nlb;       // strided: rows per TMA box, boxes per tile
  int ld;            // padded complex work elements per column
  int bstride;       // bytes between tile buffers (128-byte multiple)
  const void* src;   // global input
  void* dst;         // global output
  int* err;
};

template <typename T, int LB, int MINB, int NB, int STRIDED, int KIND, int N, int P, int C, int... Rs>
__global__ void __launch_bounds__(LB, MINB)
    tiled_pass(const PassDesc d, const __grid_constant__ CUtensorMap tin,
               const __grid_constant__ CUtensorMap tout, const TiledGeom g) {
  typedef typename cvec<T>::type V;
  constexpr int NC = C * P;
  constexpr int M = N / 2;                     // FFT length
  static_assert(M / 2 % P == 0, "whole rounds of the split / merge loops over k < M/2");
  constexpr int PS = N + 64 / (int)sizeof(T);  // contiguous tiles: elements between pencils (spread over the banks)
  static_assert(NC % 32 == 0 && NC + 32 == LB, "whole warps of stage threads plus one producer warp");
  static_assert(NB >= 2 && NB <= 4, "tile buffers");
  extern __shared__ __align__(128) unsigned char smem_tiled[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_tiled);
  uint64_t* empty = reinterpret_cast<uint64_t*>(smem_tiled + 32);
  int& s_cabort = *reinterpret_cast<int*>(smem_tiled + 64);
  long long* s_tile = reinterpret_cast<long long*>(smem_tiled + 80);  // NB entries
  unsigned char* bufs = smem_tiled + kSlabHeader;
  const size_t bst = (size_t)g.bstride;
  V* work = reinterpret_cast<V*>(bufs + NB * bst);
  const int tid = threadIdx.x;
  volatile int* verr = g.err;

  if (tid == 0) {
    for (int b = 0; b < NB; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], 1);
    }
    mbar_fence_init();
    s_cabort = 0;
    if ((smem_u32(bufs) & 127u) || (bst & 127u) ||
        (STRIDED && g.nlb > 1 && (((size_t)g.lb * C * sizeof(T)) & 127u))) {
      atomicExch(g.err, DFFT_DEVERR_TMA_ALIGN);
      s_cabort = 1;
    }
  }
  __syncthreads();
  pass_entry();

  if (tid >= NC) {
    if (tid == NC) {
      // ---------------- producer ----------------
      int fills[NB] = {};
      long long pend[NB];  // transformed tile in buffer b still to be stored, or -1
      for (int bb = 0; bb < NB; ++bb) pend[bb] = -1;
      bool failed = false;
      // waits until the stage threads hand buffer b back, then stores its
      // tile and waits until the store has read the buffer
      auto drain = [&](int b) -> bool {
        if (pend[b] < 0) return true;
        if (!mbar_wait_bounded(&empty[b], (uint32_t)((fills[b] - 1) & 1))) return false;
        unsigned char* buf = bufs + b * bst;
        if (STRIDED) {
          const int ti = (int)(pend[b] % g.tiles_i);
          const int o = (int)(pend[b] / g.tiles_i);
          for (int kb = 0; kb < g.nlb; ++kb)
            tma_store_3d(&tout, buf + (size_t)kb * g.lb * C * sizeof(T), ti * C, kb * g.lb, o);
        } else {
          const int nv = (int)min((long long)C, g.pencils - pend[b] * C);
          for (int cc = 0; cc < nv; ++cc)
            bulk_store_1d(reinterpret_cast<T*>(g.dst) + (pend[b] * C + cc) * N, buf + (size_t)cc * PS * sizeof(T),
                          (uint32_t)(N * sizeof(T)));
        }
        bulk_commit();
        bulk_wait_read_all();
        pend[b] = -1;
        return true;
      };
      long long tile = blockIdx.x;
      for (int it = 0;; ++it) {
        const int b = it % NB;
        if (!drain(b)) {
          failed = true;
          break;
        }
        const bool more = tile < g.ntiles && *verr == 0 && !s_cabort;
        s_tile[b] = more ? tile : -1;
        ++fills[b];
        if (!more) {
          mbar_arrive(&full[b]);
          break;
        }
        unsigned char* buf = bufs + b * bst;
        const int nv = STRIDED ? C : (int)min((long long)C, g.pencils - tile * C);
        mbar_expect_tx(&full[b], (uint32_t)((size_t)nv * N * sizeof(T)));
        if (STRIDED) {
          const int ti = (int)(tile % g.tiles_i);
          const int o = (int)(tile / g.tiles_i);
          for (int kb = 0; kb < g.nlb; ++kb)
            tma_load_3d(buf + (size_t)kb * g.lb * C * sizeof(T), &tin, &full[b], ti * C, kb * g.lb, o);
        } else {
          for (int cc = 0; cc < nv; ++cc)
            bulk_load_1d(buf + (size_t)cc * PS * sizeof(T), reinterpret_cast<const T*>(g.src) + (tile * C + cc) * N,
                         (uint32_t)(N * sizeof(T)), &full[b]);
        }
        pend[b] = tile;
        tile += gridDim.x;
      }
      for (int bb = 0; bb < NB && !failed; ++bb)
        if (!drain(bb)) failed = true;
      if (failed && *verr == 0) atomicExch(g.err, DFFT_DEVERR_TMA_TIMEOUT);
      bulk_wait_all();
      for (int bb = 0; bb < NB; ++bb)
        if (fills[bb] > 0) mbar_wait_bounded(&full[bb], (uint32_t)((fills[bb] - 1) & 1));
    }
  } else {
    // ---------------- stage threads ----------------
    const int c = STRIDED ? tid % C : tid / P;
    const int t = STRIDED ? tid / C : tid % P;
    const PadCol<V> col{work + (size_t)c * g.ld};
    const GlobalTw<V> tw{reinterpret_cast<const V*>(d.tw)};
    constexpr int S = STRIDED ? C : 1;
    constexpr int DIR = KIND == K_REDFT01 ? 2 : 1;  // REDFT01 runs as an inverse FFT
    const V* w = reinterpret_cast<const V*>(d.tw2);  // w^k, k <= M/2
    const V* cj = reinterpret_cast<const V*>(KIND == K_REDFT01 ? d.in.w : d.out.w);  // conj(c_j) / c_j
    for (int it = 0;; ++it) {
      const int b = it % NB;
      if (!mbar_wait_bounded(&full[b], (uint32_t)((it / NB) & 1))) s_cabort = 1;
      stage_sync<NC>();
      if (s_cabort) break;
      const long long tile = s_tile[b];
      if (tile < 0) break;
      unsigned char* buf = bufs + b * bst;
      T* x = reinterpret_cast<T*>(buf) + (STRIDED ? c : c * PS);  // element n at x[n * S]
      const DctView<T, N, S> view{x};
      if constexpr (KIND == K_REDFT01) {
        const auto merge = [&](int k) {
          const T xn = k == 0 ? (T)0 : x[(N - k) * S];
          const V A = cmul(ldg_c(cj + k), mk<V>(x[k * S], -xn));
          const V B = cconj(cmul(ldg_c(cj + M - k), mk<V>(x[(M - k) * S], -x[(M + k) * S])));
          const V U = cmul_pi(cmul(cconj(ldg_c(w + k)), csub(A, B)));
          const V Z = cadd(A, B);
          col.st(k, 0, cadd(Z, U));
          if (k > 0) col.st(M - k, 0, cconj(csub(Z, U)));
        };
#pragma unroll 4
        for (int i = 0; i < M / 2 / P; ++i) merge(t + i * P);
        if (t == 0) merge(M / 2);
        stage_sync<NC>();
        static_stages<T, M, P, 1, NC, DIR, 1, 1, 0, PadCol<V>, PadCol<V>, DctView<T, N, S>, GlobalTw<V>, Rs...>(
            d, t, col, col, view, tw, 0, 0, true);
      } else {
        static_stages<T, M, P, 1, NC, DIR, 1, 1, 0, DctView<T, N, S>, PadCol<V>, PadCol<V>, GlobalTw<V>, Rs...>(
            d, t, view, col, col, tw, 0, 0, true);
        const auto split = [&](int k) {
          const V zk = col.ld(k, 0), zm = cconj(col.ld(k == 0 ? 0 : M - k, 0));
          const V E = cscale(cadd(zk, zm), (T)0.5);
          const V U = cmul(ldg_c(w + k), cscale(cmul_mi(csub(zk, zm)), (T)0.5));
          const V q = cmul(ldg_c(cj + k), cadd(E, U));
          const V r = cmul(ldg_c(cj + M - k), cconj(csub(E, U)));
          x[k * S] = (T)2 * q.x;
          if (k > 0) x[(N - k) * S] = (T)-2 * q.y;
          x[(M - k) * S] = (T)2 * r.x;
          x[(M + k) * S] = k == 0 ? (T)2 * r.x : (T)-2 * r.y;
        };
#pragma unroll 4
        for (int i = 0; i < M / 2 / P; ++i) split(t + i * P);
        if (t == 0) split(M / 2);
      }
      fence_proxy_async_smem();  // the producer's store reads the tile next
      stage_sync<NC>();
      if (tid == 0) mbar_arrive(&empty[b]);  // hand the transformed tile to the producer
    }
    if (tid == 0 && s_cabort && *verr == 0) atomicExch(g.err, DFFT_DEVERR_TMA_TIMEOUT);
  }
  __syncthreads();
}

}  // namespace dfft
